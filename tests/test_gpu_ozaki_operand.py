"""The ozaki path's operand kernel (exponents and digits of A in one launch): rows and l ranges that
fill no block or chunk, contiguous fibres on and off 16-byte boundaries, rows of zeros, signed zeros
and magnitudes far apart. Entries are integers times a power of two per fibre, so that every digit and
every sum is exact and the product must match bit for bit; and random entries within the path's 1e-12."""
import numpy as np
import pytest

from ttm_b200 import _lib

pytestmark = pytest.mark.gpu


def _dense(n, pi):
    w = [1] * len(n)
    for r in range(1, len(n)):
        w[pi[r] - 1] = w[pi[r - 1] - 1] * n[pi[r - 1] - 1]
    return w


def _run(cuda, a, b, shift=0):
    import torch
    outer, nq, inner = a.shape
    m = b.shape[0]
    ta = torch.empty(a.size + shift, dtype=torch.float64, device=cuda)
    ta[shift:] = torch.from_numpy(a.reshape(-1)).to(cuda)
    tb = torch.from_numpy(b).to(cuda)
    tc = torch.full((outer, m, inner), float("nan"), dtype=torch.float64, device=cuda)
    na, nc, pia = [inner, nq, outer], [inner, m, outer], [1, 2, 3]
    _lib.ttm_raw(_lib.F64, _lib.PREC_OZAKI, 2, 3, ta.data_ptr() + 8 * shift, na, _dense(na, pia), pia, tb.data_ptr(),
                 [m, nq], [2, 1], tc.data_ptr(), nc, _dense(nc, pia), torch.cuda.current_stream().cuda_stream)
    assert _lib.last_kernel() == "tc_ozaki"
    torch.cuda.synchronize()
    return tc.cpu().numpy()


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("outer,nq,inner,m", [(1, 5, 31, 17), (3, 32, 43, 20), (2, 33, 128, 64), (129, 47, 1, 33),
                                              (31, 64, 1, 100), (257, 50, 1, 17), (4, 100, 129, 70)])
def test_exact_on_scaled_integers(cuda, outer, nq, inner, m, shift):
    rng = np.random.default_rng(nq + m)
    scale = 2.0 ** rng.integers(-40, 41, (outer, 1, inner))
    a = rng.integers(-1000, 1001, (outer, nq, inner)) * scale
    a[rng.random(a.shape) < 0.1] = -0.0
    a[0, :, 0] = 0.0                                       # a fibre of zeros
    b = rng.integers(-1000, 1001, (m, nq)).astype(np.float64)
    want = np.einsum("kli,jl->kji", a / scale, b) * scale   # integers below 2^53, then a power of two
    assert np.array_equal(_run(cuda, a, b, shift), want)


@pytest.mark.parametrize("outer,nq,inner,m", [(5, 70, 100, 40), (300, 70, 1, 40)])
def test_random_entries(cuda, outer, nq, inner, m):
    rng = np.random.default_rng(1)
    a = rng.standard_normal((outer, nq, inner)) * 10.0 ** rng.uniform(-4, 4, (outer, nq, inner))
    b = rng.standard_normal((m, nq))
    want = np.einsum("kli,jl->kji", a.astype(np.longdouble), b.astype(np.longdouble)).astype(np.float64)
    got = _run(cuda, a, b)
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 1e-12


@pytest.mark.parametrize("outer,nq,inner,m", [(3, 70, 43, 20), (129, 70, 1, 33)])
def test_non_finite_entries(cuda, outer, nq, inner, m):
    """A NaN of either sign has zero digits; an infinity spoils its own fibre only."""
    rng = np.random.default_rng(2)
    a = rng.integers(-1000, 1001, (outer, nq, inner)).astype(np.float64)
    b = rng.integers(-1000, 1001, (m, nq)).astype(np.float64)
    nan = rng.random(a.shape) < 0.1
    want = np.einsum("kli,jl->kji", np.where(nan, 0.0, a), b)
    bad = np.where(nan, np.where(rng.random(a.shape) < 0.5, np.nan, -np.nan), a)
    assert np.array_equal(_run(cuda, bad, b), want)
    bad[1, 7, 0] = np.inf
    bad[2, 9, 0] = -np.inf
    got = _run(cuda, bad, b)
    keep = np.ones((outer, 1, inner), bool)
    keep[1, 0, 0] = keep[2, 0, 0] = False
    assert np.array_equal(np.where(keep, got, 0.0), np.where(keep, want, 0.0))
