"""The single-SM bf16x3 kernel with M tiles in pairs (at most 128 columns): even and odd tile counts
per block, a last single tile, folded and partial tiles, contiguous fibres; and grouped launches in
which wide problems (over 128 columns) share the launch of many narrow ones.

Bound: the repository's 1e-5 (relative Frobenius norm) for the FP32-accurate arithmetic."""
import numpy as np
import pytest
import torch

from ttm_b200 import _lib

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _dense(n, pi):
    w = [1] * len(n)
    for r in range(1, len(n)):
        w[pi[r] - 1] = w[pi[r - 1] - 1] * n[pi[r - 1] - 1]
    return w


def _err(A, B, C):
    """C (outer, m, inner) against A (outer, n_q, inner) and B (m, n_q) in FP64 on the device."""
    assert torch.isfinite(C).all()
    want = torch.einsum("kli,jl->kji", A.double(), B.double())
    return float((C.double() - want).norm() / want.norm())


# blocks' shares of M tiles: under one, one, two (one and two tiles over), three, many; partial
# tiles; two and four slices per tile; n_q of one sub-block and just past a stage
@pytest.mark.parametrize("outer,nq,inner,m", [
    (1, 40, 100, 32), (1, 16, 128, 17), (150, 33, 128, 100), (149, 40, 200, 128), (443, 20, 128, 64),
    (700, 50, 60, 40), (1300, 36, 20, 24), (5001, 17, 128, 32), (128, 96, 1, 48), (38017, 36, 1, 96),
    (57000, 20, 1, 30), (100, 52, 301, 64), (20001, 45, 1, 64)])
def test_tile_pairs(cuda, outer, nq, inner, m):
    g = torch.Generator(device=cuda).manual_seed(outer + m)
    A = torch.randn(outer, nq, inner, device=cuda, generator=g)
    B = torch.randn(m, nq, device=cuda, generator=g)
    C = torch.full((outer, m, inner), float("nan"), device=cuda)
    na, nc, pia = [inner, nq, outer], [inner, m, outer], [1, 2, 3]
    _lib.ttm_raw(_lib.F32, _lib.PREC_BF16X3, 2, 3, A.data_ptr(), na, _dense(na, pia), pia, B.data_ptr(), [m, nq], [2, 1],
                 C.data_ptr(), nc, _dense(nc, pia), torch.cuda.current_stream().cuda_stream)
    assert _lib.last_kernel() == "tc_bf16x3"
    torch.cuda.synchronize()
    assert _err(A, B, C) <= TOL


@pytest.mark.parametrize("narrow,wide,launches", [(700, 3, 2), (3, 700, 2), (700, 700, 3)])
def test_wide_and_narrow_problems_in_one_group(cuda, narrow, wide, launches):
    """Counts of M tiles on either side of the number that gets a launch of its own."""
    from ttm_b200.plans import BatchPlan
    g = torch.Generator(device=cuda).manual_seed(3)
    probs = []
    for outer, nq, m in ((narrow - 1, 20, 96), (1, 50, 17), (wide - 1, 36, 256), (1, 70, 300)):
        na = [128, nq, outer]
        probs.append(dict(q=2, na=na, pia=[1, 2, 3], m=m, A=torch.randn(outer, nq, 128, device=cuda, generator=g),
                          B=torch.randn(m, nq, device=cuda, generator=g),
                          C=torch.full((outer, m, 128), float("nan"), device=cuda)))
    plan = BatchPlan(probs, precision="bf16x3")
    assert plan.launches == launches
    plan.run()
    torch.cuda.synchronize()
    for p in probs:
        assert _err(p["A"], p["B"], p["C"]) <= TOL, (p["na"], p["m"])
    plan.close()
