"""The single-SM bf16x3 kernel with M tiles made of two half tiles of 64 rows (inner past a multiple of
128 by at most 64): odd and even numbers of halves, halves of one tile in different slices, partial
halves, one tile at a time and pairs, C with and without a tensor map, and a grouped launch.

Bound: the repository's 1e-5 (relative Frobenius norm) for the FP32-accurate arithmetic."""
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
    assert torch.isfinite(C).all()
    want = torch.einsum("kli,jl->kji", A.double(), B.double())
    return float((C.double() - want).norm() / want.norm())


CASES = [(1, 20, 132, 32), (3, 33, 132, 100), (5, 16, 192, 64), (2, 50, 300, 96), (151, 40, 300, 128), (149, 36, 148, 48),
         (7, 300, 300, 200), (4, 20, 320, 300), (333, 17, 68, 24), (100, 52, 188, 20)]


@pytest.mark.parametrize("outer,nq,inner,m", CASES)
def test_half_tiles(cuda, outer, nq, inner, m):
    g = torch.Generator(device=cuda).manual_seed(outer + m)
    A = torch.randn(outer, nq, inner, device=cuda, generator=g)
    B = torch.randn(m, nq, device=cuda, generator=g)
    C = torch.full((outer * m * inner + 64,), float("nan"), device=cuda)
    na, nc, pia = [inner, nq, outer], [inner, m, outer], [1, 2, 3]
    _lib.ttm_raw(_lib.F32, _lib.PREC_BF16X3, 2, 3, A.data_ptr(), na, _dense(na, pia), pia, B.data_ptr(), [m, nq], [2, 1],
                 C.data_ptr(), nc, _dense(nc, pia), torch.cuda.current_stream().cuda_stream)
    assert _lib.last_kernel() == "tc_bf16x3"
    torch.cuda.synchronize()
    assert torch.isnan(C[outer * m * inner:]).all()
    assert _err(A, B, C[:outer * m * inner].view(outer, m, inner)) <= TOL


def test_half_tiles_in_a_grouped_launch(cuda):
    from ttm_b200.plans import BatchPlan
    g = torch.Generator(device=cuda).manual_seed(3)
    probs = []
    for outer, nq, inner, m in CASES + [(6, 40, 256, 64), (9, 24, 40, 80), (1301, 24, 164, 40)]:
        na = [inner, nq, outer]
        probs.append(dict(q=2, na=na, pia=[1, 2, 3], m=m, A=torch.randn(outer, nq, inner, device=cuda, generator=g),
                          B=torch.randn(m, nq, device=cuda, generator=g),
                          C=torch.full((outer, m, inner), float("nan"), device=cuda)))
    plan = BatchPlan(probs, precision="bf16x3")
    for _ in range(2):
        plan.run()
    torch.cuda.synchronize()
    for p in probs:
        assert _err(p["A"], p["B"], p["C"]) <= TOL, (p["na"], p["m"])
    plan.close()
