"""The memory for the parts of a split l range (small m): calls that found none before go on without it
where there is none, no graph that a caller captures holds an allocation for it, and plans hold their
own."""
import numpy as np
import pytest

import known_answer as ka
from ttm_b200 import _lib

pytestmark = pytest.mark.gpu

# rows of i (the column kernel's otherwise) and contiguous fibres (the l-split kernels')
STRIDED, FIBRES = ([2047, 4000, 1], 2, 8, "colvec"), ([4097, 2048], 1, 3, "bvec")


@pytest.fixture(autouse=True)
def _clear_injections():
    yield
    _lib.inject(_lib.INJECT_NONE)


class Problem:
    def __init__(self, cuda, na, q, m, dtype="float32"):
        import torch
        self.na, self.q, self.m = na, q, m
        self.pia = list(range(1, len(na) + 1))
        self.nc = list(na)
        self.nc[q - 1] = m
        dt = getattr(torch, dtype)
        self.A = torch.randn(int(np.prod(na)), device=cuda, dtype=dt)
        self.B = torch.randn(m, na[q - 1], device=cuda, dtype=dt)
        self.C = torch.zeros(int(np.prod(self.nc)), device=cuda, dtype=dt)

    def call(self):
        import torch
        _lib.ttm_raw(_lib.F32, _lib.PREC_PLAIN, self.q, len(self.na), self.A.data_ptr(), self.na,
                     ka.dense_strides(self.na, self.pia), self.pia, self.B.data_ptr(), [self.m, self.na[self.q - 1]], [2, 1],
                     self.C.data_ptr(), self.nc, ka.dense_strides(self.nc, self.pia),
                     torch.cuda.current_stream().cuda_stream)
        return _lib.last_kernel()

    def error(self):
        """Relative error of C (first-order layout: torch dims are the modes reversed)."""
        import torch
        p = len(self.na)
        A = self.A.double().view(*reversed(self.na))
        want = torch.movedim(torch.tensordot(A, self.B.double(), dims=([p - self.q], [1])), -1, p - self.q).reshape(-1)
        return float((self.C.double() - want).norm() / want.norm())


@pytest.mark.parametrize("na,q,m,other", [STRIDED, FIBRES])
def test_no_memory_for_the_parts(cuda, na, q, m, other):
    pr = Problem(cuda, na, q, m)
    assert pr.call() == "simt_gemm"
    pr.C.fill_(float("nan"))
    _lib.inject(_lib.INJECT_FAIL_ALLOC, 1)
    assert pr.call() == other and pr.error() <= 2e-6
    pr.C.fill_(float("nan"))
    assert pr.call() == "simt_gemm" and pr.error() <= 2e-6


def test_captured_call_holds_no_allocation(cuda):
    import torch
    na, q, m, other = STRIDED
    pr = Problem(cuda, na, q, m)
    pr.call()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        assert pr.call() == other
    pr.A.normal_()
    for _ in range(2):
        pr.C.fill_(float("nan"))
        g.replay()
        assert pr.error() <= 2e-6


@pytest.mark.parametrize("na,q,m,other", [STRIDED, FIBRES])
def test_plans_hold_their_own(cuda, na, q, m, other):
    from ttm_b200.plans import BatchPlan
    pr = Problem(cuda, na, q, m)

    def plan():
        return BatchPlan([dict(q=q, A=pr.A, B=pr.B, C=pr.C, na=na, pia=pr.pia, m=m)], precision="plain")

    p = plan()
    assert p.launches == 2
    _lib.inject(_lib.INJECT_FAIL_ALLOC, 1)   # at the first run: nothing is allocated there
    for run in (p.run, p.run_graph, p.run_graph):
        pr.C.fill_(float("nan"))
        run()
        assert pr.error() <= 2e-6
    p.close()
    _lib.inject(_lib.INJECT_FAIL_ALLOC, 1)   # when the plan is made: it goes on without
    p = plan()
    assert p.launches == (1 if other == "colvec" else 2)
    for run in (p.run, p.run_graph):
        pr.C.fill_(float("nan"))
        run()
        assert _lib.last_kernel() == other and pr.error() <= 2e-6
    p.close()
