"""Small m, float, contiguous fibres longer than 2^18 and off 16-byte boundaries: the l-split kernels keep
these problems (the slice-GEMM splits a range into at most 256 parts of 1024 l), on both sides of the
longest range that the split slice-GEMM takes. Bound: the repository's 2e-6 for plain float arithmetic."""
import pytest

import known_answer as ka
from ttm_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,nq,m,kernel", [(1921, (1 << 18) + 2, 3, "bvec"), (1921, (1 << 18) + 2, 9, "bvec"),
                                              (1921, (1 << 18) - 2, 3, "simt_gemm")])
def test_longest_ranges(cuda, rows, nq, m, kernel):
    import torch
    A = torch.randn(rows, nq, device=cuda)
    B = torch.randn(m, nq, device=cuda)
    C = torch.full((rows, m), float("nan"), device=cuda)
    na, nc, pia = [nq, rows], [m, rows], [1, 2]
    _lib.ttm_raw(_lib.F32, _lib.PREC_PLAIN, 1, 2, A.data_ptr(), na, ka.dense_strides(na, pia), pia, B.data_ptr(), [m, nq],
                 [2, 1], C.data_ptr(), nc, ka.dense_strides(nc, pia), torch.cuda.current_stream().cuda_stream)
    assert _lib.last_kernel() == kernel
    torch.cuda.synchronize()
    pick = [0, 1, 127, 128, 1000, rows - 1]
    want = A[pick].double() @ B.double().t()
    assert float((C[pick].double() - want).norm() / want.norm()) <= 2e-6
    assert torch.isfinite(C).all()
