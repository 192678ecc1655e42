"""The 8-bit tensor-core paths with C off a 16-byte boundary (a view into a larger buffer): contiguous
fibres, whose rows of outputs leave with 16-byte stores where they can, and rows of i. The outputs
equal those of the same call into an aligned C bit for bit, and nothing around C is written."""
import numpy as np
import pytest

import known_answer as ka
from ttm_b200 import _lib

pytestmark = pytest.mark.gpu


def _run(cuda, ta, tb, outer, nq, inner, m, prec, shift):
    import torch
    na, nc, pia = [inner, nq, outer], [inner, m, outer], [1, 2, 3]
    n = outer * m * inner
    tc = torch.full((n + shift + 64,), float("nan"), device=cuda, dtype=ta.dtype)
    es = tc.element_size()
    assert tc.data_ptr() % 16 == 0
    _lib.ttm_raw(_lib.F32 if es == 4 else _lib.F64, prec, 2, 3, ta.data_ptr(), na, ka.dense_strides(na, pia), pia,
                 tb.data_ptr(), [m, nq], [2, 1], tc.data_ptr() + es * shift, nc, ka.dense_strides(nc, pia),
                 torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    got = tc.cpu().numpy()
    assert np.isnan(got[:shift]).all() and np.isnan(got[shift + n:]).all()
    return got[shift:shift + n]


# m even and odd, below and past one and several chunks of 16 or 32 columns
@pytest.mark.parametrize("outer,nq,inner,m", [(130, 40, 1, 18), (130, 40, 1, 64), (129, 33, 1, 33), (257, 70, 1, 100),
                                              (3, 40, 44, 32)])
@pytest.mark.parametrize("path,shifts", [("ozaki", (1,)), ("fp8", (1, 2, 3))])
def test_outputs_do_not_depend_on_the_alignment_of_c(cuda, outer, nq, inner, m, path, shifts):
    import torch
    rng = np.random.default_rng(m)
    dt = np.float64 if path == "ozaki" else np.float32
    ta = torch.from_numpy(rng.standard_normal(outer * nq * inner).astype(dt)).to(cuda)
    tb = torch.from_numpy(rng.standard_normal(m * nq).astype(dt)).to(cuda)
    prec = _lib.PREC_OZAKI if path == "ozaki" else _lib.PREC_FP8
    want = _run(cuda, ta, tb, outer, nq, inner, m, prec, 0)
    assert _lib.last_kernel() == "tc_" + path
    assert np.isfinite(want).all()
    for shift in shifts:
        assert np.array_equal(_run(cuda, ta, tb, outer, nq, inner, m, prec, shift), want), shift
