"""The warp-per-rows kernel (float, m <= 8, contiguous fibres off 16-byte boundaries) against the C
oracle: every column bucket and the remainders of rows and l, both B layouts, and the edges of its
rule, where the other row kernels take over.

Bound: the repository's 2e-6 (relative Frobenius norm) for plain float arithmetic."""
import numpy as np
import pytest

import known_answer as ka
from ttm_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("m,nqs", [(1, (31, 32, 33, 65, 1023)), (2, (33, 130, 1025)), (3, (95, 97, 129)), (4, (96, 161)),
                                   (5, (255, 257)), (7, (258, 1022)), (8, (257, 511))])
def test_rowwarp_against_oracle(cuda, oracle_c, m, nqs, shift):
    import torch
    rng = np.random.default_rng(m)
    for nq in nqs:
        for rows, b_cm in ((1, False), (7, True), (33, False), (70003 if nq < 100 else 5003, True)):
            na, nc, pia = [nq, rows], [m, rows], [1, 2]
            wa, wc = ka.dense_strides(na, pia), ka.dense_strides(nc, pia)
            a = rng.standard_normal(nq * rows).astype(np.float32)
            b = rng.standard_normal(m * nq).astype(np.float32)
            ta = torch.empty(a.size + shift, device=cuda)
            ta[shift:] = torch.from_numpy(a).to(cuda)
            tb = torch.from_numpy(b).to(cuda)
            tc = torch.full((rows * m + 64,), float("nan"), device=cuda)
            _lib.ttm_raw(_lib.F32, _lib.PREC_PLAIN, 1, 2, ta.data_ptr() + 4 * shift, na, wa, pia, tb.data_ptr(), [m, nq],
                         [1, 2] if b_cm else [2, 1], tc.data_ptr(), nc, wc, torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            got = tc.cpu().numpy()
            assert np.isnan(got[rows * m:]).all()   # nothing past C
            ref = np.zeros(rows * m, dtype=np.float32)
            oracle_c.ttm(1, a, na, wa, pia, b, [m, nq], [1, 2] if b_cm else [2, 1], ref, nc, wc)
            c = got[:ref.size].astype(np.float64)
            assert np.linalg.norm(c - ref) / np.linalg.norm(ref) <= 2e-6, (nq, rows, m, _lib.last_kernel())
