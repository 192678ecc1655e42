"""The few-column kernel (m <= 8, rows of i off 16-byte boundaries) against the C oracle: every shift
of a line, partial tiles of rows, l below, at and past a stage, every column bucket, both B layouts,
and the rule's edges, where the column kernel takes over.

Bound: the repository's 2e-6 (relative Frobenius norm) for plain float arithmetic."""
import numpy as np
import pytest

import known_answer as ka
from ttm_b200 import _lib

pytestmark = pytest.mark.gpu
TOL = 2e-6


# (outer, n_q, inner): 128 tiles of 256 rows at least; inner 1, 2 and 3 mod 4 with n_q odd and even;
# then one value past the rule (tiles, fill, n_q, alignment of the rows)
@pytest.mark.parametrize("outer,nq,inner", [(64, 33, 301), (130, 34, 150), (50, 49, 767), (64, 48, 510), (128, 35, 255),
                                            (63, 33, 301), (130, 33, 127), (64, 32, 301), (64, 33, 300)])
@pytest.mark.parametrize("m,b_cm", [(1, False), (1, True), (2, False), (3, True), (4, False), (5, True), (7, False), (8, True)])
def test_few_columns_against_oracle(cuda, oracle_c, outer, nq, inner, m, b_cm):
    import torch
    rng = np.random.default_rng(outer + nq + inner + m)
    na, nc, pia = [inner, nq, outer], [inner, m, outer], [1, 2, 3]
    wa, wc = ka.dense_strides(na, pia), ka.dense_strides(nc, pia)
    a = rng.standard_normal(outer * nq * inner).astype(np.float32)
    b = rng.standard_normal(m * nq).astype(np.float32)
    ta, tb = torch.from_numpy(a).to(cuda), torch.from_numpy(b).to(cuda)
    tc = torch.full((outer * m * inner + 64,), float("nan"), device=cuda)
    _lib.ttm_raw(_lib.F32, _lib.PREC_PLAIN, 2, 3, ta.data_ptr(), na, wa, pia, tb.data_ptr(), [m, nq],
                 [1, 2] if b_cm else [2, 1], tc.data_ptr(), nc, wc, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert _lib.last_kernel() == "colvec"
    got = tc.cpu().numpy()
    assert np.isnan(got[outer * m * inner:]).all()   # nothing past C
    ref = np.zeros(outer * m * inner, dtype=np.float32)
    oracle_c.ttm(2, a, na, wa, pia, b, [m, nq], [1, 2] if b_cm else [2, 1], ref, nc, wc)
    c = got[:ref.size].astype(np.float64)
    assert np.linalg.norm(c - ref) / np.linalg.norm(ref) <= TOL


def test_infinities_stay_in_their_fibres(cuda):
    """Lines are copied past their ends only with zeros: a fibre of infinities leaves its neighbours finite."""
    import torch
    outer, nq, inner, m = 64, 37, 301, 3
    A = torch.randn(outer, nq, inner, device=cuda)
    A[5, :, 300] = float("inf")
    A[9, :, 0] = float("nan")
    B = torch.rand(m, nq, device=cuda) + 0.5
    C = torch.empty(outer, m, inner, device=cuda)
    na, nc, pia = [inner, nq, outer], [inner, m, outer], [1, 2, 3]
    _lib.ttm_raw(_lib.F32, _lib.PREC_PLAIN, 2, 3, A.data_ptr(), na, ka.dense_strides(na, pia), pia, B.data_ptr(), [m, nq],
                 [2, 1], C.data_ptr(), nc, ka.dense_strides(nc, pia), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    bad = ~torch.isfinite(C)
    assert bad[5, :, 300].all() and bad[9, :, 0].all() and int(bad.sum()) == 2 * m
