"""The FP64 slice-GEMM on the matrix instruction (gemm_f64.cuh) against the C oracle: every column
width, partial tiles of rows, columns and l, each form of A (contiguous fibres, rows of i; 16-byte
and 8-byte copies) and of B, the split l range, and the small-m problems that take it.

Bound: the repository's 1e-13 (relative Frobenius norm) for plain double arithmetic."""
import numpy as np
import pytest

import known_answer as ka
from ttm_b200 import _lib

pytestmark = pytest.mark.gpu
TOL = 1e-13


def _run(cuda, oracle_c, outer, nq, inner, m, b_cm, shift=0, sched=None):
    """Relative error of C (outer, m, inner) and the kernel; A and C start `shift` elements into
    their allocations."""
    import torch
    from ttm_b200.selector import lib
    rng = np.random.default_rng(outer + 3 * nq + 5 * inner + 7 * m)
    na, nc, pia = [inner, nq, outer], [inner, m, outer], [1, 2, 3]
    wa, wc = ka.dense_strides(na, pia), ka.dense_strides(nc, pia)
    a, b = rng.standard_normal(outer * nq * inner), rng.standard_normal(m * nq)
    ta = torch.empty(a.size + shift, dtype=torch.float64, device=cuda)
    ta[shift:] = torch.from_numpy(a).to(cuda)
    tb = torch.from_numpy(b).to(cuda)
    tc = torch.full((outer * m * inner + shift + 64,), float("nan"), dtype=torch.float64, device=cuda)
    args = (2, 3, ta.data_ptr() + 8 * shift, _lib.sz(na), _lib.sz(wa), _lib.sz(pia), tb.data_ptr(), _lib.sz([m, nq]),
            _lib.sz([1, 2] if b_cm else [2, 1]), tc.data_ptr() + 8 * shift, _lib.sz(nc), _lib.sz(wc), None)
    _lib.check(lib().tlibttm_ttm_ex(_lib.F64, _lib.PREC_PLAIN, *args) if sched is None
               else lib().tlibttm_ttm_sched(_lib.F64, sched, *args))
    kernel = _lib.last_kernel()
    torch.cuda.synchronize()
    got = tc.cpu().numpy()
    assert np.isnan(got[:shift]).all() and np.isnan(got[shift + outer * m * inner:]).all()   # nothing past C
    ref = np.zeros(outer * m * inner)
    oracle_c.ttm(2, a, na, wa, pia, b, [m, nq], [1, 2] if b_cm else [2, 1], ref, nc, wc)
    c = got[shift:shift + ref.size]
    return np.linalg.norm(c - ref) / np.linalg.norm(ref), kernel


@pytest.mark.parametrize("b_cm", [False, True])
@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 31, 33, 48, 56, 64, 65, 100, 130])
def test_widths_and_forms(cuda, oracle_c, m, b_cm):
    # rows: one partial tile, a tile and a row, odd and even extents; l: below, at and past a stage
    for outer, nq, inner in ((5, 15, 26), (3, 17, 43), (129, 16, 1), (65, 33, 1), (2, 1, 64), (1, 50, 129)):
        err, kernel = _run(cuda, oracle_c, outer, nq, inner, m, b_cm, sched=1)
        assert kernel == "simt_gemm" and err <= TOL, (outer, nq, inner, m, err)


@pytest.mark.parametrize("m", [40, 64, 72])
def test_wide_tiles_that_fill_the_gpu(cuda, oracle_c, m):
    # enough rows for the 64-column tiles; n_q = 16: a fixed set of blocks walks the tiles
    for outer, nq, inner in ((1, 16, 40000), (313, 20, 130), (39999, 18, 1)):
        err, kernel = _run(cuda, oracle_c, outer, nq, inner, m, False)
        assert kernel == "simt_gemm" and err <= TOL, (outer, nq, inner, m, err)


@pytest.mark.parametrize("shift", [0, 1])
def test_operands_off_16_byte_boundaries(cuda, oracle_c, shift):
    for outer, nq, inner, m in ((7, 40, 66, 20), (300, 40, 1, 24)):
        err, _ = _run(cuda, oracle_c, outer, nq, inner, m, True, shift=shift)
        assert err <= TOL, (outer, nq, inner, m, err)


def test_split_l_range_takes_the_tile(cuda, oracle_c):
    for outer, nq, inner, m in ((1, 4100, 70, 12), (90, 4096, 1, 80)):
        err, kernel = _run(cuda, oracle_c, outer, nq, inner, m, False, sched=8)
        assert kernel == "simt_gemm" and err <= TOL, (outer, nq, inner, m, err)


@pytest.mark.parametrize("outer,nq,inner,m,taken", [
    (2100, 12, 16, 9, True), (2100, 11, 16, 9, False), (300, 17, 1, 16, True), (300, 16, 1, 16, False),
    (101, 32, 21, 12, True), (101, 31, 21, 12, False), (40, 128, 410, 5, True), (40, 127, 410, 8, False),
    (40, 128, 411, 3, True), (40, 128, 410, 4, False), (100, 128, 1, 2, True), (100, 127, 1, 8, False),
    (2047, 1024, 1, 9, True), (1920, 1024, 1, 9, False)])
def test_small_m_rule(cuda, oracle_c, outer, nq, inner, m, taken):
    err, kernel = _run(cuda, oracle_c, outer, nq, inner, m, False)
    assert (kernel == "simt_gemm") == taken, kernel
    assert err <= TOL, err
