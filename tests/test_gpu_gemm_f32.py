"""The FP32 slice-GEMM on packed FFMA (gemm_f32.cuh) against the C oracle: every column width of the
wide and narrow tiles, partial tiles of rows, columns and l, each form of A (contiguous fibres, rows
of i; 16-byte and 4-byte copies) and of B, the split l range, the grouped launch of batched plans,
and the small-m problems that take it.

Bound: the repository's 2e-6 (relative Frobenius norm) for plain float arithmetic."""
import numpy as np
import pytest

import known_answer as ka
from ttm_b200 import _lib

pytestmark = pytest.mark.gpu
TOL = 2e-6


def _run(cuda, oracle_c, outer, nq, inner, m, b_cm, shift=0, sched=None):
    """Relative error of C (outer, m, inner) and the kernel; A and C start `shift` elements into
    their allocations."""
    import torch
    from ttm_b200.selector import lib
    rng = np.random.default_rng(outer + 3 * nq + 5 * inner + 7 * m)
    na, nc, pia = [inner, nq, outer], [inner, m, outer], [1, 2, 3]
    wa, wc = ka.dense_strides(na, pia), ka.dense_strides(nc, pia)
    a = rng.standard_normal(outer * nq * inner).astype(np.float32)
    b = rng.standard_normal(m * nq).astype(np.float32)
    ta = torch.empty(a.size + shift, device=cuda)
    ta[shift:] = torch.from_numpy(a).to(cuda)
    tb = torch.from_numpy(b).to(cuda)
    tc = torch.full((outer * m * inner + shift + 64,), float("nan"), device=cuda)
    args = (2, 3, ta.data_ptr() + 4 * shift, _lib.sz(na), _lib.sz(wa), _lib.sz(pia), tb.data_ptr(), _lib.sz([m, nq]),
            _lib.sz([1, 2] if b_cm else [2, 1]), tc.data_ptr() + 4 * shift, _lib.sz(nc), _lib.sz(wc), None)
    _lib.check(lib().tlibttm_ttm_ex(_lib.F32, _lib.PREC_PLAIN, *args) if sched is None
               else lib().tlibttm_ttm_sched(_lib.F32, sched, *args))
    kernel = _lib.last_kernel()
    torch.cuda.synchronize()
    got = tc.cpu().numpy()
    assert np.isnan(got[:shift]).all() and np.isnan(got[shift + outer * m * inner:]).all()   # nothing past C
    ref = np.zeros(outer * m * inner, dtype=np.float32)
    oracle_c.ttm(2, a, na, wa, pia, b, [m, nq], [1, 2] if b_cm else [2, 1], ref, nc, wc)
    c = got[shift:shift + ref.size].astype(np.float64)
    return np.linalg.norm(c - ref) / np.linalg.norm(ref), kernel


@pytest.mark.parametrize("b_cm", [False, True])
@pytest.mark.parametrize("m", [1, 5, 9, 13, 17, 21, 25, 29, 32, 33, 70])
def test_narrow_widths_and_forms(cuda, oracle_c, m, b_cm):
    # rows: one partial tile, a tile and a row, odd and even extents; l: below, at and past a stage
    for outer, nq, inner in ((5, 15, 28), (3, 17, 43), (129, 16, 1), (65, 33, 1), (2, 1, 64), (1, 50, 129)):
        err, kernel = _run(cuda, oracle_c, outer, nq, inner, m, b_cm, sched=1)
        assert kernel == "simt_gemm" and err <= TOL, (outer, nq, inner, m, err)


@pytest.mark.parametrize("m", [12, 20, 32])
def test_narrow_tiles_of_256_rows(cuda, oracle_c, m):
    # at least four tiles per SM; rows of i with 4-byte copies take two parts per thread
    for outer, nq, inner in ((401, 19, 381), (300, 18, 512), (152001, 20, 1), (152001, 21, 1), (1520, 16, 100)):
        err, kernel = _run(cuda, oracle_c, outer, nq, inner, m, False, sched=1)
        assert kernel == "simt_gemm" and err <= TOL, (outer, nq, inner, m, err)


@pytest.mark.parametrize("m", [33, 48, 56, 64, 100])
def test_wide_tiles_that_fill_the_gpu(cuda, oracle_c, m):
    for outer, nq, inner, b_cm in ((1, 16, 76000, True), (251, 35, 304, False), (253, 20, 301, True),
                                   (76001, 20, 1, False), (76001, 33, 1, True)):
        err, kernel = _run(cuda, oracle_c, outer, nq, inner, m, b_cm)
        assert kernel == "simt_gemm" and err <= TOL, (outer, nq, inner, m, err)


@pytest.mark.parametrize("shift", [0, 1, 2])
def test_operands_off_16_byte_boundaries(cuda, oracle_c, shift):
    for outer, nq, inner, m in ((7, 40, 68, 20), (300, 40, 1, 24)):
        err, _ = _run(cuda, oracle_c, outer, nq, inner, m, True, shift=shift)
        assert err <= TOL, (outer, nq, inner, m, err)


def test_split_l_range_takes_the_tile(cuda, oracle_c):
    for outer, nq, inner, m in ((1, 4100, 70, 12), (90, 4096, 1, 80)):
        err, kernel = _run(cuda, oracle_c, outer, nq, inner, m, False, sched=8)
        assert kernel == "simt_gemm" and err <= TOL, (outer, nq, inner, m, err)


@pytest.mark.parametrize("outer,nq,inner,m,taken", [
    (64, 64, 64, 9, True), (64, 63, 64, 9, False), (64, 64, 63, 12, False), (63, 64, 65, 16, True),
    (40, 64, 64, 16, False), (64, 64, 64, 8, False), (300, 64, 1, 9, True), (300, 60, 1, 9, False),
    (300, 513, 1, 10, True), (300, 511, 1, 10, False), (2047, 1024, 1, 9, True), (1920, 1024, 1, 9, False)])
def test_small_m_rule(cuda, oracle_c, outer, nq, inner, m, taken):
    err, kernel = _run(cuda, oracle_c, outer, nq, inner, m, False)
    assert (kernel == "simt_gemm") == taken, kernel
    assert err <= TOL, err


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_grouped_widths(cuda, oracle_c, dtype):
    """The grouped slice-GEMM of a plain batched plan: each of its column widths, two column tiles,
    each form of A and B."""
    import torch
    from ttm_b200.plans import BatchPlan
    rng = np.random.default_rng(5)
    probs = []
    for n, m in enumerate((17, 30, 40, 48, 50, 64, 65, 97, 130)):
        for na, pia, q in (([36, 20, 7], [1, 2, 3], 2), ([35, 19, 7], [1, 2, 3], 2), ([20, 150], [1, 2], 1),
                           ([19, 131], [1, 2], 1)):
            a = rng.standard_normal(int(np.prod(na))).astype(dtype)
            b = rng.standard_normal(m * na[q - 1]).astype(dtype)
            nc = list(na)
            nc[q - 1] = m
            probs.append(dict(q=q, na=na, pia=pia, m=m, nc=nc, a=a, b=b, b_cm=bool(n % 2),
                              A=torch.from_numpy(a).to(cuda), B=torch.from_numpy(b).to(cuda),
                              C=torch.full((int(np.prod(nc)),), float("nan"), device=cuda,
                                           dtype=torch.float32 if dtype == np.float32 else torch.float64)))
    plan = BatchPlan(probs, precision="plain")
    assert plan.launches == 1
    plan.run()
    torch.cuda.synchronize()
    for p in probs:
        ref = np.zeros(int(np.prod(p["nc"])), dtype=dtype)
        oracle_c.ttm(p["q"], p["a"], p["na"], ka.dense_strides(p["na"], p["pia"]), p["pia"], p["b"],
                     [p["m"], p["na"][p["q"] - 1]], [1, 2] if p["b_cm"] else [2, 1], ref, p["nc"],
                     ka.dense_strides(p["nc"], p["pia"]))
        c = p["C"].cpu().numpy()
        err = np.linalg.norm(c - ref) / np.linalg.norm(ref)
        assert err <= (TOL if dtype == np.float32 else 1e-13), (p["na"], p["m"], err)
    plan.close()
