"""Small m with a long l range: the slice-GEMM with its l range split over more blocks, at the edges
of its rule (rows, n_q, elements of A, m), against the oracle, deterministic."""
import numpy as np
import pytest

from ttm_b200 import _lib
from test_gpu_split import TOL, _check, _run

pytestmark = pytest.mark.gpu

F32, F64 = np.float32, np.float64


@pytest.mark.parametrize("dtype,na,pia,q,m,b_cm,taken", [
    # contiguous fibres the l-split kernels took: 2^21 elements, any m
    (F32, [2048, 1024], [1, 2], 1, 1, True, True), (F64, [2049, 1025], [1, 2], 1, 4, False, True),
    (F32, [2049, 1023], [1, 2], 1, 8, True, False),          # fewer elements
    (F32, [233017, 9], [1, 2], 1, 7, False, True), (F64, [262144, 8], [1, 2], 1, 7, False, False),
    (F32, [(1 << 18) + 2, 9], [1, 2], 1, 2, True, False),    # parts would be longer than 1024 l
    # below n_q = 2048: unsplit tiles from 16 row tiles on
    (F32, [1030, 2047], [1, 2], 1, 3, True, True), (F32, [1030, 1900], [1, 2], 1, 3, True, False),
    # strided rows: the l-split kernels' (n_q >= 16384) and the column kernel's
    (F64, [129, 16400], [1, 2], 2, 2, False, True), (F32, [3, 16400, 43], [1, 2, 3], 2, 5, True, True),
    (F64, [1025, 2051], [1, 2], 2, 1, True, True), (F64, [8193, 2051], [1, 2], 2, 4, True, False),
    (F32, [1025, 2051], [1, 2], 2, 9, False, True), (F32, [63, 2051, 17], [1, 2, 3], 2, 9, False, False),
    # 64 MB and more, which the TMA-fed kernel takes otherwise: few row tiles
    (F32, [4096, 4100], [1, 2], 2, 11, True, True), (F64, [4100, 2048], [1, 2], 1, 16, False, True),
    (F32, [4096, 4100], [1, 2], 2, 8, True, False), (F32, [32768, 512], [1, 2], 1, 5, True, True),
    (F32, [32768, 513], [1, 2], 1, 5, True, False), (F32, [9216, 2040], [1, 2], 2, 16, True, False)])
def test_split_small_m(cuda, oracle_c, dtype, na, pia, q, m, b_cm, taken):
    a, b, got, md, kern = _run(cuda, na, pia, q, m, b_cm, dtype)
    assert (kern == "simt_gemm") == taken, kern
    assert _check(oracle_c, q, a, b, got, md) <= TOL[dtype]
    _, _, again, _, _ = _run(cuda, na, pia, q, m, b_cm, dtype, a=a, b=b)
    assert np.array_equal(got, again)
