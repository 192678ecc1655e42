"""How far off small-m sums may be: the slice-GEMM tiles and the few-column kernel add up in short
chains, as the kernels they replace do, so that the error does not grow with one chain of n_q.

Model of the bound: a sum of n terms in order makes, at step k, a rounding error of at most half an ulp
of a partial sum that carries k / n of the total's variance. In units of the variance of one rounding of
the total, a chain of n is (n + 1) / 2, and a sum of sums adds the levels. One rounding is at most
2^-24 / sqrt(3) (2^-53 in double) of the value in the root mean square; the bound is that times the root
of the units."""
import numpy as np
import pytest

import known_answer as ka
from ttm_b200 import _lib

pytestmark = pytest.mark.gpu


def _chain(n):
    return (n + 1) / 2


def _tile_units(nq, chain=8, kept=True):
    """Chains, their sums over 128 l, and the sums of those (whose roundings are kept, or one chain more),
    and the result's own rounding twice (parts of a split range, the result)."""
    units = _chain(min(nq, chain)) + _chain(-(-min(nq, 128) // chain)) + 2
    return units if kept else units + _chain(-(-nq // 128))


def _few_units(nq):
    """Four warps take every fourth l, in chains of 8, or 16 from n_q = 128 on."""
    own, chain = -(-nq // 4), 8 if nq < 128 else 16
    return _chain(min(own, chain)) + _chain(-(-own // chain)) + _chain(4) + 1


def _error(cuda, dt, outer, nq, inner, m, b_cm):
    """Relative Frobenius error against long double (float: double) and the kernel."""
    import torch
    rng = np.random.default_rng(outer + nq + inner + m)
    a = rng.standard_normal((outer, nq, inner)).astype(dt)
    b = rng.standard_normal((m, nq)).astype(dt)
    na, nc, pia = [inner, nq, outer], [inner, m, outer], [1, 2, 3]
    ta, tb = torch.from_numpy(a).to(cuda), torch.from_numpy(np.ascontiguousarray(b.T) if b_cm else b).to(cuda)
    tc = torch.empty((outer, m, inner), device=cuda, dtype=ta.dtype)
    _lib.ttm_raw(_lib.F32 if dt == np.float32 else _lib.F64, _lib.PREC_PLAIN, 2, 3, ta.data_ptr(), na,
                 ka.dense_strides(na, pia), pia, tb.data_ptr(), [m, nq], [1, 2] if b_cm else [2, 1], tc.data_ptr(), nc,
                 ka.dense_strides(nc, pia), torch.cuda.current_stream().cuda_stream)
    kernel = _lib.last_kernel()
    torch.cuda.synchronize()
    wide = np.float64 if dt == np.float32 else np.longdouble
    want = np.tensordot(b.astype(wide), a.astype(wide), axes=([1], [1])).transpose(1, 0, 2)
    return float(np.sqrt(((tc.cpu().numpy().astype(wide) - want) ** 2).sum() / (want ** 2).sum())), kernel


# unsplit and split ranges, rows of i and contiguous fibres, on and off 16-byte boundaries, one to four
# groups of columns; problems that the column, row, TMA-fed or l-split kernels took before
@pytest.mark.parametrize("outer,nq,inner,m,b_cm", [
    (64, 64, 64, 9, True), (64, 200, 65, 16, False), (40, 1000, 130, 12, True), (300, 64, 1, 9, True),
    (2000, 1030, 1, 1, False), (2047, 1030, 1, 3, True), (2048, 4096, 1, 8, False), (1500, 9001, 1, 5, True),
    (1, 8191, 400, 13, False), (1, 2051, 1025, 9, True), (2, 7999, 20000, 10, False)])
def test_float_tiles(cuda, outer, nq, inner, m, b_cm):
    err, kernel = _error(cuda, np.float32, outer, nq, inner, m, b_cm)
    assert kernel == "simt_gemm"
    assert err <= 2.0 ** -24 * (_tile_units(nq) / 3) ** 0.5


@pytest.mark.parametrize("outer,nq,inner,m", [(64, 33, 301, 8), (64, 100, 301, 1), (130, 400, 150, 4), (50, 801, 767, 7)])
def test_few_columns(cuda, outer, nq, inner, m):
    err, kernel = _error(cuda, np.float32, outer, nq, inner, m, False)
    assert kernel == "colvec"
    assert err <= 2.0 ** -24 * (_few_units(nq) / 3) ** 0.5


@pytest.mark.parametrize("outer,nq,inner,m,b_cm", [
    (60, 60, 64, 9, True), (64, 200, 65, 16, False), (3000, 24, 96, 12, True),
    (2049, 1025, 1, 4, False), (1, 2051, 1025, 1, True), (1025, 4096, 1, 12, False)])
def test_double_tiles(cuda, outer, nq, inner, m, b_cm):
    err, kernel = _error(cuda, np.float64, outer, nq, inner, m, b_cm)
    assert kernel == "simt_gemm"
    units = _tile_units(nq, 16) if inner == 1 else _tile_units(nq, 8 if nq < 160 else 16, kept=False)
    assert err <= 2.0 ** -53 * (units / 3) ** 0.5


# problems that the row kernels and the TMA-fed kernel took with one chain of n_q per output
@pytest.mark.parametrize("dt,outer,nq,inner,m,b_cm", [
    (np.float32, 160000, 64, 1, 12, True), (np.float32, 100, 128, 2048, 16, False), (np.float64, 300, 384, 1, 16, False),
    (np.float64, 300, 250, 1, 8, True), (np.float64, 100, 128, 1024, 9, False)])
def test_no_further_off_than_one_chain(cuda, dt, outer, nq, inner, m, b_cm):
    err, kernel = _error(cuda, dt, outer, nq, inner, m, b_cm)
    assert kernel == "simt_gemm"
    assert err <= (2.0 ** -24 if dt == np.float32 else 2.0 ** -53) * ((_chain(nq) + 1) / 3) ** 0.5


# m > 64 with a long l range and few tiles: parts of nq / S, S two blocks per SM over the tiles of 128 x 128
# (and parts of 1024 l at least)
@pytest.mark.parametrize("outer,nq,inner,m,parts", [(9600, 4096, 1, 100, 4), (1, 9000, 9500, 70, 4), (1000, 30000, 1, 256, 19)])
def test_split_parts(cuda, outer, nq, inner, m, parts):
    err, kernel = _error(cuda, np.float32, outer, nq, inner, m, False)
    assert kernel == "simt_gemm"
    assert err <= 2.0 ** -24 * ((_chain(-(-nq // parts) + 16) + 2) / 3) ** 0.5
