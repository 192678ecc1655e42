"""The few-column and warp-per-rows kernels run on their side of each edge of their rules, and the kernels
they belong with on the other, for the default call; the tuner's schedules reach them too."""
import ctypes as C

import pytest

import known_answer as ka
from ttm_b200 import _lib

pytestmark = pytest.mark.gpu


def _call(cuda, outer, nq, inner, m, sched=None, shift=0, dtype="float32"):
    """The variant that ran C (outer, m, inner) = A x B, A `shift` elements into its allocation, and the
    result's relative error."""
    import torch
    from ttm_b200.selector import lib
    dt = getattr(torch, dtype)
    es, n = (4 if dtype == "float32" else 8), outer * nq * inner
    buf = torch.randn(n + shift, device=cuda, dtype=dt)
    B = torch.randn(m, nq, device=cuda, dtype=dt)
    out = torch.empty(outer, m, inner, device=cuda, dtype=dt)
    na, nc, pia = [inner, nq, outer], [inner, m, outer], [1, 2, 3]
    args = (2, 3, C.c_void_p(buf.data_ptr() + es * shift), _lib.sz(na), _lib.sz(ka.dense_strides(na, pia)), _lib.sz(pia),
            C.c_void_p(B.data_ptr()), _lib.sz([m, nq]), _lib.sz([2, 1]), C.c_void_p(out.data_ptr()), _lib.sz(nc),
            _lib.sz(ka.dense_strides(nc, pia)), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    dtype_id = _lib.F32 if dtype == "float32" else _lib.F64
    _lib.check(lib().tlibttm_ttm_ex(dtype_id, _lib.PREC_PLAIN, *args) if sched is None
               else lib().tlibttm_ttm_sched(dtype_id, sched, *args))
    variant = _lib.last_variant()
    want = torch.einsum("kli,jl->kji", buf[shift:].view(outer, nq, inner).double(), B.double())
    return variant, float((out.double() - want).norm() / want.norm())


# its rule: m <= 8, rows off 16-byte boundaries but A on one, 128 tiles of 256 rows, n_q >= 33 (17 at
# m = 1), tiles filled to 8/16 (m <= 4) or 9/16
@pytest.mark.parametrize("outer,nq,inner,m,shift,variant", [
    (64, 33, 301, 2, 0, "few_columns"), (64, 32, 301, 2, 0, "colvec"), (63, 33, 301, 2, 0, "colvec"),
    (64, 33, 300, 2, 0, "colvec"), (64, 33, 301, 2, 1, "colvec"), (64, 17, 301, 1, 0, "few_columns"),
    (64, 16, 301, 1, 0, "colvec"), (128, 35, 129, 4, 0, "few_columns"), (128, 35, 127, 4, 0, "colvec"),
    (64, 35, 289, 8, 0, "few_columns"), (64, 35, 287, 8, 0, "colvec"), (64, 35, 301, 9, 0, "colvec")])
def test_few_columns_rule(cuda, outer, nq, inner, m, shift, variant):
    got, err = _call(cuda, outer, nq, inner, m, shift=shift)
    assert got == variant and err <= 2e-6
    # the tuner's schedule with rows spread over warps takes it by the same rule, the l-split one never
    assert _call(cuda, outer, nq, inner, m, sched=2, shift=shift)[0] == variant
    assert _call(cuda, outer, nq, inner, m, sched=3, shift=shift)[0] == "colvec"


# its rule: float, m <= 8, fibres off 16-byte boundaries of 32 / 96 / 256 (m <= 2 / 4 / 8) to 1024
@pytest.mark.parametrize("nq,m,shift,variant", [
    (33, 1, 0, "rowwarp"), (31, 1, 0, "rowdot"), (32, 2, 1, "rowwarp"), (32, 2, 0, "rowdot"), (97, 3, 0, "rowwarp"),
    (95, 3, 0, "rowdot"), (257, 5, 0, "rowwarp"), (255, 5, 0, "rowdot"), (1023, 8, 0, "rowwarp"), (1025, 8, 0, "rowdot"),
    (257, 9, 0, "rowdot")])
def test_rowwarp_rule(cuda, nq, m, shift, variant):
    # (the schedule: the default call sends fibres from 1024 on to the l-split kernels)
    got, err = _call(cuda, 300, nq, 1, m, sched=4, shift=shift)
    assert got == variant and err <= 2e-6
    if nq < 1024:
        assert _call(cuda, 300, nq, 1, m, shift=shift)[0] == variant


def test_double_takes_neither(cuda):
    assert _call(cuda, 64, 33, 301, 2, dtype="float64")[0] == "colvec"
    assert _call(cuda, 300, 97, 1, 2, dtype="float64")[0] == "rowdot"
