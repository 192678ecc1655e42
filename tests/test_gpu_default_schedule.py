"""tlibttm_default_schedule names what the planner's call runs: kernel for kernel, over small and large m,
rows of i and contiguous fibres, on and off 16-byte boundaries, short and long l ranges, both types."""
import ctypes as C

import numpy as np
import pytest

import known_answer as ka
from ttm_b200 import _lib

pytestmark = pytest.mark.gpu

# schedule -> the kernels that tlibttm_last_kernel may name for it
KERNELS = {1: {"simt_gemm"}, 2: {"colvec"}, 3: {"colvec"}, 4: {"rowdot"}, 5: {"tc_bf16x3"}, 6: {"stream_cols", "stream_rows"},
           7: {"tc_bf16x3_pair"}, 8: {"simt_gemm"}, 9: {"bvec"}}


def _views():
    rng = np.random.default_rng(7)
    out = []
    for _ in range(120):
        outer, nq, inner = (int(round(np.exp(rng.uniform(0, np.log(hi))))) for hi in (400, 3000, 600))
        inner = 1 if rng.random() < 0.35 else inner
        if rng.random() < 0.5:
            nq, inner = -(-nq // 4) * 4, inner if inner == 1 else -(-inner // 4) * 4
        m = int(round(np.exp(rng.uniform(0, np.log(300)))))
        if outer * nq * inner <= 1 << 25 and outer * m * inner <= 1 << 25:
            out.append((outer, nq, inner, m))
    out += [(1, 512, 70000, 8), (78000, 384, 1, 16), (2, 5000, 3, 40), (3000, 24, 96, 12), (401, 64, 509, 7), (9, 1 << 16, 1, 3)]
    return out


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("precision", ["plain", "auto"])
def test_default_schedule_is_what_runs(cuda, dtype, precision):
    import torch
    from ttm_b200.selector import lib
    dt, dtype_id, prec = getattr(torch, dtype), _lib.F32 if dtype == "float32" else _lib.F64, _lib.PRECISIONS[precision]
    L, seen = lib(), set()
    A, B, out = (torch.zeros(n, device=cuda, dtype=dt) for n in (1 << 26, 1 << 22, 1 << 26))
    for outer, nq, inner, m in _views():
        na, nc, pia = [inner, nq, outer], [inner, m, outer], [1, 2, 3]
        s = L.tlibttm_default_schedule(dtype_id, prec, 2, 3, _lib.sz(na), _lib.sz(pia), m)
        seen.add(s)
        args = (2, 3, C.c_void_p(A.data_ptr()), _lib.sz(na), _lib.sz(ka.dense_strides(na, pia)), _lib.sz(pia),
                C.c_void_p(B.data_ptr()), _lib.sz([m, nq]), _lib.sz([1, 2]), C.c_void_p(out.data_ptr()), _lib.sz(nc),
                _lib.sz(ka.dense_strides(nc, pia)), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        _lib.launch_count(reset=True)
        _lib.check(L.tlibttm_ttm_ex(dtype_id, prec, *args))
        kernel, variant, launches = _lib.last_kernel(), _lib.last_variant(), _lib.launch_count()
        if s == 0:
            assert kernel == "bvec" and m <= 16
            continue
        assert kernel in KERNELS[s], (outer, nq, inner, m, s, kernel)
        if m <= 16 and kernel == "simt_gemm":
            assert launches == (2 if s == 8 else 1)
        _lib.check(L.tlibttm_ttm_sched(dtype_id, s, *args))
        assert _lib.last_variant() == variant
    assert {1, 3, 4} <= seen
    torch.cuda.synchronize()


def test_invalid_arguments(cuda):
    from ttm_b200.selector import lib
    na, pia = _lib.sz([4, 5]), _lib.sz([1, 2])
    assert lib().tlibttm_default_schedule(_lib.F32, _lib.PREC_FP8, 1, 2, na, pia, 3) == -1
    assert lib().tlibttm_default_schedule(2, _lib.PREC_PLAIN, 1, 2, na, pia, 3) == -1
    assert lib().tlibttm_default_schedule(_lib.F32, _lib.PREC_PLAIN, 3, 2, na, pia, 3) == -1
    assert lib().tlibttm_default_schedule(_lib.F32, _lib.PREC_PLAIN, 1, 2, na, pia, 0) == -1
