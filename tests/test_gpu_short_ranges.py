"""Slice-GEMM tiles of contiguous fibres and rows of i on short l ranges: a last stage of at most 8 l (half
a stage, multiplied alone where fibres are short), of 9 and of 16, and the range where the half stages
end, with one and several column tiles. Integer data, exact in float: bit for bit."""
import numpy as np
import pytest

import known_answer as ka
from ttm_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("m,b_cm", [(17, True), (40, False), (64, True), (99, False), (130, True)])
@pytest.mark.parametrize("rows,inner", [(76001, 1), (1, 76001), (19, 4000)])
def test_short_ranges_are_exact(cuda, dtype, m, b_cm, rows, inner):
    import torch
    dt = getattr(torch, dtype)
    g = torch.Generator(device=cuda).manual_seed(m)
    for nq in (1, 7, 8, 9, 16, 17, 24, 25, 40, 57, 64, 65, 72):
        A = torch.randint(-50, 51, (rows, nq, inner), device=cuda, generator=g).to(dt)
        B = torch.randint(-50, 51, (m, nq), device=cuda, generator=g).to(dt)
        out = torch.full((rows, m, inner), float("nan"), device=cuda, dtype=dt)
        b = B.t().contiguous() if b_cm else B
        na, nc, pia = [inner, nq, rows], [inner, m, rows], [1, 2, 3]
        _lib.ttm_raw(_lib.F32 if dtype == "float32" else _lib.F64, _lib.PREC_PLAIN, 2, 3, A.data_ptr(), na,
                     ka.dense_strides(na, pia), pia, b.data_ptr(), [m, nq], [1, 2] if b_cm else [2, 1], out.data_ptr(), nc,
                     ka.dense_strides(nc, pia), torch.cuda.current_stream().cuda_stream)
        assert _lib.last_kernel() == "simt_gemm"
        want = torch.einsum("kli,jl->kji", A.double(), B.double())
        assert torch.equal(out.double(), want), (nq, np.abs((out.double() - want).cpu().numpy()).max())


def test_wide_results_of_short_fibres_leave_in_whole_lines(cuda):
    """128000 fibres of 8, m = 512: the result's 262 MB are all there is. A warp's stores that cover eight rows
    by half a line took 115 us, whole lines 73; a copy of as many bytes takes about 80. At most 1.25 copies."""
    import torch
    from ttm_b200 import ttmpy
    A, B = torch.randn(128000, 8, device=cuda), torch.randn(512, 8, device=cuda)
    src, dst = (torch.empty(128000 * 512, device=cuda) for _ in range(2))

    def best(call):
        times = []
        for _ in range(6):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            for _ in range(10):
                call()
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1))
        return min(times)

    assert best(lambda: ttmpy.ttm(2, A, B)) <= 1.25 * best(lambda: dst.copy_(src))
