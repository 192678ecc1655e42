"""FP32 slice-GEMM with few rows and a long l range: tiles of 128 rows where 256 would mostly be padding.
The wide form must not be what runs there: its time on one row tile of 128 was 1.8 times the narrow one's,
so the l-split call of 128 rows may take at most 0.8 of the call of 256 rows (twice the work)."""
import pytest

from ttm_b200 import _lib

pytestmark = pytest.mark.gpu


def test_half_the_rows_take_less_time(cuda):
    import torch
    from ttm_b200 import ttmpy
    times = {}
    B = torch.randn(256, 1 << 17, device=cuda)
    for rows in (128, 256):
        A = torch.randn(rows, 1 << 17, device=cuda)
        C = ttmpy.ttm(2, A, B)
        assert _lib.last_kernel() == "simt_gemm"
        want = A[:2].double() @ B.double().t()
        assert float((C[:2].double() - want).norm() / want.norm()) <= 2e-6
        best = float("inf")
        for _ in range(5):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            for _ in range(5):
                ttmpy.ttm(2, A, B)
            e1.record()
            e1.synchronize()
            best = min(best, e0.elapsed_time(e1))
        times[rows] = best
    assert times[128] <= 0.8 * times[256], times
