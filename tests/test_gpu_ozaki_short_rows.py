"""The ozaki operand kernel on short rows (one to four chunks of 32 l, kept in registers) and one chunk
more, rows that fill no block, contiguous fibres on and off 16-byte boundaries: integers times a power of
two per fibre, whose product must match bit for bit."""
import numpy as np
import pytest

from test_gpu_ozaki_operand import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("nq", [1, 16, 17, 32, 33, 64, 65, 96, 97, 128, 129, 160])
@pytest.mark.parametrize("outer,inner", [(1, 29), (3, 43), (131, 1), (200, 1)])
def test_exact_on_scaled_integers(cuda, outer, nq, inner, shift):
    rng = np.random.default_rng(nq + outer)
    scale = 2.0 ** rng.integers(-40, 41, (outer, 1, inner))
    a = rng.integers(-1000, 1001, (outer, nq, inner)) * scale
    a[rng.random(a.shape) < 0.1] = -0.0
    a[0, :, 0] = 0.0
    a[outer - 1, :nq - 1, inner - 1] = 0.0   # the last element alone gives the exponent
    b = rng.integers(-1000, 1001, (20, nq)).astype(np.float64)
    want = np.einsum("kli,jl->kji", a / scale, b) * scale
    assert np.array_equal(_run(cuda, a, b, shift), want)
