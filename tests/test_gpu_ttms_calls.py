"""ttmpy.ttms as consecutive calls: the results of one ChainPlan of the same products, the errors of
its arguments, and metadata given as numpy integers."""
import numpy as np
import pytest

from ttm_b200 import _lib, ttmpy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("shape,q,ms,order", [((30, 20, 25), 1, (8, 20), "optimal"), ((7, 40, 9, 5), 3, (3, 33, 64), "backward"),
                                              ((1, 50, 3), 2, (2, 4), "forward"), ((64, 33), 2, (17,), "forward")])
def test_ttms_equals_a_chain_plan(cuda, dtype, shape, q, ms, order):
    import torch
    from ttm_b200.plans import ChainPlan
    dt = getattr(torch, dtype)
    p = len(shape)
    modes = [r for r in range(1, p + 1) if r != q]
    A = torch.randn(shape, device=cuda, dtype=dt)
    Bs = [torch.randn(m, shape[r - 1], device=cuda, dtype=dt) for r, m in zip(modes, ms)]
    got = ttmpy.ttms(q, A, Bs, order)
    seq = ttmpy._ttms_sequence(q, p, Bs, order)
    ext = list(shape)
    for r, k in seq:
        ext[r - 1] = int(Bs[k].shape[0])
    C = torch.empty(ext, device=cuda, dtype=dt)
    plan = ChainPlan(A, list(shape), list(range(p, 0, -1)), [r for r, _ in seq], [Bs[k] for _, k in seq], C)
    plan.run()
    torch.cuda.synchronize()
    plan.close()
    assert list(got.shape) == ext and got.is_contiguous()
    tol = 2e-6 if dtype == "float32" else 1e-13
    assert float((got.double() - C.double()).norm() / C.double().norm()) <= tol
    host = ttmpy.ttms(q, A.cpu().numpy(), [b.cpu().numpy() for b in Bs], order)
    assert isinstance(host, np.ndarray) and np.array_equal(host, got.cpu().numpy())


def test_ttms_refusals(cuda):
    import torch
    A = torch.randn(6, device=cuda)
    with pytest.raises(_lib.TtmError, match="the chain is empty"):
        ttmpy.ttms(1, A, [])
    A = torch.randn(6, 0, device=cuda)
    with pytest.raises(_lib.TtmError, match="^step 0: "):
        ttmpy.ttms(1, A, [torch.randn(3, 0, device=cuda)])
    A = torch.randn(40, 40, device=cuda)
    with pytest.raises(_lib.TtmError) as e:
        ttmpy.ttms(1, A, [torch.randn(20, 40, device=cuda)], precision="ozaki")
    assert e.value.code == _lib.ERR_UNSUPPORTED


def test_metadata_of_numpy_integers(cuda):
    import torch
    A = torch.randn(10, 12, device=cuda, dtype=torch.float64)
    B = torch.randn(5, 12, device=cuda, dtype=torch.float64)
    C = torch.empty(10, 5, device=cuda, dtype=torch.float64)
    na, nc = np.array([10, 12]), np.array([10, 5])
    _lib.ttm_raw(_lib.F64, _lib.PREC_PLAIN, 2, 2, A.data_ptr(), na, np.array([12, 1]), [2, 1], B.data_ptr(),
                 np.array([5, 12]), [2, 1], C.data_ptr(), nc, np.array([5, 1]),
                 torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert torch.allclose(C, A @ B.t())
