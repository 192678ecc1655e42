"""The memory for the parts of a split l range comes from a pool of the library's own: the device's default
memory pool, which belongs to the process, keeps its settings; threads and streams share the pool, and
its memory can be given back between calls."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu


def test_default_memory_pool_keeps_its_threshold(cuda):
    code = """
import torch
from cuda.bindings import runtime as rt
from ttm_b200 import ttmpy, _lib
A, B = torch.randn(4000, 2047, device="cuda"), torch.randn(8, 4000, device="cuda")
ttmpy.ttm(1, A, B)
assert _lib.last_kernel() == "simt_gemm"
torch.cuda.synchronize()
pool = rt.cudaDeviceGetDefaultMemPool(0)[1]
keeps = rt.cudaMemPoolGetAttribute(pool, rt.cudaMemPoolAttr.cudaMemPoolAttrReleaseThreshold)[1]
assert int(keeps) == 0, keeps
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


def test_threads_and_streams_share_the_pool(cuda):
    import threading

    import torch
    from ttm_b200 import _lib, ttmpy
    g = torch.Generator(device=cuda).manual_seed(3)
    probs = []
    for n in range(4):
        A = torch.randn(4000 + n, 2047, device=cuda, generator=g)
        B = torch.randn(5 + n, 4000 + n, device=cuda, generator=g)
        probs.append((A, B, ttmpy.ttm(1, A, B).clone()))
    torch.cuda.synchronize()
    bad = []

    def work(A, B, want):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for n in range(30):
                C = ttmpy.ttm(1, A, B)
                if _lib.last_kernel() != "simt_gemm":
                    bad.append(_lib.last_kernel())
                if n % 10 == 9:
                    stream.synchronize()
                    if not torch.equal(C, want):
                        bad.append("wrong result")

    threads = [threading.Thread(target=work, args=pr) for pr in probs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
    _lib.lib().tlibttm_release_buffers()
    assert torch.equal(ttmpy.ttm(1, *probs[0][:2]), probs[0][2])
