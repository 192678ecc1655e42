"""The memory for the parts of a split l range comes from a pool of the library's own: the device's default
memory pool, which belongs to the process, keeps its settings."""
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
