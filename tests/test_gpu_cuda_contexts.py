"""Solver contexts in two CUDA contexts of one device: what is set on kernels belongs to the CUDA
context (as after a device reset), so the second one's launches above 48 KB need it set again."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from gatt_dns_b200 import case as cs
from gatt_dns_b200.solver import GattDNS

# the tensor-copy solver with the tensor-copy-fed assembly, the any-length solver (walls, 2-D and 3-D)
cases = [cs.periodic_box(nxyz=(128, 32, 32)), cs.lid_driven(nxy=(400, 96)), cs.cavity_channel(nx=120, ny=75, nz=9)]
flows = [cs.random_flow(c, seed=3, amp=0.02) for c in cases]

def all_of_it():
    out = []
    for c, f in zip(cases, flows):
        with GattDNS(c) as g:
            g.upload(f)
            g.apply_bound_cond()
            g.run(2, 0.0, 0.1 * c.cfl_dt(f["U"], f["V"], f["W"], 1.0))
            out.append(g.download())
    return out

first = all_of_it()
cuda = ctypes.CDLL("libcuda.so.1")
ctx, dev = ctypes.c_void_p(), ctypes.c_int()
assert cuda.cuInit(0) == 0 and cuda.cuDeviceGet(ctypes.byref(dev), 0) == 0
assert cuda.cuCtxCreate_v2(ctypes.byref(ctx), 0, dev) == 0  # now the current one
second = all_of_it()
assert cuda.cuCtxDestroy_v2(ctx) == 0
for a, b in zip(first, second):
    for k in a:
        assert np.array_equal(a[k], b[k]), k
"""


def test_second_cuda_context(cuda_lib):
    subprocess.run([sys.executable, "-c", CHILD, ROOT], check=True, timeout=300)
