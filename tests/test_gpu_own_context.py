"""A program that makes its own CUDA context (driver API) and runs lattices in
it: large arrays go in and out as they do in the device's primary context."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = """
import ctypes
import numpy as np
import octlb_b200 as ob

n = 65  # populations of 41.7 MB, fields of 2.2 and 6.6 MB
mesh = ob.Mesh(n, [0], [0, 0, 0, 1, 1, 1], periodic=1)
pops = 1e-3 * np.random.default_rng(1).standard_normal((n ** 3, 19))
rho, u = 1.0 + pops[:, 0], pops[:, 1:4].copy()

def run():
    out = []
    with_pops = ob.GpuLattice(mesh, 1.0 / 0.6)
    with_pops.set_populations(pops)
    with_pops.advance(3)
    out += [with_pops.get_populations(), *with_pops.get_fields()]
    with_pops.set_equilibrium(rho, u)
    out.append(with_pops.get_populations())
    with_pops.close()
    return out

want = run()  # the primary context
cu = ctypes.CDLL("libcuda.so.1")
dev, ctx = ctypes.c_int(), ctypes.c_void_p()
assert cu.cuInit(0) == 0 and cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
assert cu.cuCtxCreate_v2(ctypes.byref(ctx), 0, dev) == 0
got = run()
now = ctypes.c_void_p()
assert cu.cuCtxGetCurrent(ctypes.byref(now)) == 0 and now.value == ctx.value
assert cu.cuCtxDestroy_v2(ctx) == 0
assert all(np.array_equal(a, b) for a, b in zip(want, got))
print("own context ok")
"""


def test_lattices_in_a_context_of_the_caller():
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "own context ok" in r.stdout, r.stdout + r.stderr
