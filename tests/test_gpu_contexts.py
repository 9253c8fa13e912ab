"""The potential solve in a second CUDA context of the same process.

A kernel's allowance of more than 48 KB of shared memory belongs to the context it
was set in, so what the library remembers of a launch must too. Run in a process of
its own; forces in each context equal the first context's bit for bit.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import ctypes, sys
import numpy as np
import hyowon_b200 as hb
cuda = ctypes.CDLL("libcuda.so.1")
form, mesh = sys.argv[1], int(sys.argv[2])
pos = np.random.default_rng(1).uniform(0.0, 50.0, (3, 20000))

def forces():
    with hb.PMSolver(hb.MeshGeometry(50.0, mesh), hb.PMForceMethod.pure_pm(False), form) as s:
        s.upload(*pos, uniform_mass=1.0)
        s.solve_forces()
        d = s.download()
    return np.stack([d[k] for k in ("ax", "ay", "az")])

first = forces()
device, context = ctypes.c_int(), ctypes.c_void_p()
assert cuda.cuInit(0) == 0 and cuda.cuDeviceGet(ctypes.byref(device), 0) == 0
assert cuda.cuCtxCreate_v2(ctypes.byref(context), 0, device) == 0
second = forces()
assert cuda.cuCtxDestroy_v2(context) == 0
third = forces()
assert np.array_equal(first, second) and np.array_equal(first, third)
print("same")
"""


@pytest.mark.parametrize("form,mesh", [("fp64", 512), ("fp32", 512), ("fp64", 64)])
def test_solve_in_a_second_context(form, mesh):
    out = subprocess.run([sys.executable, "-c", SCRIPT, form, str(mesh)], cwd=ROOT,
                         capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    assert out.stdout.strip() == "same"
