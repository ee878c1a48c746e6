"""The one-launch front: what a context's device can hold, and the plan from it.

GPU: a context does not lean on another context's set-up.  Its clusters of 16 blocks and its shared memory above 48 KB are attributes that
the kernels carry on one device.  A process that has stepped a small simulation
and then gets its device anew (cudaDeviceReset; a second GPU is the same to a
new context) steps the same simulations to the same bytes.

CPU: the plan for a table of resident clusters (B200's: 296 blocks one by one,
14 clusters of 16), and that sizes without a plan ask the device nothing.
"""
import ctypes
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import ctypes, importlib
import numpy as np
ge = importlib.import_module("galaxy-engine_b200")
ics = importlib.import_module("galaxy-engine_b200.ics")

def run(dims, n):
    st = ics.plummer3d(n, seed=1) if dims == 3 else ics.disk2d(n, seed=1)
    with ge.Simulation(ge.default_params(dims, G=1.0, theta=0.8, eps2=1e-4, dt=1e-3)) as s:
        s.upload(st)
        s.step(2)
        return s.download()

cases = [(2, 600), (2, 16384), (2, 32768), (3, 16384)]
first = [run(*c) for c in cases]
path = {l.split()[-1] for l in open("/proc/self/maps") if "libcudart" in l}.pop()
assert ctypes.CDLL(path).cudaDeviceReset() == 0
for c, a in zip(cases, first):
    b = run(*c)
    for k in a:
        assert np.array_equal(a[k], b[k]), (c, k)
print("same")
"""


class Limits(ctypes.Structure):
    _fields_ = [("known", ctypes.c_bool), ("fit", ctypes.c_int * 5)]


def _plan(ge, largest, sims, lim):
    f = ge.lib()._ZN2ge10front_planEillRNS_11FrontLimitsE
    f.argtypes = [ctypes.c_int, ctypes.c_int64, ctypes.c_int64, ctypes.POINTER(Limits)]
    v = f(2, largest, sims, ctypes.byref(lim))
    return v >> 8, v & 255


@pytest.mark.parametrize("largest,sims,blocks,items", [
    (1, 1, 1, 1), (512, 148, 1, 1), (513, 1, 2, 1), (2048, 35, 4, 1), (2048, 36, 2, 2),
    (2048, 148, 1, 4), (2048, 296, 1, 4), (2048, 297, 0, 0), (2049, 148, 2, 4),
    (8192, 7, 16, 1), (8192, 8, 8, 2), (8192, 17, 4, 4), (8192, 74, 4, 4), (8192, 75, 0, 0),
    (16384, 8, 8, 4), (16384, 37, 8, 4), (16384, 38, 0, 0), (16385, 14, 16, 4),
    (32768, 15, 16, 4), (32768, 16, 0, 0), (32769, 1, 0, 0)])
def test_plan(ge, largest, sims, blocks, items):
    lim = Limits(True, (ctypes.c_int * 5)(296, 148, 71, 33, 14))
    assert _plan(ge, largest, sims, lim) == (blocks, items)
    lim.fit[4] = 0   # a device without clusters of 16
    c, k = _plan(ge, largest, sims, lim)
    assert c < 16 and (c == 0 or c * 512 * k >= largest)


def test_no_plan_asks_nothing(ge):
    lim = Limits()
    assert _plan(ge, 32769, 1, lim) == (0, 0) and not lim.known


@pytest.mark.gpu
def test_a_new_device_context_is_set_up(tmp_path):
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("same"), r.stdout + r.stderr
