"""A process that resets its device (CUDA.jl's ``device_reset!``) after destroying its contexts goes
on with new ones: what the library keeps per device - its memory pool, the kernels' attributes,
the address of the no-allocation scratch - belongs to the context that is gone and is made anew.

In a child process, so that no other test loses its context.  The results after the reset are
those before it, bit for bit (the same kernels on the same inputs, no atomics on values)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import ctypes, sys
sys.path.insert(0, "tests")
import conftest
import numpy as np
from pssfss_b200 import engine
from pssfss_b200.analyze import analyze
from pssfss_b200.elements import polyring, rectstrip
from pssfss_b200.layers import Layer
from pssfss_b200.rwg import setup_rwg, unique_face_pairs
from pssfss_b200.units import mm

ring = polyring(s1=[9, 0], s2=[0, 9], a=[3.15], b=[3.6], sides=24, ntri=500, units=mm)  # tabulated sums
patch = rectstrip(Lx=8, Ly=8, Px=10, Py=10, Nx=9, Ny=9, units=mm)
rng = np.random.default_rng(1)
Z = rng.standard_normal((300, 300)) + 20 * np.eye(300)

def everything():
    out = {}
    ufpm, rep, n = unique_face_pairs(patch, where="device")
    out.update(ufpm=ufpm, rep=rep)
    for name, sheet in (("ring", ring), ("patch", patch)):
        got = engine.face_integrals(sheet, setup_rwg(sheet), 0.35, 0.4, 0.2)
        out.update({name + k: np.asarray(v) for k, v in got.items()})
    for p in ("fp64", "fp32r"):
        out["x" + p] = engine.lu_solve(Z, np.ones((300, 5)), p)[0]
        out["s" + p] = np.stack([r.gsm.s11 for r in analyze([Layer(), patch, Layer()], [12.0], dict(zip("θϕ", (0, 0))),
                                                            precision=p)])
    return out

def finish():
    engine._sheets.clear()
    for c in engine._ctx.values():
        assert engine.lib().pss_ctx_destroy(c) == 0
    engine._ctx.clear()

first = everything()
finish()
cu = ctypes.CDLL("libcuda.so.1")
dev = ctypes.c_int()
assert cu.cuInit(0) == 0 and cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
assert cu.cuDevicePrimaryCtxReset_v2(dev) == 0
second = everything()
for k, v in first.items():
    assert np.array_equal(v, second[k]), k
finish()
print("same after reset")
"""


def test_new_contexts_after_a_device_reset():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same after reset" in r.stdout, r.stdout + r.stderr
