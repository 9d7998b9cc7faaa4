"""A device with no memory left for the tables of the face integrals: the direct sums run, as they do
on sheets that take no tables.  In a process of its own, which fills the device."""
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
import numpy as np, torch
from pssfss_b200 import engine
from pssfss_b200.elements import rectstrip
from pssfss_b200.rwg import setup_rwg
from pssfss_b200.units import mm

# a long cell: 6800 panels, 49 MB of tables, more than a chunk of the library's pool may have left
strip = lambda: rectstrip(Lx=8, Ly=53, Px=10, Py=80, Nx=16, Ny=20, units=mm, fufp=False)
warm = strip()
wrwg = setup_rwg(warm)
ul = 0.5 * np.linalg.norm(warm.beta1)
want = engine.face_integrals(warm, wrwg, ul, 0.4, 0.2)  # tabulated; every kernel loaded
engine.face_integrals(warm, wrwg, 10 * ul, 0.4, 0.2)  # too many panels: direct
engine._sheets.clear()
engine.lib().pss_ctx_destroy(engine.context(0))
engine._ctx.clear()

sheet = strip()
rwg = setup_rwg(sheet)
engine.face_integrals(sheet, rwg, 10 * ul, 0.4, 0.2)  # holds the sheet and its integrals, no tables
engine.release_memory()
cu = ctypes.CDLL("libcuda.so.1")  # PyTorch's allocator rounds small requests up to 20 MB
free = lambda: torch.cuda.mem_get_info(0)[0]
fill = []
for unit in (1 << 30, 1 << 26, 1 << 22):
    while free() > unit + (4 << 20):
        p = ctypes.c_uint64()
        assert cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t((free() - (4 << 20)) // unit * unit)) == 0
        fill.append(p)
before = engine.lib().pss_kernel_launches()
got = engine.face_integrals(sheet, rwg, ul, 0.4, 0.2)
assert engine.lib().pss_kernel_launches() - before == 1
for k in ("J", "Jxi", "Jeta", "K", "Kxi", "Keta"):
    assert np.max(np.abs(got[k] - want[k])) <= 1e-13 * np.max(np.abs(want[k])), k
for p in fill:
    assert cu.cuMemFree_v2(p) == 0
before = engine.lib().pss_kernel_launches()
again = engine.face_integrals(sheet, rwg, ul, 0.4, 0.2)
assert engine.lib().pss_kernel_launches() - before == 4
assert all(np.array_equal(again[k], want[k]) for k in ("J", "K"))
print("done")
"""


def test_direct_sums_without_scratch():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr
