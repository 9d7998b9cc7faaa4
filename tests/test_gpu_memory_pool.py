"""The library's device memory pool: what it keeps is given back on request and when a context is
destroyed, and makes way when the library's own next allocation would fail; an allocation that
fails all the same is reported and leaves the context usable.  Each in a process of its own, whose
device memory nothing else moves."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = """
import sys
sys.path.insert(0, "tests")
import conftest
import numpy as np, torch
from pssfss_b200 import engine
from pssfss_b200.elements import rectstrip
from pssfss_b200.rwg import unique_face_pairs
from pssfss_b200.units import mm

MIB = 1 << 20
free = lambda: torch.cuda.mem_get_info(0)[0]
small = rectstrip(Lx=4, Ly=4, Px=10, Py=10, Nx=4, Ny=4, units=mm)
large = rectstrip(Lx=8, Ly=8, Px=10, Py=10, Nx=32, Ny=32, units=mm)  # 2048 faces: some 300 MB to class
Z = np.eye(300) * (2 + 1j)
solve = lambda: engine.lu_solve(Z, np.ones((300, 1)))[0]
unique_face_pairs(small, where="device")
want = solve()
engine.lib().pss_ctx_destroy(engine.context(0))
engine._ctx.clear()
solve()
unique_face_pairs(small, where="device")
torch.cuda.synchronize()
"""

GIVEN_BACK = HEAD + """
engine.release_memory()
before = free()
unique_face_pairs(large, where="device")
kept = before - free()
engine.release_memory()
after = before - free()
print("kept", kept / MIB, "after", after / MIB)
assert kept > 200 * MIB and after < 8 * MIB
unique_face_pairs(large, where="device")
engine.lib().pss_ctx_destroy(engine.context(0))
engine._ctx.clear()
assert before - free() < 8 * MIB
assert np.array_equal(solve(), want)
print("done")
"""

MAKES_WAY = HEAD + """
unique_face_pairs(large, where="device")  # leaves some 300 MB with the pool
rest = torch.empty(free() - 256 * MIB, dtype=torch.uint8, device="cuda:0")
n = 4800  # 369 MB: more than what is free, less than that and the pool's share
X, st = engine.lu_solve(np.asfortranarray(np.eye(n) * (2 + 1j)), np.ones((n, 1)))
assert st == 0 and np.allclose(X, 1 / (2 + 1j), rtol=1e-15, atol=0)
try:
    engine.lu_solve(np.asfortranarray(np.eye(8000, dtype=complex)), np.ones((8000, 1)))  # 1 GB
except RuntimeError as e:
    assert "device allocation of" in str(e), e
else:
    raise AssertionError("an allocation beyond the device's memory succeeded")
assert np.array_equal(solve(), want)
print("done")
"""


BOUNDED = HEAD + """
engine.release_memory()
before = free()
big = rectstrip(Lx=8, Ly=8, Px=10, Py=10, Nx=56, Ny=56, units=mm)  # 6272 faces: 4.5 GB to class
for _ in range(3):
    unique_face_pairs(big, where="device")
    kept = before - free()
    print("kept", kept / MIB)
    assert 1024 * MIB < kept <= 2048 * MIB + 64 * MIB  # the excess goes, the rest stays
print("done")
"""


@pytest.mark.parametrize("child", [GIVEN_BACK, MAKES_WAY, BOUNDED], ids=["given_back", "makes_way", "bounded"])
def test_pool(child):
    r = subprocess.run([sys.executable, "-c", child], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr
