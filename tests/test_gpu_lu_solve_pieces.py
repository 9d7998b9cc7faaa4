"""``lu_solve`` brings the caller's matrix to the device in pieces of 64 MiB: orders at the edges of
a piece against the system itself, and the device memory that a large order takes."""
import os
import subprocess
import sys

import numpy as np
import pytest

from pssfss_b200 import engine

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("precision", ["fp64", "fp32r"])
@pytest.mark.parametrize("n", [2047, 2048, 2049, 2900])  # one piece; one, exactly full; two; three
def test_orders_at_the_edges_of_a_piece(n, precision):
    """Backward error as in the tests of the chained solves: at most n eps (a well-pivoted
    factorisation without growth; the refined form stops far below)."""
    rng = np.random.default_rng(n)
    Z = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    B = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    X, st = engine.lu_solve(Z, B, precision)
    assert st == 0
    back = np.max(np.abs(B - Z @ X), axis=0) / (np.max(np.sum(np.abs(Z), axis=1)) * np.max(np.abs(X), axis=0))
    assert np.max(back) <= n * 1.1102230246251565e-16


CHILD = """
import sys
sys.path.insert(0, "tests")
import conftest
import numpy as np, torch
from pssfss_b200 import engine
n = 4500
Z = np.asfortranarray(np.full((n, n), 0.25 + 0.5j) + 3 * n * np.eye(n))
b = np.ones((n, 1))
engine.lu_solve(Z[:300, :300], b[:300])  # kernels loaded, context made
free0 = torch.cuda.mem_get_info(0)[0]
engine.lu_solve(Z, b)
free1 = torch.cuda.mem_get_info(0)[0]
print("matrices taken", (free0 - free1) / (16 * n * n))
"""


def test_one_matrix_on_the_device():
    """A call holds the matrix once (its factors), workspaces of a few columns and a piece (a fifth
    of this matrix): less than half a matrix beyond the one."""
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert 1.0 <= float(r.stdout.split()[-1]) < 1.5, r.stdout
