"""What a call copies from pageable host memory has reached the device before a kernel of another
stream reads it: the same inputs, copied anew for every call, give the same results bit for bit
(no kernel adds in a varying order).  A factorisation that began before the end of its matrix had
arrived gave other factors in one call of 24 at order 736."""
import numpy as np
import pytest

from pssfss_b200 import engine
from pssfss_b200.elements import rectstrip
from pssfss_b200.rwg import setup_rwg
from pssfss_b200.units import mm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,calls", [(200, 100), (736, 200), (1100, 60)])
def test_fp32_factors_repeat(n, calls):
    rng = np.random.default_rng(n)
    Z = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + np.sqrt(n) * np.eye(n)
    other = np.asfortranarray(Z.T * 1.5)
    LU, ipiv, info = engine.lu32_factor(Z)
    for _ in range(calls):
        engine.lu32_factor(other)  # another matrix in the same buffers
        again = engine.lu32_factor(Z)
        assert again[2] == info and np.array_equal(again[1], ipiv)
        assert np.array_equal(again[0], LU)


@pytest.mark.parametrize("precision", ["fp64", "fp32r"])
def test_solutions_repeat(precision):
    n = 736
    rng = np.random.default_rng(n)
    Z = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + np.sqrt(n) * np.eye(n)
    B = rng.standard_normal((n, 3)) + 0j
    X, _ = engine.lu_solve(Z, B, precision)
    for _ in range(60):
        engine.lu_solve(Z.T * 1.5, B, precision)
        assert np.array_equal(engine.lu_solve(Z, B, precision)[0], X)


def test_fresh_uploads_repeat():
    sheet = rectstrip(Lx=8, Ly=8, Px=10, Py=10, Nx=12, Ny=12, units=mm)
    first = None
    for k in range(60):
        rwg = setup_rwg(sheet)  # a new object: uploaded anew
        F = engine.basis_transforms(sheet, rwg, [[12.0, 30.0], [0.0, 400.0]], 0.4, -0.2)
        J = engine.face_integrals(sheet, rwg, 0.3, 0.4, -0.2)["J"]
        if first is None:
            first = F, J
        assert np.array_equal(F, first[0]) and np.array_equal(J, first[1]), k
