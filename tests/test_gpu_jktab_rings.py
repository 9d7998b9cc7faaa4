"""Tabulated face-pair integrals: which sheets take them, and the reference's stopping ring where it is
hard to see.

* The form is read off the kernels a call launches: the direct sums take one, the tables four.
* ``zeros``: a phasing at which both of ring 6's sums vanish along the sheet's long axis, within a
  strip narrower than the distance between a panel's nodes.  The reference stops at ring 6 there and
  at ring 8 around it, so a ring too many moves the integrals by some 1e-12 to 1e-10 of themselves.
* ``compact``: a sheet of less than half a cell, whose panels (0.21 wide) and sub-cells are the
  widest at the reference's smoothing parameter.

Tolerance 1e-13 of the largest value: both sides add the same summands, some 1e3 rounding errors of
1.1e-16 that mostly cancel, and the interpolation of the far sums adds 1e-15 at most."""
import importlib.util
import math
import os

import numpy as np
import pytest

import oracle
from pssfss_b200 import engine
from pssfss_b200.elements import rectstrip
from pssfss_b200.rwg import setup_rwg
from pssfss_b200.units import mm

pytestmark = pytest.mark.gpu

_spec = importlib.util.spec_from_file_location(
    "jktab_sheets", os.path.join(os.path.dirname(os.path.abspath(__file__)), "test_gpu_jktab.py"))
_mod = importlib.util.module_from_spec(_spec)
_spec.loader.exec_module(_mod)
SHEETS = {
    **_mod.SHEETS,
    "zeros": lambda: rectstrip(Lx=4.706, Ly=19.133, Px=10, Py=25.671, Nx=12, Ny=20, units=mm, fufp=False),
    "compact": lambda: rectstrip(Lx=4, Ly=4, Px=10, Py=10, Nx=8, Ny=8, units=mm, fufp=False),
}
TABULATED = {"ring", "ring_skew", "aperture", "meander", "full_cell", "zeros", "compact"}


def smoothing(sheet):
    return 0.5 * max(np.linalg.norm(sheet.beta1), np.linalg.norm(sheet.beta2))


@pytest.mark.parametrize("name", sorted(SHEETS))
def test_form_taken(name):
    sheet = SHEETS[name]()
    rwg = setup_rwg(sheet)
    engine.face_integrals(sheet, rwg, smoothing(sheet), 0.3, 0.2)  # uploads the sheet
    before = engine.lib().pss_kernel_launches()
    engine.face_integrals(sheet, rwg, smoothing(sheet), 0.3, 0.2)
    assert engine.lib().pss_kernel_launches() - before == (4 if name in TABULATED else 1)


@pytest.mark.parametrize("name,psi", [("zeros", (-2.88005, 1.07222)), ("zeros", (math.pi, math.pi)),
                                      ("compact", (0.0, 0.0)), ("compact", (1.9, -0.7)), ("compact", (math.pi, 0.0)),
                                      ("full_cell", (0.0, math.pi)), ("meander", (math.pi, math.pi)),
                                      ("ring", (3.1304, 3.1495))])
def test_integrals_match_oracle_closely(name, psi):
    sheet = SHEETS[name]()
    rwg = setup_rwg(sheet)
    ref = oracle.filljk(sheet, rwg, smoothing(sheet), *psi)
    got = engine.face_integrals(sheet, rwg, smoothing(sheet), *psi)
    for k in ("J", "Jxi", "Jeta", "K", "Kxi", "Keta"):
        r = getattr(ref, k)
        assert np.max(np.abs(got[k] - r)) <= 1e-13 * np.max(np.abs(r)), k
    assert got["nonconv"] == ref.nonconv
