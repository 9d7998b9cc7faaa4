"""Tabulated face-pair integrals (``pss_jktab.cu``) against the oracle's ring-by-ring sums.

Sheets on both sides of the rule (pair classes per panel), offsets up to a whole cell, square,
rectangular and skewed cells, zero and non-zero phasings, groups of 1 to 4.  The tolerance is
that of the direct form's own parity test (1e-11 of the largest value): interpolation adds about
1e-16 of the far sum, and a pair whose stopping ring is in doubt takes the direct form."""
import math

import numpy as np
import pytest

import oracle
from pssfss_b200 import engine
from pssfss_b200.analyze import make_plan, sheet_gblocks, sheet_io
from pssfss_b200.elements import diagstrip, meander, polyring, rectstrip
from pssfss_b200.layers import Layer
from pssfss_b200.rwg import setup_rwg
from pssfss_b200.units import mm

pytestmark = pytest.mark.gpu

H = math.sqrt(3) / 2
SHEETS = {
    "ring": lambda: polyring(s1=[9, 0], s2=[0, 9], a=[3.15], b=[3.6], sides=24, ntri=500, units=mm),
    "ring_skew": lambda: polyring(s1=[9, 0], s2=[4.5, 9 * H], a=[2.4], b=[3.2], sides=12, ntri=600, units=mm),
    "aperture": lambda: polyring(s1=[8, 0], s2=[0, 8], a=[0], b=[6 / math.sqrt(2)], sides=4, orient=45, ntri=430,
                                 units=mm, **{"class": "M"}),
    "meander": lambda: meander(a=5, b=10, h=6, w1=0.3, w2=0.3, ntri=1500, units=mm),
    "full_cell": lambda: rectstrip(Lx=8, Ly=7, Px=8, Py=10, Nx=14, Ny=13, units=mm, fufp=False),
    "diagstrip": lambda: diagstrip(P=8, w=1, orient=45, Nl=48, Nw=4, units=mm),
    "small": lambda: rectstrip(Lx=4, Ly=4, Px=10, Py=10, Nx=6, Ny=6, units=mm, fufp=False),
}


def relerr(a, b):
    return float(np.max(np.abs(np.asarray(a) - np.asarray(b))) / np.max(np.abs(np.asarray(b))))


@pytest.mark.parametrize("psi", [(0.0, 0.0), (1.9, -0.7), (math.pi, math.pi)])
@pytest.mark.parametrize("name", sorted(SHEETS))
def test_face_integrals_match_oracle(name, psi):
    sheet = SHEETS[name]()
    rwg = setup_rwg(sheet)
    ul = 0.5 * max(np.linalg.norm(sheet.beta1), np.linalg.norm(sheet.beta2))
    ref = oracle.filljk(sheet, rwg, ul, *psi)
    got = engine.face_integrals(sheet, rwg, ul, *psi)
    for k in ("J", "Jxi", "Jeta", "K", "Kxi", "Keta"):
        assert relerr(got[k], getattr(ref, k)) < 1e-11, k
    assert got["nonconv"] == ref.nonconv


@pytest.mark.parametrize("scale", [0.4, 3.0])
def test_other_smoothing_parameters(scale):
    """Slower and faster decay than the reference's choice (other stopping rings and panels)."""
    sheet = SHEETS["ring"]()
    rwg = setup_rwg(sheet)
    ul = scale * 0.5 * np.linalg.norm(sheet.beta1)
    ref = oracle.filljk(sheet, rwg, ul, 0.8, 0.3)
    got = engine.face_integrals(sheet, rwg, ul, 0.8, 0.3)
    for k in ("J", "Jxi", "Jeta", "K", "Kxi", "Keta"):
        assert relerr(got[k], getattr(ref, k)) < 1e-11, k
    assert got["nonconv"] == ref.nonconv


@pytest.mark.parametrize("npts", [2, 3, 4, 5])
def test_grouped_phasings_equal_single_ones(npts):
    """A sweep whose phasing varies (groups of up to four) against one point at a time."""
    def sweep(freqs):
        plan = make_plan([Layer(), sheet, Layer()], freqs, {"θ": 25.0, "ϕ": 10.0})
        (_, (i1, i2), _, s), = sheet_gblocks(plan)
        ios = [sheet_io(pt.layers[i1 - 1:i2], plan.sheets[0], s, pt.k0, pt.beta00) for pt in plan.points]
        return engine.partial_gsms(plan.sheets[0], plan.rwgdat[0], plan.points, (i1, i2), s, plan.uvec[0], ios)
    sheet = SHEETS["ring"]()
    freqs = np.linspace(9.0, 15.0, npts)
    together = sweep(freqs)
    for i, f in enumerate(freqs):
        alone, = sweep([f])
        assert relerr(together[i], alone) < 1e-12
