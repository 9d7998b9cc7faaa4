"""The adjoint stage with other mode counts than a plain two-layer sheet's four: the contraction's
four- and eight-wide forms and their remainders, more than one chain of right-hand sides (four to a
chain) and more than one launch of chains (sixteen to a launch) in the transposed solves, in both
precisions, with and without surface resistance.

The modes are Floquet harmonics of the cell with random sources and weights.  Against the oracle's
adjoint form at 1e-11 relative, the bound of the four-mode parity test."""
import dataclasses

import numpy as np
import pytest

import oracle
from pssfss_b200 import engine
from pssfss_b200.analyze import make_plan, sheet_gblocks, sheet_io
from pssfss_b200.elements import rectstrip
from pssfss_b200.layers import Layer
from pssfss_b200.units import Length, mm

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return float(np.max(np.abs(np.asarray(a) - np.asarray(b))) / np.max(np.abs(np.asarray(b))))


def with_modes(io, sheet, nm, rng):
    """``io`` with ``nm`` harmonics of its first mode's transform variable."""
    upm = sheet.units.units_per_meter
    b1, b2 = sheet.beta1 * upm, sheet.beta2 * upm
    mn = sorted(((m, n) for m in range(-5, 6) for n in range(-5, 6)), key=lambda t: (t[0] ** 2 + t[1] ** 2, t))[:nm]
    c = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    return dataclasses.replace(io, kvec=np.array([io.kvec[0] + m * b1 + n * b2 for m, n in mn]), src=c(nm, 2),
                               tobs=rng.standard_normal((nm, 2)), wobs=c(nm))


@pytest.mark.parametrize("precision", ["fp64", "fp32r"])
@pytest.mark.parametrize("nm,rsheet", [(1, 0.0), (1, 12.5), (3, 0.0), (5, 0.0), (5, 12.5), (7, 12.5), (8, 0.0),
                                       (9, 0.0), (9, 12.5), (12, 0.0), (13, 12.5), (70, 0.0)])
def test_adjoint_mode_counts_match_oracle(nm, rsheet, precision):
    sheet = rectstrip(Lx=10, Ly=5, Px=10, Py=9, Nx=9, Ny=7, units=mm, Rsheet=rsheet)  # spans the cell along x

    def plan_at(eps):
        plan = make_plan([Layer(), sheet, Layer(epsr=eps, width=Length(1, mm)), Layer()], [9.0],
                         {"θ": 20.0, "ϕ": 0.0})
        (_, (i1, i2), _, s), = sheet_gblocks(plan)
        rng = np.random.default_rng(nm)
        ios = [with_modes(sheet_io(pt.layers[i1 - 1:i2], plan.sheets[0], s, pt.k0, pt.beta00), sheet, nm, rng)
               for pt in plan.points]
        return plan, (i1, i2), s, ios
    p0, rng, s, ios0 = plan_at(2.2)
    assert p0.rwgdat[0].nbf > 128
    p1, _, _, ios1 = plan_at(2.2 * (1 + 1e-4))
    args = (p0.sheets[0], p0.rwgdat[0], p0.points, rng, s, p0.uvec[0], ios0,
            [(p1.sheets[0], p1.rwgdat[0], p1.points, p1.uvec[0], ios1)])
    ref0, refk = oracle.partial_gsms_linearized(*args, form="adjoint")
    got0, gotk = engine.partial_gsms_adjoint(*args, precision=precision)
    assert relerr(got0[0], ref0[0]) < 1e-11
    assert relerr(gotk[0][0], refk[0][0]) < 1e-11
