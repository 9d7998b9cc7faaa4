"""The adjoint contraction's two forms - four columns' gathers at once on sheets without resistance,
one entry after another with it - and the assembly's, on J and M sheets, against the oracle's
adjoint form (1e-11 relative, the bound of the adjoint's own parity test)."""
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


@pytest.mark.parametrize("cls,rsheet,nx", [("J", 0.0, 5), ("J", 12.5, 5), ("J", 12.5, 9), ("M", 0.0, 7)])
def test_adjoint_forms_match_oracle(cls, rsheet, nx):
    def plan_at(eps):
        kw = {"class": cls} if cls == "M" else {"Rsheet": rsheet}
        sheet = rectstrip(Lx=10, Ly=4, Px=10, Py=9, Nx=nx, Ny=4, units=mm, **kw)  # spans the cell along x
        plan = make_plan([Layer(), sheet, Layer(epsr=eps, width=Length(1, mm)), Layer()], [9.0, 14.0],
                         {"θ": 20.0, "ϕ": 0.0})
        (_, (i1, i2), _, s), = sheet_gblocks(plan)
        ios = [sheet_io(pt.layers[i1 - 1:i2], plan.sheets[0], s, pt.k0, pt.beta00) for pt in plan.points]
        return plan, (i1, i2), s, ios
    p0, rng, s, ios0 = plan_at(2.2)
    pert = []
    for eps in (2.2 * (1 + 1e-4), 2.2 * (1 - 1e-4)):
        p, _, _, ios = plan_at(eps)
        pert.append((p.sheets[0], p.rwgdat[0], p.points, p.uvec[0], ios))
    args = (p0.sheets[0], p0.rwgdat[0], p0.points, rng, s, p0.uvec[0], ios0, pert)
    ref0, refk = oracle.partial_gsms_linearized(*args, form="adjoint")
    got0, gotk = engine.partial_gsms_adjoint(*args, precision="fp64")
    for i in range(len(p0.points)):
        assert relerr(got0[i], ref0[i]) < 1e-11
        for k in range(len(pert)):
            assert relerr(gotk[k][i], refk[k][i]) < 1e-11
