"""Basis functions with three and four face incidences, which the C ABI takes (the package's own have
two): the assembly's and the adjoint contraction's general form against the oracle.

The sheet is a strip one rectangle wide that spans the cell, so the two triangles of a rectangle share
their diagonal and, across the cell, their vertical edges.  Every other diagonal's basis function is
merged with the pair of vertical edges' (four incidences), or with one edge of it (three).
Tolerances are those of the parity tests (1e-10 for the matrix, 1e-11 for the adjoint form)."""
import numpy as np
import pytest

import oracle
from pssfss_b200 import engine
from pssfss_b200.analyze import make_plan, sheet_gblocks, sheet_io
from pssfss_b200.elements import rectstrip
from pssfss_b200.layers import Layer
from pssfss_b200.rwg import RWGData
from pssfss_b200.units import Length, mm

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return float(np.max(np.abs(np.asarray(a) - np.asarray(b))) / np.max(np.abs(np.asarray(b))))


def merged(rwg, sheet):
    """Basis functions merged as described; returns the new data and each one's incidences."""
    faces = {}
    for b in range(rwg.nbf):
        faces.setdefault(frozenset(rwg.bff[:, b].tolist()), []).append(b)
    ebf, keep, count = rwg.ebf.copy(), np.ones(rwg.nbf, bool), 0
    for pair in (v for v in faces.values() if len(v) == 2):
        inner, across = sorted(pair, key=lambda b: int((rwg.eci[rwg.bfe[:, b] - 1] != 0).any()))
        count += 1
        if count % 3 == 0:
            continue
        keep[across] = False
        edges = rwg.bfe[:, across] - 1
        ebf[edges] = inner + 1
        if count % 3 == 1:
            ebf[edges[1]] = 0
    number = np.concatenate([[0], np.cumsum(keep) * keep])
    new = RWGData(rwg.bfe[:, keep], rwg.bff[:, keep], number[ebf], rwg.eci, rwg.ufpm, rwg.ufp_rep, rwg.nufp)
    inc = np.zeros(new.nbf, int)
    for f in range(sheet.nface):
        for e in sheet.fe[:, f]:
            if new.ebf[e - 1]:
                inc[new.ebf[e - 1] - 1] += 1
    return new, inc


@pytest.mark.parametrize("rsheet", [0.0, 12.5])
def test_three_and_four_incidences(rsheet):
    sheet = rectstrip(Lx=3, Ly=9, Px=3, Py=10, Nx=1, Ny=24, units=mm, Rsheet=rsheet)
    plan = make_plan([Layer(), sheet, Layer(epsr=2.2, width=Length(1, mm)), Layer()], [14.0], {"θ": 25.0, "ϕ": 15.0})
    (_, (i1, i2), _, s), = sheet_gblocks(plan)
    pt, u = plan.points[0], plan.uvec[0]
    layers = pt.layers[i1 - 1:i2]
    rwg, inc = merged(plan.rwgdat[0], sheet)
    assert set(inc.tolist()) >= {2, 3, 4} and inc.max() == 4 and rwg.nbf > 32
    io = sheet_io(layers, sheet, s, pt.k0, pt.beta00)
    Zr, _ = oracle.fill(pt.k0, u, layers, s, io.psi1, io.psi2, sheet, rwg)
    Zg, _ = engine.fill_matrix(sheet, rwg, layers, s, u, pt.k0, io.psi1, io.psi2)
    assert relerr(Zg, Zr) < 1e-10
    args = (sheet, rwg, plan.points, (i1, i2), s, u, [io], [(sheet, rwg, plan.points, u, [io])])
    ref0, refk = oracle.partial_gsms_linearized(*args, form="adjoint")
    got0, gotk = engine.partial_gsms_adjoint(*args)
    assert relerr(got0[0], ref0[0]) < 1e-11 and relerr(gotk[0][0], refk[0][0]) < 1e-11
