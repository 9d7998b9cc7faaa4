"""Pair terms and assembly (``k_pairs``, ``k_assemble``) against the oracle's fill in extended precision
(its source compiled with 80-bit reals), both from the device's own tables and face integrals.

On an unstructured sheet, whose offsets do not fall on boundaries of the tables' cells (the six-point
stencil is not continuous across them, so there a last bit may choose another cell).  Tolerance
4e-15 of the largest entry: an entry is four pair terms (sixteen with boundary pairs), each formed by
some eight operations at the size of the largest one, 32 x 1.1e-16 = 3.6e-15."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

import oracle
from pssfss_b200 import engine
from pssfss_b200.analyze import make_plan, sheet_gblocks, sheet_io
from pssfss_b200.elements import polyring
from pssfss_b200.layers import Layer
from pssfss_b200.units import Length, mm

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def extended(tmp_path_factory):
    d = tmp_path_factory.mktemp("extended")
    src = open(os.path.join(ROOT, "oracle", "pssfss_oracle.c")).read()
    src = re.sub(r"\bdouble\b", "long double", src).replace("CMPLX(", "CMPLXL(").replace("lrint(", "lrintl(")
    (d / "o.c").write_text(src.replace("#include <math.h>", "#include <tgmath.h>"))
    subprocess.run(["gcc", "-O2", "-fPIC", "-shared", "-ffp-contract=off", "-o", str(d / "o.so"), str(d / "o.c"), "-lm"],
                   check=True)
    return ctypes.CDLL(str(d / "o.so"))


def extended_fill(lib, k0, u, layers, s, psi, sheet, rwg, tables, jk):
    def wide(x):
        return np.ascontiguousarray(x, np.clongdouble if np.iscomplexobj(x) else np.longdouble)

    def p(x):
        return x.ctypes.data_as(ctypes.c_void_p)
    a, upm, n = oracle.sheet_arrays(sheet, rwg), sheet.units.units_per_meter, rwg.nbf
    eps, mu, _ = oracle._layer_arrays(layers)
    real, i32, i64 = ctypes.c_longdouble, ctypes.c_int, ctypes.c_int64
    mmax, t1, t2 = tables
    w = [wide(x) for x in (eps, mu, a["rho"], a["fr"], sheet.beta1 * upm, sheet.beta2 * upm)]
    t = [wide(jk[k]) for k in ("J", "Jxi", "Jeta", "K", "Kxi", "Keta", "rho_r", "rinv")] + [wide(t1), wide(t2)]
    Z = np.zeros((n, n), np.clongdouble, order="F")
    lib.ora_fill(i32(int(sheet.cls == "M")), real(k0), real(u), i32(len(layers)), p(w[0]), p(w[1]), i32(s), real(psi[0]),
                 real(psi[1]), i64(sheet.nface), p(w[2]), p(a["fv"]), p(a["fe"]), p(w[3]), i64(n), p(a["bff"]),
                 p(a["ebf"]), p(a["eci"]), p(a["ufpm"]), i64(rwg.nufp), p(a["rep"]), real(upm), p(w[4]), p(w[5]),
                 *[p(x) for x in t], i32(mmax), p(Z))
    return Z


@pytest.mark.parametrize("cls,rsheet", [("J", 0.0), ("J", 12.5), ("M", 0.0)])
def test_fill_against_extended_precision(extended, cls, rsheet):
    kw = {"class": "M"} if cls == "M" else {"Rsheet": rsheet}
    sheet = polyring(s1=[9, 0], s2=[0, 9], a=[2.15], b=[3.6], sides=16, ntri=150, units=mm, **kw)
    plan = make_plan([Layer(), sheet, Layer(epsr=2.2, tandel=0.01, width=Length(1, mm)), Layer()], [11.0],
                     {"θ": 20.0, "ϕ": 10.0})
    (_, (i1, i2), _, s), = sheet_gblocks(plan)
    pt, sh, rwg, u = plan.points[0], plan.sheets[0], plan.rwgdat[0], plan.uvec[0]
    layers, upm = pt.layers[i1 - 1:i2], sh.units.units_per_meter
    io = sheet_io(layers, sh, s, pt.k0, pt.beta00)
    psi = io.psi1, io.psi2
    Z, mmax = engine.fill_matrix(sh, rwg, layers, s, u, pt.k0, *psi)
    tables = engine.modal_tables(int(cls == "M"), pt.k0, u, *psi, layers, s, sh.beta1 * upm, sh.beta2 * upm)[:3]
    assert tables[0] == mmax
    ref = extended_fill(extended, pt.k0, u, layers, s, psi, sh, rwg, tables, engine.face_integrals(sh, rwg, u / upm, *psi))
    assert np.max(np.abs(Z - ref)) <= 4e-15 * np.max(np.abs(ref))
