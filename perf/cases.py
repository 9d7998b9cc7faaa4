"""What this framework is timed on: calls a program makes through its public entry points.

Four kinds of case:

* ``analyze``  - the whole call on layers and sheets: host planning, the sheet sweeps, the
  cascade; one frequency of an optimiser's loop up to a two-sheet oblique stack;
* ``sweep``    - ``engine.partial_gsms``: the scattered partial GSMs of one sheet over a sweep
  (the library's drop-in boundary), the sheet's plan in hand;
* ``batch``    - ``engine.partial_gsms_multi``: sweeps of sheets of differing size in one call;
* ``adjoint``  - ``engine.partial_gsms_adjoint``: the backward direction, one factorisation per
  point and the first-order response to each perturbed input set;
* ``solve``    - ``engine.lu_solve``: the dense complex solver alone on a caller's matrix.

A case's mesh follows from its sizes; the seed moves the band, the angle, the substrate and
(``solve``) the matrix.  Sweeps drop the sheet's face-pair integrals first, so every pass pays
for them as the first sweep of a new sheet does.
"""
import copy
import functools
import importlib.util
import math
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _load_package():
    """The package directory's name is no identifier: it is loaded under ``pssfss_b200``."""
    if "pssfss_b200" not in sys.modules:
        pkgdir = os.path.join(ROOT, "pssfss.jl_b200")
        spec = importlib.util.spec_from_file_location("pssfss_b200", os.path.join(pkgdir, "__init__.py"),
                                                      submodule_search_locations=[pkgdir])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["pssfss_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["pssfss_b200"]


_load_package()
from pssfss_b200 import elements, engine  # noqa: E402
from pssfss_b200.analyze import analyze, make_plan, sheet_gblocks, sheet_io  # noqa: E402
from pssfss_b200.layers import Layer  # noqa: E402
from pssfss_b200.rwg import setup_rwg  # noqa: E402
from pssfss_b200.units import Length, mm  # noqa: E402


def listed():
    return [
        # one frequency of a small patch, as an optimiser or a fit asks for it: latency
        dict(name="patch_point", kind="analyze", element="patch", size=8, points=1, angles=1, theta=0.0,
             precision="fp64"),
        # the square patch of the repository's workloads, whole call, default precision
        dict(name="patch_sweep", kind="analyze", element="patch", size=16, points=11, angles=1, theta=0.0,
             precision="fp64"),
        # a loaded cross scanned in angle: the face-pair integrals change with every point
        dict(name="cross_scan", kind="analyze", element="cross", size=1000, points=3, angles=4, theta=15.0,
             precision="fp32r"),
        # the two-sheet oblique stack (Jerusalem cross, lossy substrate, air gap, aperture)
        dict(name="stack_sweep", kind="analyze", element="stack", size=1500, points=7, angles=1, theta=30.0,
             precision="fp32r"),
        # the headline sweep: meanderline polariser, N = 3976, 101 frequencies
        dict(name="meander_sweep", kind="sweep", element="meander", size=3000, points=101, theta=0.0,
             precision="fp32r"),
        # the same sheet in the FP64 form
        dict(name="meander_fp64", kind="sweep", element="meander", size=3000, points=24, theta=0.0,
             precision="fp64"),
        # the largest order of the repository's benches, N = 5610
        dict(name="meander_5610", kind="sweep", element="meander", size=4000, points=48, theta=0.0,
             precision="fp32r"),
        # an oblique sweep of an unstructured ring: every face pair its own class
        dict(name="ring_sweep", kind="sweep", element="ring", size=1100, points=21, theta=30.0, precision="fp32r"),
        # an aperture (magnetic currents) at an oblique angle in the FP64 form
        dict(name="aperture_fp64", kind="sweep", element="aperture", size=900, points=13, theta=40.0,
             precision="fp64"),
        # many sheets of differing size in one call (a design-space scan)
        dict(name="ring_batch", kind="batch", count=6, small=300, size=1200, points=9, precision="fp32r"),
        # first-order response of a sweep to trace width, pitch and permittivity (both signs)
        dict(name="meander_adjoint", kind="adjoint", size=1500, points=24, precision="fp32r"),
        # the solver alone, an odd order and more right-hand sides than one sweep point has
        dict(name="solve", kind="solve", n=1501, nrhs=5, precision="fp32r"),
    ]


def _log(rng, a, b):
    return a * (b / a) ** rng.random()


def draw(rng):
    kind = rng.choice(["analyze", "analyze", "sweep", "sweep", "sweep", "batch", "adjoint", "solve"])
    precision = rng.choice(["fp64", "fp32r"])
    theta = rng.choice([0.0, 0.0, round(rng.uniform(5, 55), 2)])
    if kind == "analyze":
        element = rng.choice(["patch", "cross", "stack"])
        if element == "patch":
            return dict(kind=kind, element=element, size=round(_log(rng, 5, 20)), points=round(_log(rng, 1, 13)),
                        angles=1, theta=theta, precision=precision)
        return dict(kind=kind, element=element, size=round(_log(rng, 300, 1300)), points=rng.randint(1, 5),
                    angles=1 if theta == 0 else rng.randint(1, 2), theta=theta, precision=precision)
    if kind == "sweep":
        element = rng.choice(["meander", "ring", "aperture"])
        size = round(_log(rng, 300, 3900 if element == "meander" and precision == "fp32r" else 1700))
        most = {"meander": 30, "ring": 16, "aperture": 14}[element]
        return dict(kind=kind, element=element, size=size, points=round(_log(rng, 1, most)),
                    theta=0.0 if element == "meander" else theta, precision=precision)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 7), small=round(_log(rng, 300, 500)),
                    size=round(_log(rng, 600, 1200)), points=rng.randint(2, 9), precision=precision)
    if kind == "adjoint":
        return dict(kind=kind, size=round(_log(rng, 400, 1700)), points=round(_log(rng, 3, 24)), precision=precision)
    return dict(kind=kind, n=round(_log(rng, 150, 2600)), nrhs=rng.randint(1, 12), precision=precision)


@functools.lru_cache(maxsize=64)
def _mesh(element, size):
    if element == "patch":
        return elements.rectstrip(Lx=8, Ly=8, Px=10, Py=10, Nx=size, Ny=size, units=mm)
    if element == "meander":
        return elements.meander(a=5, b=10, h=6, w1=0.3, w2=0.3, ntri=size, units=mm)
    if element == "cross":
        return elements.loadedcross(s1=[8, 0], s2=[0, 8], L1=6, L2=1, w=0.25, ntri=size, units=mm,
                                    Rsheet=0.1)  # lossy metal
    if element == "ring":
        return elements.polyring(s1=[9, 0], s2=[0, 9], a=[3.15], b=[3.6], sides=48, ntri=size, units=mm)
    if element == "aperture":
        return elements.polyring(s1=[8, 0], s2=[0, 8], a=[0], b=[6 / math.sqrt(2)], sides=4, orient=45, ntri=size,
                                 units=mm, **{"class": "M"})
    if element == "jerusalem":
        return elements.jerusalemcross(P=8, L1=6, L2=0.5, A=3, B=0.5, w=0.25, ntri=size, units=mm)
    raise ValueError(element)


def _sheet(element, size):
    return copy.deepcopy(_mesh(element, size))  # a program's own sheet: nothing is shared between states


def _strata(element, size, rng, scale=1.0, sheet=None):
    """Layers around a sheet; the seed moves the permittivities and thicknesses by a few percent."""
    eps = 2.2 * scale * rng.uniform(0.97, 1.03)
    if element == "meander":
        return [Layer(), sheet or _sheet(element, size),
                Layer(epsr=eps, width=Length(rng.uniform(0.95, 1.05), mm)), Layer()]
    if element == "stack":
        return [Layer(), _sheet("jerusalem", size),
                Layer(epsr=3.0 * rng.uniform(0.97, 1.03), tandel=0.002, width=Length(0.5, mm)),
                Layer(width=Length(rng.uniform(1.9, 2.1), mm)), _sheet("aperture", round(0.8 * size)), Layer()]
    if element == "cross":
        return [Layer(), _sheet(element, size), Layer(epsr=eps, tandel=0.001, width=Length(0.8, mm)), Layer()]
    return [Layer(), _sheet(element, size), Layer()]


_BANDS = {"patch": (10, 20), "cross": (10, 17), "stack": (5, 25), "meander": (8, 18), "ring": (10, 18),
          "aperture": (10, 18)}


def _freqs(element, points, rng):
    lo, hi = _BANDS[element]
    shift = rng.uniform(0, 0.02 * (hi - lo))
    return np.linspace(lo, hi, points + 1)[:points] + shift


def _angle(theta, rng):
    return 0.0 if theta == 0 else theta + rng.uniform(-2, 2)


def _sweep_args(strata, flist, steering):
    """Arguments of a sheet sweep (one sheet): what a program keeps of its plan."""
    plan = make_plan(strata, flist, steering)
    (_, (i1, i2), isht, s), = sheet_gblocks(plan)
    sheet, rwg = plan.sheets[isht - 1], plan.rwgdat[isht - 1]
    ios = [sheet_io(pt.layers[i1 - 1:i2], sheet, s, pt.k0, pt.beta00) for pt in plan.points]
    return dict(sheet=sheet, rwg=rwg, points=plan.points, region_rng=(i1, i2), s=s, u=plan.uvec[isht - 1], ios=ios)


def _matrix(case, seed):
    """A matrix like a moment matrix: an oscillating kernel that decays with distance, heavier on
    the diagonal, the unknowns scattered over a cell."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    r = rng.uniform(0, 1, (n, 2))
    d = np.hypot(r[:, None, 0] - r[None, :, 0], r[:, None, 1] - r[None, :, 1])
    A = np.exp(-3j * d) / (d + 0.03) * (1 + 0.3 * rng.standard_normal((n, n))) / math.sqrt(n)
    A[np.arange(n), np.arange(n)] += 6 + 2j * rng.standard_normal(n)
    B = rng.standard_normal((n, case["nrhs"])) + 1j * rng.standard_normal((n, case["nrhs"]))
    return np.asfortranarray(A), np.asfortranarray(B)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "analyze":
        el = case["element"]
        strata = _strata(el, case["size"], rng)
        phi = 45.0 if el == "stack" else 0.0
        theta = [_angle(case["theta"] * (k + 1) / case["angles"], rng) for k in range(case["angles"])]
        return dict(case=case, strata=strata, flist=_freqs(el, case["points"], rng), steering={"θ": theta, "ϕ": phi})
    if kind == "sweep":
        el = case["element"]
        flist, th = _freqs(el, case["points"], rng), _angle(case["theta"], rng)
        return dict(case=case, args=_sweep_args(_strata(el, case["size"], rng), flist, {"θ": th, "ϕ": 0.0}))
    if kind == "batch":
        problems = []
        for k, size in enumerate(_batch_sizes(case)):
            th = _angle([30.0, 0.0, 15.0, 45.0][k % 4], rng)
            problems.append(_sweep_args(_strata("ring", size, rng), _freqs("ring", case["points"], rng),
                                        {"θ": th, "ϕ": 0.0}))
        return dict(case=case, problems=problems)
    if kind == "adjoint":
        flist, steer = _freqs("meander", case["points"], rng), {"θ": 0.0, "ϕ": 0.0}
        eps, steps = 2.2 * rng.uniform(0.97, 1.03), []
        for w, a, e in ((0.3, 5.0, eps), *((0.3 * (1 + h), 5.0, eps) for h in (1e-4, -1e-4)),
                        *((0.3, 5.0 * (1 + h), eps) for h in (1e-4, -1e-4)),
                        *((0.3, 5.0, eps * (1 + h)) for h in (1e-4, -1e-4))):
            sheet = elements.meander(a=a, b=10, h=6, w1=w, w2=w, ntri=case["size"], units=mm)
            steps.append(_sweep_args([Layer(), sheet, Layer(epsr=e, width=Length(1, mm)), Layer()], flist, steer))
        pert = [(p["sheet"], p["rwg"], p["points"], p["u"], p["ios"]) for p in steps[1:]]
        return dict(case=case, args=steps[0], pert=pert)
    A, B = _matrix(case, seed)
    return dict(case=case, A=A, B=B)


def _batch_sizes(case):
    c = case["count"]
    return [round(case["small"] * (case["size"] / case["small"]) ** (k / (c - 1))) for k in range(c)]


def _gsms(results):
    """All scattering matrices of a sweep, (points, n, n) per block."""
    return {b: np.stack([getattr(r.gsm, b) for r in results]) for b in ("s11", "s12", "s21", "s22")}


def run(state):
    case = state["case"]
    kind, precision = case["kind"], case["precision"]
    if kind == "analyze":
        return _gsms(analyze(state["strata"], state["flist"], state["steering"], precision=precision))
    if kind == "sweep":
        a = state["args"]
        engine.clear_face_integrals(a["sheet"], a["rwg"])
        return np.stack(engine.partial_gsms(**a, precision=precision))
    if kind == "batch":
        for p in state["problems"]:
            engine.clear_face_integrals(p["sheet"], p["rwg"])
        return [np.stack(o) for o in engine.partial_gsms_multi(state["problems"], precision=precision)]
    if kind == "adjoint":
        a = state["args"]
        for sheet, rwg in [(a["sheet"], a["rwg"])] + [p[:2] for p in state["pert"]]:
            engine.clear_face_integrals(sheet, rwg)
        dS, dSp = engine.partial_gsms_adjoint(a["sheet"], a["rwg"], a["points"], a["region_rng"], a["s"], a["u"],
                                              a["ios"], state["pert"], precision=precision)
        return {"dS": np.stack(dS), "dSp": np.stack([np.stack(d) for d in dSp])}
    X, status = engine.lu_solve(state["A"], state["B"], precision)
    return {"X": X, "status": status}


def exact(case, seed):
    """The solver's answer from LAPACK in 64 bits.  A sweep's answer in plain numpy would be the
    whole method of moments written again, with seconds per point: none is given."""
    if case["kind"] != "solve":
        return None
    A, B = _matrix(case, seed)
    return {"X": np.linalg.solve(A, B), "status": None}


@functools.lru_cache(maxsize=64)
def _sizes(element, size):
    """(faces, unknowns, face-pair classes) of a mesh."""
    m = _mesh(element, size)
    rwg = setup_rwg(m)
    return m.nface, rwg.nbf, rwg.nufp



def _sheet_work(element, size, points, phasings, rhs=4):
    """What a sheet sweep cannot do without.  Operations: per phasing and face-pair class 7
    quadrature points of a lattice sum (about 300 operations: the nine nearest images one by one,
    the smooth remainder by any means); per point and class 7 x 2 table look-ups (about 60 each) and the 9 edge-pair terms (about 20 each); per
    point the N x N assembly (about 32 per entry), the complex LU (8/3 N^3) and one solve per
    incident mode (8 N^2).  Bytes: the mesh's class map and representatives, the mode data of
    every point, and the partial GSMs."""
    nface, n, nufp = _sizes(element, size)
    flops = phasings * nufp * 7 * 300.0
    flops += points * (nufp * (14 * 60 + 9 * 20.0) + 32.0 * n * n + 8 / 3 * n ** 3 + 8.0 * n * n * rhs)
    return dict(bytes=8.0 * (nface * nface + nufp) + points * rhs * (64 + 16.0 * rhs), flops=flops)


def _sum(works):
    return dict(bytes=float(sum(w["bytes"] for w in works)), flops=float(sum(w["flops"] for w in works)))


def work(case):
    kind = case["kind"]
    if kind == "analyze":
        pts = case["points"] * case["angles"]
        phasings = 1 if case["theta"] == 0 else pts
        if case["element"] == "stack":
            parts = [("jerusalem", case["size"]), ("aperture", round(0.8 * case["size"]))]
        else:
            parts = [(case["element"], case["size"])]
        return _sum([_sheet_work(e, s, pts, phasings) for e, s in parts])
    if kind == "sweep":
        phasings = 1 if case["theta"] == 0 else case["points"]
        return _sheet_work(case["element"], case["size"], case["points"], phasings)
    if kind == "batch":
        return _sum([_sheet_work("ring", s, case["points"], 1 if k % 4 == 1 else case["points"])
                     for k, s in enumerate(_batch_sizes(case))])
    if kind == "adjoint":
        # the sweep with forward and transposed solves, and six perturbed sets, each with its
        # own pair terms, assembly and contraction at every point
        nface, n, nufp = _sizes("meander", case["size"])
        w = _sheet_work("meander", case["size"], case["points"], 1, rhs=8)
        w["flops"] += 6 * (nufp * 7 * 300.0
                           + case["points"] * (nufp * (14 * 60 + 9 * 20.0) + (32 + 8 * 4.0) * n * n))
        w["bytes"] *= 7
        return w
    n, nrhs = case["n"], case["nrhs"]
    return dict(bytes=16.0 * (n * n + 2 * n * nrhs), flops=8 / 3 * n ** 3 + 8.0 * n * n * nrhs)
