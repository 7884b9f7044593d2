"""Workloads of nemoh_b200: what a program has the framework compute, through its public entry points.

    listed()            the workloads, smallest to largest
    draw(rng)           one more of the same ranges
    prepare(case, seed) what the program holds before the call: a context with its mesh or resident bodies, and inputs
    run(state)          one call (or one call chain) and its results
    work(case)          bytes and operations of one pass that no program could do without
    exact(case, seed)   the results in plain numpy, for the outputs that have a closed form of moderate cost

Kinds of workload:
    problem      the Fortran Solver's own loop: one SOLVE_POTENTIAL call per problem, a factorization per frequency
    sweep        all problems of many frequencies of one hull, host arrays in and forces out
    device       the same with the pre-processor's body conditions built on the GPU and everything resident there
    bodies       (body, frequency) items of many hulls in one call
    requests     a serving batch: one frequency and heading per request, right-hand sides built on the GPU
    elevation    free-surface elevation of solved problems on a grid
    outputs      Kochin function of solved problems and the impulse responses of a coefficient table

The geometry's topology follows from the case alone (so that its work does); the seed sets the hull's scale, the
frequencies, the headings and the coefficients.
"""
import functools
import math

import numpy as np
import torch

import nemoh_b200 as nb
from nemoh_b200 import cases as C

RHO, G = 1025.0, 9.81


# ---------------------------------------------------------------------------
# hulls
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=16)
def _mesh(form, panels):
    if form == "barge":         # 100 x 20 x 10 m, y-symmetric half mesh (2,400 panels at the usual spacing)
        f = math.sqrt(panels / 2400.0)
        k = [max(2, round(v * f)) for v in (50, 20, 20, 10)]
        return C.config_barge(1, *k).mesh
    if form in ("cylinder", "half_cylinder"):   # R = 5 m, draft 10 m (300 panels at the usual spacing)
        half = form == "half_cylinder"
        f = math.sqrt(panels * (2 if half else 1) / 300.0)
        return C.cylinder_mesh(5.0, 10.0, 2 * max(2, round(12 * f)), max(2, round(10 * f)), max(1, round(5 * f)),
                               2 * max(2, round(6 * f)), half=half)
    if form == "sphere":        # floating half sphere, R = 4 m
        nlat = max(3, round(math.sqrt(panels / 2.5)))
        return C.hemisphere_mesh(4.0, nlat, max(8, round(panels / nlat)))
    if form == "two_spheres":   # two hulls side by side, 8,000 panels
        return C.config_two_spheres(1).mesh
    raise ValueError(form)


@functools.lru_cache(maxsize=8)
def _fleet(mix, count, n_max):
    """Hulls of a mixed batch: cylinders, boxes and spheres of 200 to n_max panels, half of them in finite depth."""
    rng = np.random.default_rng(mix)
    return [C.random_body(rng, 200, n_max) for _ in range(count)]


def _scaled(mesh, s):
    return C.Mesh(mesh.nodes * s, mesh.panels, mesh.isym, mesh.body, mesh.nbodies)


def _case(case, seed):
    """The hull of a case with the seed's scale, frequencies and headings."""
    rng = np.random.default_rng(seed)
    m = _scaled(_mesh(case["form"], case["panels"]), rng.uniform(0.97, 1.03))
    nw = case["omegas"]
    lo, hi = case["lo"], case["hi"]
    om = lo + (hi - lo) * (np.arange(nw) + rng.uniform(0.05, 0.95, nw)) / nw
    if case["form"] == "two_spheres":
        dofs = C.six_dofs((-10.0, 0.0, 0.0), 1) + C.six_dofs((10.0, 0.0, 0.0), 2)
    else:
        dofs = C.six_dofs()
    return C.Case(m, om, rng.uniform(0.0, 180.0, case["headings"]), dofs, list(dofs), rho=RHO, g=G,
                  depth=case["depth"])


def _fleet_cases(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for mesh, depth in _fleet(case["mix"], case["bodies"], case["n_max"]):
        nw = case.get("omegas", 1)
        om = np.sort(np.linspace(0.2, 2.4, nw) + rng.uniform(-0.1, 0.1, nw))
        out.append(C.Case(_scaled(mesh, rng.uniform(0.97, 1.03)), om, rng.uniform(0.0, 180.0, 1), C.six_dofs(),
                          C.six_dofs(), rho=RHO, g=G, depth=depth))
    return out


def _precision(case):
    return nb.MIXED if case["precision"] == "mixed" else nb.FP64


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a small hull through the drop-in boundary, problem by problem: latency and launches are all there is
        dict(name="problem half cylinder 60", kind="problem", form="half_cylinder", panels=60, depth=15.0, omegas=2,
             headings=1, lo=0.4, hi=1.6, precision="fp64"),
        # the 300-panel verification hull in deep water, a short sweep in the default precision
        dict(name="sweep cylinder 300 fp64", kind="sweep", form="cylinder", panels=300, depth=0.0, omegas=10,
             headings=1, lo=0.1, hi=2.0, precision="fp64"),
        # a preliminary-design sweep in the default precision, everything on the GPU, an order that no tile divides
        dict(name="device sphere 1311 fp64", kind="device", form="sphere", panels=1311, depth=0.0, omegas=8,
             headings=3, lo=0.2, hi=2.2, precision="fp64"),
        # the headline hull and sweep in both precisions (finite depth and deep water in one sweep)
        dict(name="sweep barge 2400 fp64", kind="sweep", form="barge", panels=2400, depth=50.0, omegas=20,
             headings=3, lo=0.05, hi=2.5, precision="fp64"),
        dict(name="sweep barge 2400 mixed", kind="sweep", form="barge", panels=2400, depth=50.0, omegas=40,
             headings=3, lo=0.05, hi=2.5, precision="mixed"),
        # the largest mesh: two hulls, 12 DOF, no symmetry
        dict(name="sweep two spheres 8000 mixed", kind="sweep", form="two_spheres", panels=8000, depth=0.0, omegas=6,
             headings=2, lo=0.2, hi=3.0, precision="mixed"),
        # parametric study over uneven hulls, both precisions
        dict(name="bodies 12 fp64", kind="bodies", mix=11, bodies=12, n_max=3000, omegas=5, precision="fp64"),
        dict(name="bodies 32 mixed", kind="bodies", mix=4, bodies=32, n_max=3000, omegas=5, precision="mixed"),
        # serving: the batch a lightly loaded server takes, and one near saturation
        dict(name="requests 6 mixed", kind="requests", mix=5, bodies=16, n_max=3000, requests=6, precision="mixed"),
        dict(name="requests 48 mixed", kind="requests", mix=5, bodies=16, n_max=3000, requests=48,
             precision="mixed"),
        # output stages of the headline hull: elevation on the pre-processor's 101 x 101 grid, and the Kochin
        # function at every degree with the impulse responses of a 40-frequency table
        dict(name="elevation barge 2400", kind="elevation", form="barge", panels=2400, depth=50.0, omegas=1,
             headings=3, lo=0.5, hi=0.9, precision="fp64", side=101),
        dict(name="outputs barge 2400", kind="outputs", form="barge", panels=2400, depth=50.0, omegas=1, headings=3,
             lo=0.5, hi=0.9, precision="fp64", directions=361, table=40, steps=1000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["problem", "sweep", "sweep", "sweep", "device", "bodies", "requests", "elevation", "outputs"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "bodies":
        return dict(kind=kind, mix=rng.randrange(1 << 16), bodies=rng.randint(3, 12), n_max=_log(rng, 600, 3000),
                    omegas=rng.randint(2, 5), precision=precision)
    if kind == "requests":
        return dict(kind=kind, mix=rng.randrange(1 << 16), bodies=rng.randint(4, 16), n_max=_log(rng, 600, 3000),
                    requests=_log(rng, 6, 48), precision="mixed")
    form = rng.choice(["barge", "half_cylinder", "cylinder", "sphere"])
    depth = 0.0 if form == "sphere" or rng.random() < 0.5 else round(rng.uniform(25.0, 120.0), 2)
    base = dict(kind=kind, form=form, depth=depth, headings=rng.randint(1, 4), lo=round(rng.uniform(0.05, 0.4), 3),
                hi=round(rng.uniform(1.2, 2.5), 3), precision=precision)
    if kind == "problem":   # the Solver executable's loop, which runs in double precision
        return dict(base, panels=_log(rng, 60, 1200), omegas=2, headings=1, precision="fp64")
    if kind in ("elevation", "outputs"):
        base.update(panels=_log(rng, 150, 2400), omegas=1, precision="fp64")
        if kind == "elevation":
            return dict(base, side=rng.randint(21, 101))
        return dict(base, directions=_log(rng, 36, 361), table=rng.randint(15, 60), steps=_log(rng, 100, 2000))
    few = 6 if precision == "mixed" else 2   # the mixed path is for sweeps
    panels = _log(rng, 100, 4000)
    return dict(base, panels=panels, omegas=rng.randint(few, max(few, min(30, int(12000 / panels)))))


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    s = nb.Solver(0, _precision(case))
    st = {"kind": kind, "solver": s}
    if kind in ("bodies", "requests"):
        fleet = _fleet_cases(case, seed)
        ids = [s.add_body(c) for c in fleet]
        if kind == "bodies":
            st["bodies"] = np.repeat(np.array(ids, dtype=np.int32), case["omegas"])
            st["omegas"] = np.concatenate([c.omegas for c in fleet])
            nv = [C.body_conditions(c) for c in fleet]
            p = 7
            st["nvel"] = [np.asfortranarray(v[:, j * p:(j + 1) * p]) for v, c in zip(nv, fleet)
                          for j in range(len(c.omegas))]
        else:
            rng = np.random.default_rng(seed + 1)
            for b, c in zip(ids, fleet):
                s.set_body_dofs(b, c.rad)
            n = case["requests"]
            # which bodies a batch meets follows from the case, so that its work does
            st["bodies"] = _asked(case)
            st["omegas"] = rng.uniform(0.1, 2.5, n)
            st["betas"] = rng.uniform(0.0, math.pi, n)
        s.prepare_bodies()
        return st
    c = _case(case, seed)
    s.set_case(c)
    nc = c.mesh.npanels * 2 ** c.mesh.isym
    nprob = len(c.betas_deg) + len(c.rad)
    st.update(omegas=c.omegas, periods=2 * np.pi / c.omegas)
    if kind == "problem":
        nv = C.body_conditions(c)
        st["nvel"] = [[np.ascontiguousarray(nv[:, i * nprob + j]) for j in range(nprob)] for i in range(len(c.omegas))]
    elif kind == "sweep":
        st["nvel"] = np.asfortranarray(C.body_conditions(c).reshape(nc, nprob, len(c.omegas), order="F"))
        st["nds"] = np.asfortranarray(C.generalised_normals(c))
    elif kind == "device":
        dev = torch.device("cuda", 0)
        nf, nw, nbeta = len(c.force), len(c.omegas), len(c.betas_deg)
        st.update(case=c, nprob=nprob, nint=nf,
                  nvel=torch.zeros(nw, nprob, nc, dtype=torch.complex128, device=dev),
                  nds=torch.zeros(nc, nf, dtype=torch.float64, device=dev),
                  fk=torch.zeros(nw, nbeta, nf, dtype=torch.complex128, device=dev),
                  force=torch.zeros(nw, nprob, nf, dtype=torch.complex128, device=dev))
    else:
        T = float(st["periods"][0])
        nv = C.body_conditions(c)
        r = [s.solve_potential(T, nv[:, j]) for j in range(nprob)]
        st.update(case=c, T=T, zigb=np.stack([x["zigb"] for x in r], axis=1),
                  zigs=np.stack([x["zigs"] for x in r], axis=1) if c.mesh.isym else None)
        if kind == "elevation":
            reach = 4.0 * np.abs(c.mesh.nodes[:, :2]).max()
            st["points"] = C.freesurface_grid(case["side"], case["side"], 2 * reach, 2 * reach)[0]
        else:
            st.update(_table(case, seed), theta=np.linspace(0.0, 2 * np.pi, case["directions"]),
                      steps=case["steps"])
    return st


def _asked(case):
    return np.random.default_rng(case["mix"] + 1).integers(0, case["bodies"], case["requests"]).astype(np.int32)


def _table(case, seed):
    """Added mass and damping of a 6-DOF body over a frequency table."""
    rng = np.random.default_rng(seed + 2)
    w = np.sort(np.linspace(0.05, 2.5, case["table"]) + rng.uniform(0.0, 0.02, case["table"]))
    B = rng.standard_normal((len(w), 6, 6)) * np.exp(-w)[:, None, None]
    A = rng.standard_normal((len(w), 6, 6))
    return dict(w=w, damping=np.asfortranarray(B), added=np.asfortranarray(A))


def run(state):
    s, kind = state["solver"], state["kind"]
    if kind == "problem":
        out = []
        for T, cols in zip(state["periods"], state["nvel"]):
            for v in cols:
                r = s.solve_potential(T, v)
                out.append([r["zigb"], r["zigs"], r["zpb"], r["zps"]])
        return np.array(out)
    if kind == "sweep":
        return s.solve_frequencies(state["omegas"], state["nvel"], state["nds"])
    if kind == "device":
        s.body_conditions_device(state["case"], state["nvel"].data_ptr(), state["nds"].data_ptr(),
                                 state["fk"].data_ptr())
        s.solve_frequencies_device(state["omegas"], state["nvel"].data_ptr(), state["nprob"], state["nint"],
                                   state["nds"].data_ptr(), state["force"].data_ptr())
        return {k: state[k] for k in ("nvel", "nds", "fk", "force")}
    if kind == "bodies":
        return np.stack(s.solve_bodies(state["bodies"], state["omegas"], state["nvel"]))
    if kind == "requests":
        return np.stack(s.solve_requests(state["bodies"], state["omegas"], state["betas"]))
    if kind == "elevation":
        return s.free_surface(state["T"], state["points"], state["zigb"], state["zigs"])
    h = s.kochin(state["T"], state["theta"], state["zigb"], state["zigs"])
    K, ainf = s.irf(state["w"], state["damping"], state["added"], state["steps"], 0.1)
    return {"kochin": h, "K": K, "ainf": ainf}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
# Operations of one ordered pair of panels and one reflection: the tabulated wave term (four 3 x 3 interpolations) and
# the Rankine images, at the smallest count that the formulas allow; in finite depth three images more and about
# twenty exponential images of a reciprocal square root each.
PAIR_DEEP, PAIR_FINITE = 150.0, 900.0


def _solve_work(n, classes, nrhs, fd):
    """(bytes, flops) of one frequency: assembly, LU, solves and potential of `classes` systems of order n."""
    pair = PAIR_FINITE if fd else PAIR_DEEP
    flops = classes * n * n * pair + classes * (8.0 / 3 * n ** 3 + 16.0 * n * n * nrhs)
    return classes * n * 16.0 * nrhs, flops


def work(case):
    kind = case["kind"]
    b = f = 0.0
    if kind in ("bodies", "requests"):
        fleet = _fleet(case["mix"], case["bodies"], case["n_max"])
        which = _asked(case) if kind == "requests" else np.repeat(np.arange(case["bodies"]), case["omegas"])
        for i in which:
            mesh, depth = fleet[i]
            x, y = _solve_work(mesh.npanels, 1 + mesh.isym, 7, depth > 0)
            b, f = b + (x if kind == "bodies" else 0) + 16 * 6 * 7, f + y
        return {"bytes": b, "flops": f}
    mesh = _mesh(case["form"], case["panels"])
    n, cls = mesh.npanels, 1 + mesh.isym
    nprob = case["headings"] + (12 if case["form"] == "two_spheres" else 6)
    if kind in ("problem", "sweep", "device"):
        x, y = _solve_work(n, cls, nprob, case["depth"] > 0)
        return {"bytes": case["omegas"] * x + 16.0 * 6 * nprob, "flops": case["omegas"] * y}
    strengths = cls * n * nprob * 16.0
    if kind == "elevation":
        pts = case["side"] ** 2
        pair = PAIR_FINITE if case["depth"] > 0 else PAIR_DEEP
        return {"bytes": strengths + pts * 16.0 * (1 + nprob), "flops": pts * n * cls * (pair + 8.0 * nprob)}
    d = case["directions"]
    # Kochin: four edges of a complex exponential (about 40 operations) and a complex quotient per panel and half
    flops = d * n * cls * (4 * 80.0 + 8.0 * nprob) + 2 * 36 * case["table"] * case["steps"] * 5.0
    return {"bytes": strengths + d * nprob * 16.0 + 36 * 8.0 * (2 * case["table"] + case["steps"]), "flops": flops}


# ---------------------------------------------------------------------------
# results in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    """Closed forms: body conditions and impulse responses. The solves, and the elevation and Kochin function of their
    source strengths, rest on the tabulated Green function of the whole mesh; evaluated in plain numpy they take far
    longer than a check may."""
    if case["kind"] == "device":
        c = _case(case, seed)
        nvel, nds, fk = _body_conditions(c)
        return {"nvel": nvel, "nds": nds, "fk": fk, "force": None}
    if case["kind"] == "outputs":
        t = _table(case, seed)
        K, ainf = _impulse_response(t["w"], t["damping"], t["added"], case["steps"], 0.1)
        return {"kochin": None, "K": K, "ainf": ainf}
    return None


def _wavenumber(w, g, depth):
    """The pre-processor's wave number: bisection on x tanh x = w^2 h / g to a relative 1e-6."""
    x0 = w * w / g * depth
    if not 0.0 < x0 <= 20.0:
        return w * w / g
    f = lambda x: x0 - x * math.tanh(x)  # noqa: E731
    a, b = 0.0, x0
    while f(a) * f(b) > 0.0:
        a, b = b, 2.0 * b
    mid = 0.5 * (a + b)
    while abs(b - a) / abs(mid) >= 1.0e-6:
        mid = 0.5 * (a + b)
        if f(a) * f(mid) > 0.0:
            a = mid
        else:
            b = mid
    return mid / depth


def _body_conditions(c):
    """Normal velocities (nw, nprob, 2^s n), generalised normals (2^s n, nint) and Froude-Krylov forces
    (nw, nbeta, nint) of the incident wave and the rigid motions."""
    x, p = c.mesh.nodes, c.mesh.panels - 1
    v = [x[p[:, k]] for k in range(4)]
    w1, w2 = np.cross(v[1] - v[0], v[3] - v[1]), np.cross(v[3] - v[2], v[1] - v[2])
    a1, a2 = 0.5 * np.linalg.norm(w1, axis=1), 0.5 * np.linalg.norm(w2, axis=1)
    area = a1 + a2
    xm = ((v[0] + v[1] + v[3]) * (a1 / area)[:, None] + (v[1] + v[2] + v[3]) * (a2 / area)[:, None]) / 3
    nrm = (w1 + w2) / np.linalg.norm(w1 + w2, axis=1)[:, None]
    if c.mesh.isym:
        flip = np.array([1.0, -1.0, 1.0])
        xm, nrm = np.concatenate([xm, xm * flip]), np.concatenate([nrm, nrm * flip])
        area = np.concatenate([area, area])
    unit = []
    for d in c.rad:
        vel = np.tile(np.asarray(d.direction, float), (len(xm), 1))
        if d.icase == 2:
            vel = np.cross(np.asarray(d.direction, float), xm - np.asarray(d.axis, float))
        unit.append((nrm * vel).sum(axis=1))
    unit = np.array(unit)
    nds = (unit * area).T
    nvel, fk = [], []
    for w in c.omegas:
        k = _wavenumber(float(w), c.g, c.depth)
        kh, z = k * c.depth, xm[:, 2]
        shallow = 0.0 < kh <= 20.0
        ch = np.cosh(k * (z + c.depth)) / math.cosh(kh) if shallow else np.exp(k * z)
        sh = np.sinh(k * (z + c.depth)) / math.cosh(kh) if shallow else np.exp(k * z)
        cols, f = [], []
        for b in np.asarray(c.betas_deg) * math.pi / 180.0:
            e = np.exp(1j * k * (xm[:, 0] * math.cos(b) + xm[:, 1] * math.sin(b)))
            a = c.g / w * k
            cols.append(-(a * math.cos(b) * ch * e * nrm[:, 0] + a * math.sin(b) * ch * e * nrm[:, 1]
                          - 1j * a * sh * e * nrm[:, 2]))
            f.append(-(nds * (c.rho * c.g * ch * e)[:, None]).sum(axis=0))
        nvel.append(cols + list(unit.astype(complex)))
        fk.append(f)
    return np.array(nvel), nds, np.array(fk)


def _impulse_response(w, damping, added, steps, dt):
    """K(t) = 2/pi int B cos(wt) dw and the mean over w of A + 1/w int K sin(wt) dt, both by the trapezoid rule."""
    t = np.arange(steps) * dt
    nw = len(w)
    B, A = damping.reshape(nw, -1), added.reshape(nw, -1)
    f = np.cos(np.outer(t, w))
    dw = np.diff(w)
    K = ((f[:, :-1] * dw) @ B[:-1] + (f[:, 1:] * dw) @ B[1:]) / math.pi
    s = np.sin(np.outer(w, t))
    step = np.diff(t)
    cm = A + 0.5 * ((s[:, :-1] * step) @ K[:-1] + (s[:, 1:] * step) @ K[1:]) / w[:, None]
    shape = damping.shape[1:]
    return K.reshape((steps,) + shape), cm.mean(axis=0).reshape(shape)
