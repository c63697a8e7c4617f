"""The work that users of this package have it do, as timed cases.

Each case is one call chain through the public entry points of
``nonlocal_gb300.thermal``, from host arrays to host arrays, as a program that
replaces the reference's solver classes runs it.  ``kind`` picks the chain:

* ``steady``   a stationary 2D heat problem.  ``oneshot``: the problem is made
  from the host mesh and closed within the pass (one mesh, one solve, as the
  reference's application runs); otherwise it stays on the GPU and the pass sets
  model and boundaries again and solves (a parameter study).
* ``fields``   several problems with a conductivity field (non-symmetric systems),
  assembled one after another and solved in one batched call.
* ``march``    a nonstationary problem: compute and a few implicit Euler steps.
* ``fleet``    one step of many nonstationary instances of uneven size.
* ``plate``    nonlocal plane elasticity.
* ``flux``     the nodal heat flux of a temperature field.
* ``plugin``   the conjugate gradient on the caller's own CSR matrices with ILLT.
* ``rod``      the stationary (``steps`` 0) or nonstationary 1D solver.

Sizes follow the package's benchmark workloads (300x300 8-node, 200x200
bilinear, 128x128 fields, 64..256 fleets) and tests (a few to a few dozen
elements a side).  Tolerances are tight enough for the temperature to be fixed
to about 1e-11, whatever path the iteration takes there.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from nonlocal_gb300 import thermal as T

TOL = 1e-12
STEP_TOL = 1e-13       # a step's right-hand side holds the fixed temperatures, far larger than its heat terms
MAX_ITER = 100000


# ------------------------------------------------------------------ the cases
def _steady(name, nx, ny, element, influence, r, p1, cond, *, precision="fp64", coarse=0, bc="ends", jitter=0.2,
            oneshot=True, p=2):
    return dict(name=name, kind="steady", nx=nx, ny=ny, element=element, influence=influence, r=r, p1=p1, cond=cond,
                precision=precision, coarse=coarse, bc=bc, jitter=jitter, oneshot=oneshot, p=p)


def listed():
    return [
        # the benchmark's metric: a fine 8-node mesh, exponential kernel, orthotropic, mixed precision
        # with the coarse space, from the host mesh to the host temperature
        _steady("steady 8-node 300x300", 300, 300, "serendipity", "exponential", 0.05, 0.3, "1,0.1",
                precision="mixed", coarse=1024),
        # the second benchmark workload, inside a parameter study: mesh resident, model and boundaries new
        _steady("steady 4-node 200x200", 200, 200, "bilinear", "fast_polynomial", 0.05, 0.5, "1", precision="mixed",
                coarse=252, bc="flux", jitter=0.0, oneshot=False),
        # the default options (FP64, ILLT) on a mesh as an engineer starts with; full anisotropy, convection, source
        _steady("steady 8-node 71x53 fp64", 71, 53, "serendipity", "polynomial", 0.08, 0.5, "2,1,0.3", bc="convection"),
        # the smallest call: a coarse mesh in a parameter study, where latency counts
        _steady("steady 4-node 17x13 fp64", 17, 13, "bilinear", "fast_polynomial", 0.2, 0.5, "1", bc="flux",
                oneshot=False),
        # the classical limit (no nonlocal part) that every study compares with, default options
        _steady("steady local 151x97 fp64", 151, 97, "bilinear", "fast_polynomial", 0.1, 1.0, "1", bc="convection"),
        # heterogeneous materials: log-normal conductivities, ordered pairs, batched BiCGSTAB
        dict(name="fields 6 x 96x96", kind="fields", count=6, nx=96, ny=96, r=0.05, p1=0.5, precision="mixed"),
        # a heating transient, 8-node, FP64 as the reference
        dict(name="march 8-node 48x37", kind="march", nx=48, ny=37, element="serendipity", influence="exponential",
             r=0.08, p1=0.5, cond="1", steps=10),
        # many transients at once (design of experiments), a dozen of the benchmark's 256
        dict(name="fleet of 12", kind="fleet", count=12, lo=64, hi=160, method="mixed_illt"),
        # nonlocal elasticity with the default solver
        dict(name="plate 8-node 33x26", kind="plate", nx=33, ny=26, element="serendipity", influence="polynomial",
             r=0.1, p1=0.5),
        # post-processing of a solution
        dict(name="flux 8-node 120x90", kind="flux", nx=120, ny=90, element="serendipity", influence="exponential",
             r=0.05, p1=0.4),
        # a caller's own matrices (the reference's CG and its ILLT plug-in)
        dict(name="plugin cg 61x45", kind="plugin", nx=61, ny=45, element="bilinear", influence="fast_polynomial",
             r=0.1, p1=0.5),
        # the 1D solver with its default mesh
        dict(name="rod 1000 quadratic", kind="rod", elements=1000, order=2, r=0.05, p1=0.5, influence="bell", steps=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi):
    n = _log_int(rng, lo, hi)
    return n, max(2, int(round(n * rng.uniform(0.6, 1.3))))


def draw(rng):
    kind = rng.choice(["steady", "steady", "steady", "steady", "fields", "march", "fleet", "plate", "flux", "plugin",
                       "rod"])
    influence = rng.choice(["fast_polynomial", "polynomial", "exponential", "exponential", "constant"])
    element = rng.choice(["bilinear", "serendipity"])
    p1 = round(rng.uniform(0.2, 0.8), 3)
    if kind == "steady":
        precision = rng.choice(["fp64", "mixed"])
        local = rng.random() < 0.15
        # FP64 problems stay in the range where a user waits for them; 8-node elements cost about twenty times as much
        hi = (60 if element == "serendipity" else 110) if precision == "fp64" else (220 if element == "serendipity" else 250)
        nx, ny = _sides(rng, 8, hi)
        reach = rng.uniform(2.0, 12.0)          # radius in elements
        n_nodes = (nx + 1) * (ny + 1) * (3 if element == "serendipity" else 1)
        return dict(kind=kind, nx=nx, ny=ny, element=element, influence=influence,
                    r=round(min(0.3, reach / max(nx, ny)), 4), p1=1.0 if local else p1,
                    cond=rng.choice(["1", "1,0.2", "2,1,0.3"]), precision=precision,
                    coarse=min(1024, max(64, n_nodes // 160)) if precision == "mixed" and rng.random() < 0.5 else 0,
                    bc=rng.choice(["ends", "flux", "convection"]), jitter=rng.choice([0.1, 0.2]),
                    oneshot=rng.random() < 0.5, p=rng.choice([2, 4]))
    if kind == "fields":
        nx, ny = _sides(rng, 12, 100)
        return dict(kind=kind, count=rng.randint(1, 6), nx=nx, ny=ny, r=round(rng.uniform(2.5, 6.0) / max(nx, ny), 4), p1=p1,
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "march":
        nx, ny = _sides(rng, 8, 50)
        return dict(kind=kind, nx=nx, ny=ny, element=element, influence=influence,
                    r=round(min(0.3, rng.uniform(2.0, 6.0) / max(nx, ny)), 4), p1=p1, cond=rng.choice(["1", "1,0.2"]),
                    steps=rng.randint(1, 12))
    if kind == "fleet":
        return dict(kind=kind, count=rng.randint(2, 10), lo=rng.randint(16, 60), hi=rng.randint(64, 150),
                    method=rng.choice(["mixed_illt", "mixed_illt", "identity_fp64"]))
    if kind == "plate":
        nx, ny = _sides(rng, 6, 30)
        return dict(kind=kind, nx=nx, ny=ny, element=element, influence=influence,
                    r=round(min(0.3, rng.uniform(2.0, 5.0) / max(nx, ny)), 4), p1=p1)
    if kind == "flux":
        nx, ny = _sides(rng, 10, 150)
        return dict(kind=kind, nx=nx, ny=ny, element=element, influence=influence,
                    r=round(min(0.3, rng.uniform(2.0, 8.0) / max(nx, ny)), 4), p1=p1)
    if kind == "plugin":
        nx, ny = _sides(rng, 6, 60)
        return dict(kind=kind, nx=nx, ny=ny, element="bilinear", influence="fast_polynomial",
                    r=round(min(0.3, rng.uniform(2.0, 6.0) / max(nx, ny)), 4), p1=p1)
    elements = _log_int(rng, 40, 1000)
    return dict(kind="rod", elements=elements, order=rng.choice([1, 2]),
                r=round(min(0.3, rng.uniform(3.0, 50.0) / elements), 5), p1=rng.choice([p1, p1, 1.0]),
                influence=rng.choice(["bell", "triangle", "normal", "constant"]), steps=rng.choice([0, 0, 5, 20]))


# ------------------------------------------------------------------ inputs
def _mesh(nx, ny, element, jitter, rng):
    """A structured mesh of [0, 1] x [0, ny / nx], nodes row by row, interior corners moved by up to
    jitter x the element size, mid-sides in the middle of their edges."""
    w, h = 1.0, ny / nx
    X, Y = np.meshgrid(np.linspace(0.0, w, nx + 1), np.linspace(0.0, h, ny + 1))
    move = rng.uniform(-jitter, jitter, (2, ny - 1, nx - 1)) if jitter > 0.0 else np.zeros((2, ny - 1, nx - 1))
    X[1:-1, 1:-1] += move[0] * (w / nx)
    Y[1:-1, 1:-1] += move[1] * (h / ny)
    if element == "bilinear":
        ids = np.arange((nx + 1) * (ny + 1)).reshape(ny + 1, nx + 1)
        nodes = np.stack([X.ravel(), Y.ravel()], axis=1)
        el = np.stack([ids[:-1, :-1], ids[:-1, 1:], ids[1:, 1:], ids[1:, :-1]], axis=-1).reshape(-1, 4)
        edge = lambda a, b: np.stack([a, b], axis=1)  # noqa: E731
        sides = {"down": edge(ids[0, :-1], ids[0, 1:]), "right": edge(ids[:-1, -1], ids[1:, -1]),
                 "up": edge(ids[-1, 1:], ids[-1, :-1]), "left": edge(ids[1:, 0], ids[:-1, 0])}
        return nodes, el.astype(np.int64), {k: v.astype(np.int64) for k, v in sides.items()}
    gx, gy = np.zeros((2 * ny + 1, 2 * nx + 1)), np.zeros((2 * ny + 1, 2 * nx + 1))
    for g, C in ((gx, X), (gy, Y)):
        g[::2, ::2] = C
        g[::2, 1::2] = 0.5 * (C[:, :-1] + C[:, 1:])
        g[1::2, ::2] = 0.5 * (C[:-1] + C[1:])
    real = np.ones(gx.shape, dtype=bool)
    real[1::2, 1::2] = False
    ids = np.full(gx.shape, -1, dtype=np.int64)
    ids[real] = np.arange(int(real.sum()))
    nodes = np.stack([gx[real], gy[real]], axis=1)
    c = lambda dy, dx: ids[dy:dy + 2 * ny - 1:2, dx:dx + 2 * nx - 1:2].ravel()  # noqa: E731
    el = np.stack([c(0, 0), c(0, 1), c(0, 2), c(1, 2), c(2, 2), c(2, 1), c(2, 0), c(1, 0)], axis=1)

    def edges(line):
        return np.stack([line[:-2:2], line[1:-1:2], line[2::2]], axis=1)

    sides = {"down": edges(ids[0]), "right": edges(ids[:, -1]), "up": edges(ids[-1, ::-1]), "left": edges(ids[::-1, 0])}
    return nodes, el, sides


def _profile(points, rng, base, swing):
    """A smooth boundary temperature: base + a few random harmonics along the unit square."""
    v = np.full(points.shape[:-1], base)
    for k in (1, 2, 3):
        a, b, c = rng.uniform(-1.0, 1.0, 3)
        v = v + swing / k * (a * np.sin(k * math.pi * points[..., 0]) + b * np.cos(k * math.pi * points[..., 0])
                             + c * np.cos(k * math.pi * points[..., 1]))
    return v


def _heat_setup(case, seed):
    """Mesh, boundaries and source of a heat problem: plain arrays and numbers."""
    rng = np.random.default_rng(seed)
    nodes, el, sides = _mesh(case["nx"], case["ny"], case["element"], case.get("jitter", 0.15), rng)
    bc, src = [], 0.0
    kind = case.get("bc", "ends")
    if kind == "ends":
        for side, base in (("up", 2.0), ("down", 1.0)):
            bc.append(dict(side=side, kind="temperature", values=_profile(nodes[sides[side]], rng, base, 0.3)))
    elif kind == "flux":
        bc.append(dict(side="left", kind="temperature", values=_profile(nodes[sides["left"]], rng, 1.0, 0.2)))
        bc.append(dict(side="right", kind="flux", flux=float(rng.uniform(0.5, 1.5))))
    else:
        bc.append(dict(side="left", kind="temperature", values=_profile(nodes[sides["left"]], rng, 1.0, 0.2)))
        bc.append(dict(side="right", kind="convection", h=float(rng.uniform(1.0, 4.0)), ambient=float(rng.uniform(1.5, 2.5))))
        src = float(rng.uniform(0.5, 2.0))
    return dict(nodes=nodes, elements=el, sides=sides, bc=bc, source=src)


def _q(influence):
    return 0.5 if influence == "exponential" else 1.0


def _conductivity(text):
    return tuple(float(v) for v in text.split(","))


def _model(case):
    return T.Model2D(influence=case["influence"], radius=(case["r"], case["r"]), local_weight=case["p1"], n=2,
                     p=case.get("p", 2), q=_q(case["influence"]), conductivity=_conductivity(case.get("cond", "1")))


def _boundary(b, sides):
    if b["kind"] == "temperature":
        return T.Boundary(edges=sides[b["side"]], kind="temperature", node_values=b["values"])
    if b["kind"] == "flux":
        return T.Boundary(edges=sides[b["side"]], kind="flux", value=b["flux"])
    return T.Boundary(edges=sides[b["side"]], kind="convection", heat_transfer=b["h"], ambient_temperature=b["ambient"])


def _field(points, seed):
    """A log-normal conductivity: exp of a few random plane waves of correlation length about 0.1."""
    rng = np.random.default_rng(seed + 77)
    g = np.zeros(points.shape[:-1])
    for _ in range(24):
        k = rng.normal(0.0, 8.0, 2)
        g += np.cos(points @ k + rng.uniform(0.0, 2.0 * math.pi))
    return np.exp(0.5 * g / math.sqrt(12.0))


def _fleet_specs(case):
    rng = np.random.default_rng([case["count"], case["lo"], case["hi"]])
    return [(int(rng.integers(case["lo"], case["hi"] + 1)), float(rng.uniform(0.03, 0.1))) for _ in range(case["count"])]


def _bilinear_points(nodes, el):
    """Quadrature coordinates [E][4][2] of bilinear elements."""
    return np.einsum("iq,eid->eqd", _tables("bilinear")[0], nodes[el])


def _rod_args(case, seed):
    rng = np.random.default_rng(seed)
    return dict(left=float(rng.uniform(-1.0, 1.0)), right=float(rng.uniform(0.5, 1.5)),
                conductivity=float(rng.uniform(0.5, 2.0)), initial=float(rng.uniform(0.0, 1.0)))


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("steady", "march", "flux", "plugin"):
        s["setup"] = _heat_setup(case, seed)
        s["model"] = _model(case)
        s["boundaries"] = [_boundary(b, s["setup"]["sides"]) for b in s["setup"]["bc"]]
    if kind == "steady" and not case["oneshot"]:
        s["problem"] = T.Problem2D(case["element"], s["setup"]["nodes"], s["setup"]["elements"])
    elif kind == "march":
        p = s["problem"] = T.Problem2D(case["element"], s["setup"]["nodes"], s["setup"]["elements"])
        p.set_model(s["model"])
        p.set_capacity(1.0, 1.0)
        for b in s["boundaries"]:
            p.add_boundary(b)
        rng = np.random.default_rng(seed + 1)
        s["initial"] = _profile(s["setup"]["nodes"], rng, 0.5, 0.1)
        s["values"] = [float(v) for v in rng.uniform(0.5, 1.5, case["steps"])]
    elif kind == "flux":
        p = s["problem"] = T.Problem2D(case["element"], s["setup"]["nodes"], s["setup"]["elements"])
        p.set_model(s["model"])
        s["temperature"] = _profile(s["setup"]["nodes"], np.random.default_rng(seed + 1), 1.0, 0.5)
    elif kind == "plugin":
        p = s["problem"] = T.Problem2D(case["element"], s["setup"]["nodes"], s["setup"]["elements"])
        p.set_model(s["model"])
        for b in s["boundaries"]:
            p.add_boundary(b)
        p.conductivity_matrix("FULL")
        p.conductivity_matrix("LOCAL")
        s["matrix"], s["local"], s["rhs"] = p.matrix("inner"), p.matrix("local"), p.rhs()[0]
    elif kind == "fields":
        s["problems"] = []
        for k in range(case["count"]):
            c = dict(case, element="bilinear", jitter=0.1, bc="flux")
            u = _heat_setup(c, seed + 1000 * k)
            p = T.Problem2D("bilinear", u["nodes"], u["elements"])
            p.set_model(T.Model2D(influence="fast_polynomial", radius=(case["r"], case["r"]), local_weight=case["p1"]))
            p.set_conductivity_field(_field(_bilinear_points(u["nodes"], u["elements"]), seed + 1000 * k))
            for b in u["bc"]:
                p.add_boundary(_boundary(b, u["sides"]))
            p.set_assembly_precision("ff" if case["precision"] == "mixed" else "auto")
            p.find_neighbours()
            s["problems"].append(p)
    elif kind == "fleet":
        solvers = []
        rng = np.random.default_rng(seed + 5)
        for edges, r in _fleet_specs(case):
            nodes, el, sides = _mesh(edges, edges, "bilinear", 0.0, rng)
            p = T.Problem2D("bilinear", nodes, el)
            p.set_model(T.Model2D(influence="fast_polynomial", radius=(r, r), local_weight=0.5))
            p.add_boundary(T.Boundary(edges=sides["left"], kind="temperature", value=0.0))
            p.set_assembly_precision("ff")
            p.set_assembly_warps(32)
            p.find_neighbours()
            solver = T.NonstationaryHeatEquationSolver2D(p, 1e-3)
            solver.compute(_profile(nodes, rng, 0.0, 0.1))
            solvers.append(solver)
        s["batch"] = T.BatchNonstationary(solvers)
        s["batch"].set_method(case["method"])
        s["phase"], s["step"] = float(rng.uniform(0.0, 2.0 * math.pi)), 0
    elif kind == "plate":
        rng = np.random.default_rng(seed)
        nodes, el, sides = _mesh(case["nx"], case["ny"], case["element"], 0.15, rng)
        s["problem"] = T.MechanicalProblem2D(case["element"], nodes, el)
        s["model"] = _model(dict(case, cond="1"))
        s["elastic"] = T.ElasticParameters("isotropic", (210.0,), (float(rng.uniform(0.2, 0.35)),))
        s["load"] = (float(rng.uniform(0.5, 1.5)), float(rng.uniform(-0.5, 0.5)))
        s["mesh"] = (nodes, el, sides)
        s["boundaries"] = [
            T.MechanicalBoundary(sides["left"], x=("displacement", 0.0), y=("displacement", 0.0)),
            T.MechanicalBoundary(sides["right"], x=("pressure", s["load"][0]), y=("pressure", s["load"][1]))]
    elif kind == "rod":
        s["context"] = T.Context()
        s["args"] = _rod_args(case, seed)
    return s


def _solve_steady(p, s):
    """stationary_heat_equation_solver_2d with the solve options it does not pass on."""
    case = s["case"]
    p.set_model(s["model"])
    p.clear_boundaries()
    for b in s["boundaries"]:
        p.add_boundary(b)
    if s["setup"]["source"]:
        p.set_source(s["setup"]["source"])
    t, _ = p.stationary(tolerance=TOL, max_iterations=MAX_ITER, precision=case["precision"],
                        coarse_aggregates=case["coarse"])
    return t


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "steady":
        if not case["oneshot"]:
            return _solve_steady(s["problem"], s)
        p = T.Problem2D(case["element"], s["setup"]["nodes"], s["setup"]["elements"])
        t = _solve_steady(p, s)
        p.close()
        return t
    if kind == "fields":
        for p in s["problems"]:
            p.conductivity_matrix("FULL")
        return T.solve_assembled_batch(s["problems"], tolerance=TOL, max_iterations=MAX_ITER, precision=case["precision"])[0]
    if kind == "march":
        solver = T.NonstationaryHeatEquationSolver2D(s["problem"], 1e-3)
        solver.compute(s["initial"])
        for v in s["values"]:
            t = solver.calc_step(v, tolerance=STEP_TOL)
        return t
    if kind == "fleet":
        s["step"] += 1
        batch = s["batch"]
        batch.step(np.full(case["count"], math.sin(0.3 * s["step"] + s["phase"])), tolerance=STEP_TOL)
        return [batch.temperature(k) for k in range(case["count"])]
    if kind == "plate":
        return T.equilibrium_equation(s["problem"], s["model"], s["elastic"], s["boundaries"], tolerance=TOL,
                                      max_iterations=MAX_ITER)[0]
    if kind == "flux":
        return s["problem"].calc_flux(s["temperature"])
    if kind == "plugin":
        return T.conjugate_gradient(s["problem"], s["matrix"], s["rhs"], preconditioner_csr=s["local"], tolerance=TOL,
                                    max_iterations=MAX_ITER)[0]
    a = s["args"]
    if not case["steps"]:
        return T.stationary_heat_equation_solver_1d(s["context"], case["elements"], case["order"], 1.0, case["r"],
                                                    case["p1"], case["influence"], a["conductivity"], a["left"], a["right"])
    solver = T.NonstationaryHeatEquationSolver1D(s["context"], case["elements"], case["order"], 1.0, case["r"],
                                                 case["p1"], case["influence"], a["conductivity"], 1.0, 1.0, 1e-3)
    solver.compute(("temperature", a["left"]), ("flux", a["right"]), np.full(solver.n, a["initial"]))
    for _ in range(case["steps"]):
        t = solver.calc_step()
    return t


# ------------------------------------------------------------------ what a pass cannot do without
def _sizes(nx, ny, element, r):
    e = nx * ny
    n = (nx + 1) * (ny + 1) + (nx * (ny + 1) + ny * (nx + 1) if element == "serendipity" else 0)
    reach = r * nx + 1.5                         # widened radius in elements
    per = min(float(e), math.pi * reach * reach)
    return e, n, e * per, n * min(float(n), math.pi * reach * reach * n / e)


PAIR = {"bilinear": 2 * 2 * (4 * 4 * 4 + 4 * 4 * 4), "serendipity": 2 * 2 * (9 * 9 * 8 + 8 * 9 * 8)}


def work(case):
    """Inputs and outputs once; for a solve also its matrix, written once and read once (upper triangle,
    12 bytes an entry), and the pair integrals, each unordered pair once."""
    kind = case["kind"]
    if kind == "rod":
        n, bw = case["elements"] * case["order"] + 1, (round(case["r"] * case["elements"]) + 1) * case["order"]
        if case["p1"] >= 0.999:
            bw = case["order"]
        return {"bytes": 16 * n * (bw + 1), "flops": n * bw * bw + 4 * n * bw * max(1, case["steps"])}
    if kind == "fleet":
        b = f = 0.0
        for edges, r in _fleet_specs(case):
            _, n, _, nnz = _sizes(edges, edges, "bilinear", r)
            b += 12 * nnz / 2 + 32 * n
            f += 2 * nnz
        return {"bytes": b, "flops": f}
    element = case.get("element", "bilinear")
    e, n, pairs, nnz = _sizes(case["nx"], case["ny"], element, case["r"])
    nen = 4 if element == "bilinear" else 8
    mesh = 16 * n + 8 * nen * e
    if case["p1"] >= 0.999:
        pairs, nnz = float(e), 3.0 * nen * n
    flops = pairs / 2 * PAIR[element]
    if kind == "flux":
        nq = 4 if element == "bilinear" else 9
        return {"bytes": mesh + 24 * n, "flops": pairs * nq * nq * 8}
    if kind == "plugin":
        return {"bytes": 16 * nnz / 2 + 24 * n, "flops": 2 * nnz}
    if kind == "fields":
        return {"bytes": case["count"] * (8 * n + 24 * nnz), "flops": case["count"] * 2 * flops}
    if kind == "plate":
        return {"bytes": mesh + 16 * n + 4 * 12 * nnz, "flops": 4 * flops}
    return {"bytes": mesh + 8 * n + 12 * nnz, "flops": flops}


# ------------------------------------------------------------------ the same in 64 bits, plainly
def _tables(element):
    """Values and derivatives of the shape functions at the Gauss points (index ix * m + iy), the weights, and the
    values at the centre."""
    if element == "bilinear":
        g, w = np.array([-1.0, 1.0]) / math.sqrt(3.0), np.ones(2)
        corners = [(-1, -1), (1, -1), (1, 1), (-1, 1)]

        def shape(x, y):
            return np.array([[(1 + a * x) * (1 + b * y) / 4, a * (1 + b * y) / 4, b * (1 + a * x) / 4] for a, b in corners])
    else:
        g, w = np.array([-1.0, 0.0, 1.0]) * math.sqrt(0.6), np.array([5.0, 8.0, 5.0]) / 9.0
        a, b, c = 1.0, 5.0, -3.0                 # 9 p - 1, 9 p + 3, 9 p - 5 with p = 2 / 9
        places = [(-1, -1), (0, -1), (1, -1), (1, 0), (1, 1), (0, 1), (-1, 1), (-1, 0)]

        def shape(x, y):
            rows = []
            for s, t in places:
                if s and t:
                    u, v, k = 1 + s * x, 1 + t * y, a * (1 - s * x - t * y) + s * t * b * x * y
                    rows.append([u * v * k / 16, (s * v * k + u * v * (s * t * b * y - s * a)) / 16,
                                 (t * u * k + u * v * (s * t * b * x - t * a)) / 16])
                elif t:
                    v, k = 1 + t * y, c - t * b * y
                    rows.append([-(1 - x * x) * v * k / 16, 2 * x * v * k / 16, -(1 - x * x) * (t * k - t * b * v) / 16])
                else:
                    u, k = 1 + s * x, c - s * b * x
                    rows.append([-(1 - y * y) * u * k / 16, -(1 - y * y) * (s * k - s * b * u) / 16, 2 * y * u * k / 16])
            return np.array(rows)
    at = np.stack([shape(x, y) for x in g for y in g], axis=-1)       # [i][value, d/dx, d/dy][q]
    return at[:, 0], at[:, 1], at[:, 2], np.outer(w, w).ravel(), shape(0.0, 0.0)[:, 0]


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Fem:
    """Quadrature data and neighbours of a mesh, in 64 bits on `device`."""

    def __init__(self, element, nodes, el, r, device):
        N, Nx, Ny, w, centre = (torch.tensor(t, dtype=torch.float64, device=device) for t in _tables(element))
        self.el = torch.tensor(el, device=device)
        x = torch.tensor(nodes, dtype=torch.float64, device=device)
        self.n, self.N, self.w = x.shape[0], N, w
        xe = x[self.el]                                                # [e][i][2]
        self.q = torch.einsum("iq,eid->eqd", N, xe)
        J = torch.stack([torch.einsum("iq,eid->eqd", Nx, xe), torch.einsum("iq,eid->eqd", Ny, xe)], dim=-1)
        self.jac = (J[..., 0, 0] * J[..., 1, 1] - J[..., 0, 1] * J[..., 1, 0]).abs()
        gx = Nx * J[:, None, :, 1, 1] - Ny * J[:, None, :, 1, 0]
        gy = -Nx * J[:, None, :, 0, 1] + Ny * J[:, None, :, 0, 0]
        self.g = torch.stack([gx, gy], dim=-1)                         # [e][i][q][2], times |J|
        self.c = torch.einsum("i,eid->ed", centre, xe)
        share = torch.zeros(el.shape[0], self.n, device=device)
        share.scatter_(1, self.el, 1.0)
        share = share @ share.T > 0
        d = torch.cdist(self.c, self.c, compute_mode="donot_use_mm_for_euclid_dist")
        self.R = r + float(d[share].max())
        self.near = d <= self.R

    def phi(self, influence, r, p, part):
        """The normalised influence between the points of elements `part` and all others: [c][q][e][q']."""
        z = (self.q[part][:, :, None, None] - self.q[None, None]) / r
        d = (z * z).sum(-1)
        q = _q(influence)
        if influence == "fast_polynomial":
            return torch.clamp(1 - d, min=0.0) * (2 / (math.pi * r * r))
        if influence == "constant":
            return (d <= 1).to(d) * (math.gamma(2) / (4 * r * r * math.gamma(1.5) ** 2))
        beta = lambda a, b: math.gamma(a) * math.gamma(b) / math.gamma(a + b)  # noqa: E731
        dp = d ** (p // 2)
        if influence == "polynomial":
            norm = 2 * p / (4 * r * r * beta(0.5, 0.5) * beta(2 / p, q + 1))
            return torch.where(d < 1, (1 - dp) ** int(q), torch.zeros_like(d)) * norm
        norm = 2 * p * 2.0 * q ** (2 / p) / (8 * r * r * math.gamma(2 / p) * beta(0.5, 0.5))
        return torch.exp(-q * dp) * norm

    def _add(self, K, block, part):
        """block [c][i][e][j] into the rows of the part's nodes."""
        c, nen = block.shape[0], block.shape[1]
        rows = torch.zeros(c * nen, self.n, dtype=torch.float64, device=K.device)
        rows.index_add_(1, self.el.reshape(-1), block.reshape(c * nen, -1))
        K.index_add_(0, self.el[part].reshape(-1), rows)

    def gradients(self, influence, r, p1, p, pairs, lam=None):
        """For each (a, b) of `pairs` the matrix p1 int dN_i/da dN_j/db + (1 - p1) int int phi dN_i/da dN_j/db
        (lam: a factor at the second point)."""
        E = self.el.shape[0]
        gw = self.g * self.w[None, None, :, None]
        lam = torch.ones_like(self.jac) if lam is None else lam
        K = [torch.zeros(self.n, self.n, dtype=torch.float64, device=self.q.device) for _ in pairs]
        chunk = max(1, int(2.5e8 / (E * self.q.shape[1] ** 2 * 8)))
        for s in range(0, E, chunk):
            part = slice(s, min(E, s + chunk))
            if p1 < 0.999:
                f = self.phi(influence, r, p, part) * (1 - p1) * self.near[part][:, None, :, None]
                h = torch.einsum("cqep,ejpd->cqejd", f, gw * lam[:, None, :, None])
            for k, (a, b) in enumerate(pairs):
                own = p1 * torch.einsum("ciq,cjq->cij", gw[part][..., a] * (lam / self.jac)[part][:, None], self.g[part][..., b])
                if p1 < 0.999:
                    block = torch.einsum("ciq,cqej->ciej", gw[part][..., a], h[..., b])
                    self._add(K[k], block, part)
                i = self.el[part][:, :, None].expand(-1, -1, own.shape[2]).reshape(-1)
                j = self.el[part][:, None, :].expand(-1, own.shape[1], -1).reshape(-1)
                K[k].view(-1).index_add_(0, i * self.n + j, own.reshape(-1))
        return K

    def conductivity(self, case, cond, lam=None):
        l = (cond[0], cond[0], 0.0) if len(cond) == 1 else (cond[0], cond[1], 0.0) if len(cond) == 2 else cond
        pairs = [(0, 0), (1, 1)] + ([(0, 1), (1, 0)] if l[2] else [])
        G = self.gradients(case.get("influence", "fast_polynomial"), case["r"], case["p1"], case.get("p", 2), pairs, lam)
        K = l[0] * G[0] + l[1] * G[1]
        return K + l[2] * (G[2] + G[3]) if l[2] else K

    def vector(self, value):
        """int value N_i."""
        f = torch.zeros(self.n, dtype=torch.float64, device=self.q.device)
        return f.index_add_(0, self.el.reshape(-1), (value * torch.einsum("iq,eq->ei", self.N * self.w, self.jac)).reshape(-1))

    def mass(self):
        m = torch.einsum("iq,jq,eq->eij", self.N * self.w, self.N, self.jac)
        C = torch.zeros(self.n, self.n, dtype=torch.float64, device=self.q.device)
        i = self.el[:, :, None].expand(-1, -1, m.shape[2]).reshape(-1)
        j = self.el[:, None, :].expand(-1, m.shape[1], -1).reshape(-1)
        C.view(-1).index_add_(0, i * self.n + j, m.reshape(-1))
        return C


def _edge_integrals(nodes, edges):
    """int N_i [k][i] and int N_i N_j [k][i][j] over line elements (one Gauss point for 2 nodes, two for 3)."""
    if edges.shape[1] == 2:
        N, D, w = np.array([[0.5], [0.5]]), np.array([[-0.5], [0.5]]), np.array([2.0])
    else:
        x, w = np.array([-1.0, 1.0]) / math.sqrt(3.0), np.ones(2)
        N, D = np.array([x * (x - 1) / 2, 1 - x * x, x * (x + 1) / 2]), np.array([x - 0.5, -2 * x, x + 0.5])
    length = np.linalg.norm(np.einsum("iq,kid->kqd", D, nodes[edges]), axis=-1)
    return np.einsum("iq,q,kq->ki", N, w, length), np.einsum("iq,jq,q,kq->kij", N, N, w, length)


def _heat_system(case, setup, fem, cond, lam=None):
    """K, f, the temperature nodes' mask and values."""
    dev = fem.q.device
    K = fem.conductivity(case, cond, lam)
    f = fem.vector(setup["source"])
    fixed = torch.zeros(fem.n, dtype=torch.bool, device=dev)
    xd = torch.zeros(fem.n, dtype=torch.float64, device=dev)
    for b in setup["bc"]:
        edges = setup["sides"][b["side"]]
        at = torch.tensor(edges.ravel(), device=dev)
        if b["kind"] == "temperature":
            fixed[at] = True
            xd[at] = torch.tensor(b["values"].ravel(), dtype=torch.float64, device=dev)
            continue
        one, two = (torch.tensor(v, dtype=torch.float64, device=dev) for v in _edge_integrals(setup["nodes"], edges))
        f.index_add_(0, at, (one * (b["flux"] if b["kind"] == "flux" else b["h"] * b["ambient"])).reshape(-1))
        if b["kind"] == "convection":
            e = torch.tensor(edges, device=dev)
            m = e.shape[1]
            K.view(-1).index_add_(0, (e[:, :, None] * fem.n + e[:, None, :]).reshape(-1), (b["h"] * two).reshape(-1))
    return K, f, fixed, xd


def _eliminate(K, f, fixed, xd):
    free = ~fixed
    x = xd.clone()
    A = K[free][:, free]
    b = (f - K @ torch.where(fixed, xd, torch.zeros_like(xd)))[free]
    x[free] = torch.linalg.solve(A, b)
    return x


def _exact_heat(case, seed):
    setup = _heat_setup(case, seed)
    fem = _Fem(case["element"], setup["nodes"], setup["elements"], case["r"], _device())
    if case["kind"] == "flux":
        return _exact_flux(case, setup, fem, seed)
    K, f, fixed, xd = _heat_system(case, setup, fem, _conductivity(case.get("cond", "1")))
    if case["kind"] != "march":
        return _eliminate(K, f, fixed, xd).cpu().numpy()
    rng = np.random.default_rng(seed + 1)
    t = torch.tensor(_profile(setup["nodes"], rng, 0.5, 0.1), dtype=torch.float64, device=fem.q.device)
    free = ~fixed
    # the capacity of the fixed nodes' columns stays out, as in the reference's step
    C = fem.mass() * (free[:, None] & free[None, :])
    dt = 1e-3
    A = torch.linalg.lu_factor((dt * K + C)[free][:, free])
    coupling = dt * K[free][:, fixed].sum(1)
    for v in rng.uniform(0.5, 1.5, case["steps"]):
        b = (dt * f + C @ t)[free] - coupling * float(v)
        t = torch.full_like(t, float(v))
        t[free] = torch.linalg.lu_solve(*A, b[:, None])[:, 0]
    return t.cpu().numpy()


def _exact_flux(case, setup, fem, seed):
    dev = fem.q.device
    t = torch.tensor(_profile(setup["nodes"], np.random.default_rng(seed + 1), 1.0, 0.5), dtype=torch.float64, device=dev)
    local = -torch.einsum("ei,eiqd->eqd", t[fem.el], fem.g) / fem.jac[..., None]
    E = fem.el.shape[0]
    mixed = torch.empty_like(local)
    chunk = max(1, int(2.5e8 / (E * fem.q.shape[1] ** 2 * 8)))
    src = local * (fem.w * fem.jac)[..., None]
    for s in range(0, E, chunk):
        part = slice(s, min(E, s + chunk))
        f = fem.phi(case["influence"], case["r"], 2, part) * fem.near[part][:, None, :, None]
        mixed[part] = case["p1"] * local[part] + (1 - case["p1"]) * torch.einsum("cqep,epd->cqd", f, src)
    area = (fem.w * fem.jac).sum(1)
    m = 2 if case["element"] == "bilinear" else 3
    last = m * m - 1
    # the Gauss point nearest to each local node
    point = [0, last - (m - 1), last, m - 1] if m == 2 else [0, 3, 6, 7, 8, 5, 2, 1]
    num = torch.zeros(fem.n, 2, dtype=torch.float64, device=dev)
    den = torch.zeros(fem.n, dtype=torch.float64, device=dev)
    for i, q in enumerate(point):
        num.index_add_(0, fem.el[:, i], mixed[:, q] * area[:, None])
        den.index_add_(0, fem.el[:, i], area)
    v = (num / den[:, None]).cpu().numpy()
    return np.ascontiguousarray(v[:, 0]), np.ascontiguousarray(v[:, 1])


def _exact_fields(case, seed):
    out = []
    for k in range(case["count"]):
        setup = _heat_setup(dict(case, element="bilinear", jitter=0.1, bc="flux"), seed + 1000 * k)
        fem = _Fem("bilinear", setup["nodes"], setup["elements"], case["r"], _device())
        lam = torch.tensor(_field(_bilinear_points(setup["nodes"], setup["elements"]), seed + 1000 * k),
                           dtype=torch.float64, device=fem.q.device)
        out.append(_eliminate(*_heat_system(case, setup, fem, (1.0,), lam)).cpu().numpy())
    return out


def _exact_plate(case, seed):
    rng = np.random.default_rng(seed)
    nodes, el, sides = _mesh(case["nx"], case["ny"], case["element"], 0.15, rng)
    nu = float(rng.uniform(0.2, 0.35))
    load = (float(rng.uniform(0.5, 1.5)), float(rng.uniform(-0.5, 0.5)))
    fem = _Fem(case["element"], nodes, el, case["r"], _device())
    xx, xy, yx, yy = fem.gradients(case["influence"], case["r"], case["p1"], 2, [(0, 0), (0, 1), (1, 0), (1, 1)])
    h11 = 210.0 / (1 - nu * nu)
    h12, h66 = nu * h11, 0.5 * 210.0 / (1 + nu)
    n = fem.n
    K = torch.zeros(n, 2, n, 2, dtype=torch.float64, device=fem.q.device)
    K[:, 0, :, 0] = h11 * xx + h66 * yy
    K[:, 0, :, 1] = h12 * xy + h66 * yx
    K[:, 1, :, 0] = h12 * yx + h66 * xy
    K[:, 1, :, 1] = h11 * yy + h66 * xx
    one = torch.tensor(_edge_integrals(nodes, sides["right"])[0], dtype=torch.float64, device=fem.q.device)
    f = torch.zeros(n, 2, dtype=torch.float64, device=fem.q.device)
    at = torch.tensor(sides["right"].ravel(), device=fem.q.device)
    for d in range(2):
        f[:, d].index_add_(0, at, (one * load[d]).reshape(-1))
    fixed = torch.zeros(n, 2, dtype=torch.bool, device=fem.q.device)
    fixed[torch.tensor(sides["left"].ravel(), device=fem.q.device)] = True
    x = _eliminate(K.view(2 * n, 2 * n), f.view(-1), fixed.view(-1), torch.zeros(2 * n, dtype=torch.float64, device=f.device))
    return x.view(n, 2).cpu().numpy()


def _exact_rod(case, seed):
    a = _rod_args(case, seed)
    E, order, r, p1 = case["elements"], case["order"], case["r"], case["p1"]
    h, n = 1.0 / E, E * order + 1
    if order == 1:
        g, w = np.array([-1.0, 1.0]) / math.sqrt(3.0), np.ones(2)
        N, D = np.array([(1 - g) / 2, (1 + g) / 2]), np.array([-0.5 + 0 * g, 0.5 + 0 * g])
    else:
        g, w = np.array([-1.0, 0.0, 1.0]) * math.sqrt(0.6), np.array([5.0, 8.0, 5.0]) / 9.0
        N, D = np.array([g * (g - 1) / 2, 1 - g * g, g * (g + 1) / 2]), np.array([g - 0.5, -2 * g, g + 0.5])
    x = (np.arange(E)[:, None] + (g + 1) / 2) * h
    K = np.zeros((n, n))
    at = np.arange(E)[:, None] * order + np.arange(order + 1)
    lam = a["conductivity"]
    own = np.einsum("iq,jq,q->ij", D, D, w) * lam * p1 / (h / 2)
    np.add.at(K, (at[:, :, None], at[:, None, :]), np.broadcast_to(own, (E,) + own.shape))
    if p1 < 0.999:
        reach = math.floor(r / h + 0.5)
        for s in range(-reach, reach + 1):
            e = np.arange(max(0, -s), min(E, E - s))
            d = np.abs(x[e][:, :, None] - x[e + s][:, None, :])
            if case["influence"] == "bell":
                f = np.where(d < r, 0.75 / r * (1 - (d / r) ** 2), 0.0)
            elif case["influence"] == "triangle":
                f = np.where(d < r, (1 - d / r) / r, 0.0)
            elif case["influence"] == "normal":
                f = np.exp(-0.5 * (d / r) ** 2) / (r * math.sqrt(2 * math.pi))
            else:
                f = np.where(d < r, 0.5 / r, 0.0)
            np.add.at(K, (at[e][:, :, None], at[e + s][:, None, :]),
                      (1 - p1) * lam * np.einsum("iq,eqp,jp->eij", D * w, f, D * w))
    if not case["steps"]:
        f = np.zeros(n)
        np.add.at(f, at, np.einsum("iq,eq->ei", N * w, np.sin(math.pi * x)) * h / 2)
        f[-1] += a["right"]
        t = np.empty(n)
        t[0] = a["left"]
        t[1:] = np.linalg.solve(K[1:, 1:], f[1:] - K[1:, 0] * a["left"])
        return t
    C = np.zeros((n, n))
    np.add.at(C, (at[:, :, None], at[:, None, :]), np.broadcast_to(np.einsum("iq,jq,q->ij", N, N, w) * h / 2, (E,) + own.shape))
    dt, t = 1e-3, np.full(n, a["initial"])
    A = np.linalg.inv((dt * K + C)[1:, 1:])
    for _ in range(case["steps"]):
        b = C[1:, 1:] @ t[1:] - dt * K[1:, 0] * a["left"]
        b[-1] += dt * a["right"]
        t = np.concatenate([[a["left"]], A @ b])
    return t


def exact(case, seed):
    kind = case["kind"]
    if kind == "rod":
        return _exact_rod(case, seed) if case["elements"] * case["order"] <= 2500 else None
    if kind == "fleet":
        return None                                     # the state moves on from pass to pass
    element = case.get("element", "bilinear")
    e, n, _, _ = _sizes(case["nx"], case["ny"], element, case["r"])
    if kind == "fields":
        return _exact_fields(case, seed) if e <= 9500 and e * case["count"] <= 60000 else None
    if kind == "flux":
        return _exact_heat(case, seed) if e <= 12000 else None
    if n > 15000 or (e > 4200 and case["p1"] < 0.999):
        return None
    if kind == "plate":
        return _exact_plate(case, seed) if n <= 7000 else None
    return _exact_heat(case, seed)
