"""The work that a user of this framework has it do, as measurable cases.

Every case goes through the public entry points a program calls:
``SolidModel.evolve`` (one mesh, one load), ``evolve_cases`` (many load cases
on one mesh), ``solve_batch`` (many meshes in one launch), ``Server`` (whole
requests: upload, solve, results), ``step`` (time steps) and the operator
product ``op_amul_dot_noalloc``.  Meshes are the seeded jittered hex boxes
(and the cantilever) of solids4foam_gb300.cases.

Segregated solves take some hundred correctors.  The larger cases stop at
``nCorrectors`` (the results are returned, as the solver does for a run that
reaches it), so that a pass is a stretch of the same correctors that a whole
solve consists of; the smallest ones run to convergence.
"""
from __future__ import annotations

import math

import numpy as np

import solids4foam_gb300 as sg
from solids4foam_gb300.cases import block_parts

SOLVER = dict(tolerance=1e-9, relTol=0.1, maxIter=1000)

# PCG iterations per corrector (relTol 0.1), measured: about this times the
# cells along an edge, by preconditioner
ITERS = {"blocks": 1.1, "tiled": 1.0, "exact": 0.65, "diagonal": 1.6}


def listed():
    return [
        # the smallest request of a served stream, to convergence: latency
        dict(name="cube8_fp64_exact", kind="solve", nx=8, ny=8, nz=8, precision="FP64",
             dic="exact", correctors=400, nu=0.3),
        # a small request on the mixed-precision path over caller blocks, to
        # convergence (ragged: 13 x 11 x 10 cells in blocks of 8)
        dict(name="box13_fp32_blocks", kind="solve", nx=13, ny=11, nz=10,
             precision="FP32_REFINE", dic="blocks", correctors=600, nu=0.28),
        # the 80 x 8 x 8 cantilever in plain FP64 with the serial run's DIC
        dict(name="cantilever_fp64_exact", kind="cantilever", nx=80, ny=8, nz=8,
             precision="FP64", dic="exact", correctors=16, nu=0.3),
        # an odd-sized mesh on the library's own parts
        dict(name="box37_fp32_tiled", kind="solve", nx=37, ny=29, nz=23,
             precision="FP32_REFINE", dic="tiled", correctors=100, nu=0.3),
        # a mid-sized mesh on the mixed-precision path
        dict(name="cube64_fp32_blocks", kind="solve", nx=64, ny=64, nz=64,
             precision="FP32_REFINE", dic="blocks", correctors=40, nu=0.33),
        # the headline mesh: 2.1M cells, mixed precision, 8^3-cell blocks
        dict(name="cube128_fp32_blocks", kind="solve", nx=128, ny=128, nz=128,
             precision="FP32_REFINE", dic="blocks", correctors=20, nu=0.33),
        # plain FP64 of the same form (0.9M cells)
        dict(name="cube96_fp64_blocks", kind="solve", nx=96, ny=96, nz=96,
             precision="FP64", dic="blocks", correctors=10, nu=0.33),
        # the exact DIC's scheduled sweeps on the mixed-precision path
        dict(name="box48_fp32_exact", kind="solve", nx=48, ny=44, nz=52,
             precision="FP32_REFINE", dic="exact", correctors=5, nu=0.3),
        # many load cases on one mesh in one call
        dict(name="loads16_cube40_fp32", kind="loads", nx=40, ny=40, nz=40,
             precision="FP32_REFINE", dic="blocks", correctors=24, nu=0.3, n=16),
        # many meshes of 10-40 cells a side in one launch
        dict(name="batch24_fp32", kind="batch", nx=10, ny=10, nz=40, precision="FP32_REFINE",
             dic="blocks", correctors=40, nu=0.3, n=24),
        # total Lagrangian neoHookean, two load increments, relaxed as the
        # served stream's requests
        dict(name="tl24_fp32_blocks", kind="tl", nx=24, ny=20, nz=22, precision="FP32_REFINE",
             dic="blocks", correctors=40, nu=0.0, n=2),
        # the operator product for callers that must not allocate
        dict(name="amul_dot_47x33x29", kind="amul", nx=47, ny=33, nz=29, precision="FP64",
             dic="exact", correctors=0, nu=0.33),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve", "solve", "solve", "solve", "loads", "batch", "tl", "server",
                       "step", "amul"])
    c = dict(kind=kind, precision=rng.choice(["FP64", "FP32_REFINE"]),
             dic=rng.choice(["blocks", "blocks", "tiled", "exact", "diagonal"]),
             nu=round(rng.uniform(0.2, 0.35), 3), n=1)
    big = 110 if kind == "solve" else 36
    if c["dic"] in ("exact", "diagonal"):
        big = min(big, 56)
    s = size(6, big)
    c.update(nx=max(4, int(s * rng.uniform(0.8, 1.25))), ny=max(4, int(s * rng.uniform(0.8, 1.25))),
             nz=max(4, s))
    if kind in ("loads", "batch", "server"):
        c.update(dic="blocks", precision="FP32_REFINE" if kind != "loads" else c["precision"])
    if kind == "loads":
        c["n"] = rng.randint(2, 24)
    elif kind == "batch":
        c.update(nx=8, ny=8, nz=rng.randint(16, 44), n=rng.randint(3, 24))
    elif kind == "server":
        c.update(nx=6, ny=6, nz=rng.randint(12, 30), n=rng.randint(3, 10))
    elif kind == "tl":
        c.update(dic="blocks", nx=min(c["nx"], 26), ny=min(c["ny"], 26), nz=min(c["nz"], 26),
                 n=rng.randint(1, 3))
    elif kind == "step":
        c.update(n=2)
    elif kind == "amul":
        c.update(precision="FP64", dic="exact", nx=size(6, 62), correctors=0)
    if kind != "amul":
        # as many correctors as about 0.6 s hold
        chain = 9e-6 * (c["nx"] + c["ny"] + c["nz"]) if c["dic"] == "exact" else 0.0
        per = _iters(c) * ((4e-5 + chain) * (c["n"] if kind in ("tl", "step") else 1)
                           + 2.5e-10 * _cells(c) * c["n"])
        c["correctors"] = max(2, min(200, int(0.6 / per)))
    return c


def _cells(c):
    if c["kind"] in ("batch", "server"):  # boxes of nx..nz cells a side
        return ((c["nx"] + c["nz"]) / 2.0) ** 3
    return c["nx"] * c["ny"] * c["nz"]


def _iters(c):
    """PCG iterations of one corrector."""
    edge = (c["nx"] + c["nz"]) / 2.0 if c["kind"] in ("batch", "server") else max(
        c["nx"], c["ny"], c["nz"])
    return max(3.0, ITERS[c["dic"]] * edge)


def _box(c, seed, nx, ny, nz):
    L = float(max(nx, ny, nz))
    return sg.box_mesh(nx, ny, nz, nx / L, ny / L, nz / L, 0.2, seed)


def _request(c, rng, seed, nx, ny, nz):
    """Mesh, law, boundary conditions and controls of one solve: bottom
    fixed, a drawn top traction, E log-uniform in 1-300 GPa."""
    mesh = _box(c, seed, nx, ny, nz)
    outer = dict(nCorrectors=c["correctors"])
    if c["kind"] == "tl":
        mu = rng.uniform(0.5e6, 5e6)
        law = dict(type="neoHookeanElastic", mu=mu, K=mu * rng.uniform(10.0, 20.0))
        tr = np.array([0.0, 0.05 * mu, -0.05 * mu])
        outer.update(fieldRelaxation=0.7, solutionTolerance=1e-7, alternativeTolerance=1e-8)
        top = ("solidTraction", tr, None, 0.5)
    else:
        law = dict(type="linearElastic", E=math.exp(rng.uniform(math.log(1e9), math.log(3e11))),
                   nu=c["nu"])
        top = ("solidTraction", rng.normal(0.0, 1e6, 3), None)
        if c["nu"] > 0.3 and c["correctors"] > 100:  # a long loop needs it to contract
            outer.update(fieldRelaxation=0.7)
    parts = block_parts(nx, ny, nz, 8) if c["dic"] == "blocks" else None
    return dict(mesh=mesh, law=law, bcs={"zmin": ("fixedDisplacement", None, None), "zmax": top},
                outer=outer, parts=parts)


def _options(c, parts):
    kw = dict(precision=c["precision"])
    if parts is not None:
        kw["parts"] = parts
    elif c["dic"] == "tiled":
        kw.update(renumber="tiled", dic_subdomains=True)
    return kw


def _solver(c):
    return dict(SOLVER, preconditioner="diagonal") if c["dic"] == "diagonal" else dict(SOLVER)


def _boxes(c, rng):
    return [tuple(int(v) for v in rng.integers(c["nx"], c["nz"] + 1, 3)) for _ in range(c["n"])]


def prepare(case, seed):
    c, seed = case, int(seed) % (1 << 31)
    rng = np.random.default_rng(seed)
    kind = c["kind"]
    st = dict(case=c)
    if kind == "server":
        st["server"] = sg.Server(0, max_slots=4)
        shapes = _boxes(dict(c), np.random.default_rng(17 * c["n"] + c["nz"]))
        st["requests"] = [_request(c, rng, seed + i, *s) for i, s in enumerate(shapes)]
        return st
    st["ctx"] = ctx = sg.Context(0)
    if kind == "batch":
        # the shapes belong to the case, so that another seed's batch is as much work
        shapes = _boxes(dict(c), np.random.default_rng(17 * c["n"] + c["nz"]))
        st["models"] = []
        for i, s in enumerate(shapes):
            q = _request(c, rng, seed + i, *s)
            st["models"].append(sg.SolidModel(ctx, q["mesh"], q["law"], q["bcs"],
                                              solver=_solver(c), outer=q["outer"],
                                              **_options(c, q["parts"])))
        return st
    if kind == "cantilever":
        mesh = sg.box_mesh(c["nx"], c["ny"], c["nz"], 2.0, 0.2, 0.2, 0.0, 1)
        bcs = {"xmin": ("fixedDisplacement", None, None),
               "xmax": ("solidTraction", np.array([0.0, -1e6, 0.0]) * rng.uniform(0.5, 1.5)
                        + rng.normal(0.0, 1e5, 3), None)}
        st["model"] = sg.SolidModel(ctx, mesh, dict(type="linearElastic", E=200e9, nu=c["nu"]),
                                    bcs, solver=_solver(c), outer=dict(nCorrectors=c["correctors"]),
                                    **_options(c, None))
        return st
    if kind == "amul":
        mesh = _box(c, seed, c["nx"], c["ny"], c["nz"])
        m = sg.SolidModel(ctx, mesh, dict(type="linearElastic", E=70e9, nu=c["nu"]),
                          {"zmin": ("fixedDisplacement", None, None)}, **_options(c, None))
        m.op_matrix()
        st.update(model=m, x=rng.normal(0.0, 1.0, (_cells(c), 3)))
        return st
    q = _request(c, rng, seed, c["nx"], c["ny"], c["nz"])
    kw = _options(c, q["parts"])
    if kind == "tl":
        kw["model"] = "nonLinearGeometryTotalLagrangian"
    st["model"] = sg.SolidModel(ctx, q["mesh"], q["law"], q["bcs"], solver=_solver(c),
                                outer=q["outer"], **kw)
    if kind == "loads":
        st["cases"] = [{"zmin": ("fixedDisplacement", None, None),
                        "zmax": ("solidTraction", rng.normal(0.0, 1e6, 3), None)}
                       for _ in range(c["n"])]
    if kind == "step":
        top = q["bcs"]["zmax"]
        st["steps"] = [{"zmax": (top[0], (i + 1.0) / c["n"] * top[1], None)}
                       for i in range(c["n"])]
    return st


def run(state):
    kind = state["case"]["kind"]
    if kind == "amul":
        return state["model"].op_amul_dot_noalloc(state["x"])
    if kind == "loads":
        D, sig, _ = state["model"].evolve_cases(state["cases"])
        return D, sig
    if kind == "batch":
        return [(D, sig) for D, sig, _ in sg.solve_batch(state["models"])]
    if kind == "server":
        s, c = state["server"], state["case"]
        ids = [s.submit(q["mesh"], q["law"], q["bcs"], solver=_solver(c), outer=q["outer"],
                        precision=c["precision"], parts=q["parts"]) for q in state["requests"]]
        return [s.result(i)[1:3] for i in ids]
    if kind == "step":
        m = state["model"]
        m.reset_state()
        return [m.step(bcs)[:2] for bcs in state["steps"]]
    n = state["case"].get("n", 1) if kind == "tl" else 1
    D, sig, _ = state["model"].evolve(n)
    return D, sig


def work(case):
    """Bytes and operations of one pass: per PCG iteration the matrix (a
    diagonal, three faces a cell with their coefficient and index), the DIC
    factor and the vectors x, r, p read and written, w and q written and read
    once; per corrector the face geometry, D, its gradient and the stress
    in FP64; the results written once."""
    c = case
    N = float(_cells(c))
    if c["kind"] == "amul":
        return {"bytes": N * (8 + 3 * 12 + 6 * 8), "flops": N * 3 * 16}
    v = 4.0 if c["precision"] == "FP32_REFINE" else 8.0
    it = N * (v + 3 * (v + 4) + v + 3 * v * 9)
    corr = N * (3 * 8 * 6 + 8 * 30)
    k = float(c["correctors"])
    many = float(c.get("n", 1) or 1)
    return {"bytes": many * (k * (_iters(c) * it + corr) + N * 72),
            "flops": many * k * N * (_iters(c) * 3 * 40 + 600)}


def exact(case, seed):
    """The operator product in 64 bits: the momentum matrix of the
    segregated solve (Gauss linear corrected, impK = 2 mu + lambda) applied
    to x.  The solves are iterations stopped by their own tests, which have
    no value apart from the iteration."""
    if case["kind"] != "amul":
        return None
    c, seed = case, int(seed) % (1 << 31)
    rng = np.random.default_rng(seed)
    m = _box(c, seed, c["nx"], c["ny"], c["nz"])
    x = rng.normal(0.0, 1.0, (_cells(c), 3))
    E, nu = 70e9, c["nu"]
    gamma = E / (1.0 + nu) + nu * E / ((1.0 + nu) * (1.0 - 2.0 * nu))
    own, nei = m["owner"], m["neighbour"]
    ni, S = nei.shape[0], m["Sf"]
    magS = np.sqrt((S * S).sum(1))
    n = S / magS[:, None]
    d = m["C"][nei] - m["C"][own[:ni]]
    delta = 1.0 / np.maximum((n[:ni] * d).sum(1), 0.05 * np.sqrt((d * d).sum(1)))
    a = gamma * magS[:ni] * delta
    y = np.zeros_like(x)
    flux = a[:, None] * (x[own[:ni]] - x[nei])
    np.add.at(y, own[:ni], flux)
    np.add.at(y, nei, -flux)
    p = list(m["patch_names"]).index("zmin")
    f = np.arange(m["patch_start"][p], m["patch_start"][p] + m["patch_size"][p])
    dn = np.abs((n[f] * (m["Cf"][f] - m["C"][own[f]])).sum(1))
    np.add.at(y, own[f], (gamma * magS[f] / dn)[:, None] * x[own[f]])
    return y, (x * y).sum(0)
