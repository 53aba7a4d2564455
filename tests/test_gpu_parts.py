"""The part kernels of the processor-local PCG (kernels_part.cu) against the CPU
oracle with the same subdomains: ragged and tiny parts, rows with more than
three entries of a sweep, levels wider than the threads that walk them, parts
of more rows than a thread keeps, several load cases.  A profiled context runs
them on any mesh; an ordinary one beyond the cluster-resident PCG's sizes.

Tolerances: FP64 runs the oracle's iteration with sums in another order, and
a few correctors amplify their round-off to well below 1e-10; FP32 inner
solves agree to about the FP32 unit round-off, 6e-8, times the condition of a
few iterations: 1e-5.
"""
import numpy as np
import pytest

import solids4foam_gb300 as sg
from oracle import pyoracle
from solids4foam_gb300.cases import block_parts, oracle_bcs

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def case(shape, seed=3):
    m = sg.box_mesh(*shape, 1.0, 0.9, 0.8, 0.2, seed)
    t = np.tile([1e5, 2e5, -3e5], (int(m["patch_size"][5]), 1))
    return m, {"zmin": ("fixedDisplacement", None, None), "zmax": ("solidTraction", t, None)}


@pytest.mark.parametrize("shape,kw", [
    ((7, 5, 3), dict(part_size=32)),
    ((17, 15, 10), dict(part_size=512)),
    ((20, 20, 20), dict(part_size=1000)),   # levels of more rows than walking threads
    ((13, 11, 10), dict(blocks=8)),
])
@pytest.mark.parametrize("precision", ["FP64", "FP32_REFINE"])
def test_part_kernels_match_oracle(shape, kw, precision):
    kw = dict(kw)
    m, bcs = case(shape)
    if "blocks" in kw:
        kw["parts"] = block_parts(*shape, kw.pop("blocks"))
    ctx = sg.Context(0, profile=True)
    model = sg.SolidModel(ctx, m, dict(type="linearElastic", E=70e9, nu=0.3), bcs,
                          outer=dict(nCorrectors=4), precision=precision,
                          dic_subdomains=True, **kw)
    D, sig, perf = model.evolve()
    assert perf["kernel_launches_by"]["loc_precond"] > 0
    okw = (dict(dic_domain=kw["parts"]) if "parts" in kw
           else dict(perm=model.permutation(), dic_domain=model.parts()))
    Do, so, _, po = pyoracle.solve(m, oracle_bcs(m, bcs), E=70e9, nu=0.3, n_correctors=4, **okw)
    tol = 1e-10 if precision == "FP64" else 1e-5
    assert rel(D, Do) < tol and rel(sig, so) < 10 * tol
    if precision == "FP64":
        assert perf["total_lin_iters"] == po["total_lin_iters"]
    model.close()
    ctx.close()


@pytest.mark.parametrize("precision,tol", [("FP64", 1e-12), ("FP32_REFINE", 0.0)])
def test_part_kernels_equal_the_resident_pcg(precision, tol):
    """Blocks in a shuffled cell order (up to six entries of a sweep in a row,
    wide levels): the part kernels and the cluster-resident PCG, two
    implementations of the same iteration, agree -- in FP32 to the bit, in FP64
    to the round-off of sums in another order over four correctors."""
    m0, _ = case((12, 12, 12))
    order = np.random.default_rng(2).permutation(12 ** 3)
    m = pyoracle.renumber_mesh(m0, order)
    parts = block_parts(12, 12, 12, 6)[order]
    t = np.tile([1e5, 2e5, -3e5], (int(m["patch_size"][5]), 1))
    bcs = {"zmin": ("fixedDisplacement", None, None), "zmax": ("solidTraction", t, None)}
    out = []
    for profile in (False, True):
        ctx = sg.Context(0, profile=profile)
        model = sg.SolidModel(ctx, m, dict(type="linearElastic", E=70e9, nu=0.3), bcs,
                              outer=dict(nCorrectors=4), precision=precision, parts=parts)
        assert model.info()["local_slots"] == 0
        out.append(model.evolve())
        model.close()
        ctx.close()
    assert out[0][2]["total_lin_iters"] == out[1][2]["total_lin_iters"]
    assert rel(out[0][0], out[1][0]) <= tol and rel(out[0][1], out[1][1]) <= 10 * tol


@pytest.mark.parametrize("precision", ["FP64", "FP32_REFINE"])
def test_part_kernels_beyond_the_resident_sizes(ctx, precision):
    """33^3 cells, ragged blocks: against the oracle, and three load cases in
    one call equal to their single solves bit for bit."""
    m, bcs = case((33, 33, 33))
    parts = block_parts(33, 33, 33, 8)
    model = sg.SolidModel(ctx, m, dict(type="linearElastic", E=70e9, nu=0.3), bcs,
                          outer=dict(nCorrectors=3), precision=precision, parts=parts)
    D, sig, perf = model.evolve()
    Do, so, _, po = pyoracle.solve(m, oracle_bcs(m, bcs), E=70e9, nu=0.3, n_correctors=3,
                                   dic_domain=parts)
    tol = 1e-10 if precision == "FP64" else 1e-5
    assert rel(D, Do) < tol and rel(sig, so) < 10 * tol
    top = bcs["zmax"][1]
    cases = [{"zmin": bcs["zmin"], "zmax": ("solidTraction", f * top, None)} for f in (1.0, -0.5, 3.0)]
    Db, sb, _ = model.evolve_cases(cases)
    assert np.array_equal(Db[0], D) and np.array_equal(sb[0], sig)
    model.set_bc(5, "solidTraction", 3.0 * top)
    D2, s2, _ = model.evolve()
    assert np.array_equal(Db[2], D2) and np.array_equal(sb[2], s2)
    model.close()
