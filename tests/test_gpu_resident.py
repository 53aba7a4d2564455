"""The cluster-resident PCG (kernels_resident.cu) against the CPU oracle in the
same DIC order, at the sizes where its split over CTAs and threads changes:
fewer rows than a warp, remainders of the CTAs' chunks, levels wider than the
threads that walk them, rows with more than three entries of a sweep, the
exact DIC inside one CTA and across the cluster.

Tolerances: FP64 runs the oracle's iteration with sums in another order, and
a few correctors amplify their round-off to well below 1e-10; FP32 inner
solves reach the PCG's relTol 0.1 residual with FP32 rounding, so after the
same number of correctors D agrees to about the FP32 unit round-off, 6e-8,
times the condition of a few iterations: 1e-5.
"""
import numpy as np
import pytest

import solids4foam_gb300 as sg
from oracle import pyoracle
from solids4foam_gb300.cases import block_parts, oracle_bcs

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("shape,kw", [
    ((1, 1, 3), dict(renumber="none")),                       # fewer rows than a warp
    ((7, 5, 3), dict(part_size=32, dic_subdomains=True)),     # ragged parts of 32
    ((17, 16, 16), dict(part_size=512, dic_subdomains=True)), # several parts per CTA
    ((24, 24, 18), dict(parts=8)),                            # blocks, uneven last blocks
    ((40, 40, 4), dict(renumber="RCM")),                      # wide levels, exact, one CTA
    ((20, 12, 16), dict(renumber="tiled")),                   # rows of > 3 lower entries
    ((26, 24, 26), dict(renumber="tiled")),                   # exact across the cluster
    ((9, 8, 7), dict(renumber="none", diagonal=True)),
])
@pytest.mark.parametrize("precision", ["FP64", "FP32_REFINE"])
def test_resident_pcg_matches_oracle(ctx, shape, kw, precision):
    kw = dict(kw)
    m = sg.box_mesh(*shape, 1.0, 0.9, 0.8, 0.2, 3)
    t = np.tile([1e5, 2e5, -3e5], (int(m["patch_size"][5]), 1))
    bcs = {"zmin": ("fixedDisplacement", None, None), "zmax": ("solidTraction", t, None)}
    solver = dict(tolerance=1e-9, relTol=0.1, maxIter=1000)
    okw = {}
    if kw.pop("diagonal", False):
        solver["preconditioner"] = "diagonal"
        okw["preconditioner"] = 1
    if "parts" in kw:
        kw["parts"] = block_parts(*shape, kw["parts"])
    model = sg.SolidModel(ctx, m, dict(type="linearElastic", E=70e9, nu=0.3), bcs, solver=solver,
                          outer=dict(nCorrectors=4), precision=precision, **kw)
    D, sig, perf = model.evolve()
    if "parts" in kw:
        okw["dic_domain"] = kw["parts"]
    elif kw.get("dic_subdomains"):
        okw.update(perm=model.permutation(), dic_domain=model.parts())
    else:
        okw["perm"] = model.permutation()
    Do, so, _, po = pyoracle.solve(m, oracle_bcs(m, bcs), E=70e9, nu=0.3, n_correctors=4, **okw)
    assert perf["n_correctors"] == po["n_correctors"] == 4
    tol = 1e-10 if precision == "FP64" else 1e-5
    assert rel(D, Do) < tol and rel(sig, so) < 10 * tol
    if precision == "FP64":
        assert perf["total_lin_iters"] == po["total_lin_iters"]
    model.close()


def test_resident_pcg_with_a_converged_start(ctx):
    """A corrector whose components start below the tolerance runs no
    iteration and leaves D as it is: the loop still converges to 1e-10."""
    m = sg.box_mesh(9, 9, 9, 1.0, 1.0, 1.0, 0.2, 6)
    bcs = {"zmin": ("fixedDisplacement", None, None),
           "zmax": ("solidTraction", None, np.full(int(m["patch_size"][5]), 1e7))}
    model = sg.SolidModel(ctx, m, dict(type="linearElastic", E=70e9, nu=0.3), bcs,
                          outer=dict(nCorrectors=5000, solutionTolerance=1e-10,
                                     alternativeTolerance=1e-11), precision="FP32_REFINE")
    D, sig, perf = model.evolve()
    assert perf["converged"] == 1
    Do, so, _, po = pyoracle.solve(m, oracle_bcs(m, bcs), perm=model.permutation(), E=70e9, nu=0.3,
                                   n_correctors=5000, solution_tol=1e-10, alternative_tol=1e-11)
    assert rel(D, Do) < 1e-6 and rel(sig, so) < 1e-5
    model.close()
