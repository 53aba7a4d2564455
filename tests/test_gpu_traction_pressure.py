"""A patch with traction, pressure and a relaxation factor together: the bits of D and
sigma after a few correctors against recorded ones (golden/traction_pressure.npz: the
kernels that formed cells and boundary faces in one pass, sm_103a, nvcc 13.0).

Tolerance: none.  In t - p n the product may be rounded first or contracted with the
subtraction; the corrector loop amplifies that last bit (4e-9 of D after 60 correctors).
"""
import os

import numpy as np
import pytest

import solids4foam_gb300 as sg
from solids4foam_gb300.cases import block_parts

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "traction_pressure.npz")

CASES = {
    "fp64_diagonal": ((5, 3, 9), "FP64", dict(blocks=9), dict(preconditioner="diagonal", maxIter=3), 20),
    "fp64_exact": ((5, 1, 7), "FP64", dict(renumber="none"), dict(), 8),
    "fp32_local": ((9, 2, 4), "FP32_REFINE", dict(renumber="tiled", dic_subdomains=True), dict(), 5),
}


def solve(ctx, name):
    shape, precision, kw, solver, n = CASES[name]
    kw = dict(kw)
    if "blocks" in kw:
        kw["parts"] = block_parts(*shape, kw.pop("blocks"))
    m = sg.box_mesh(*shape, 1.0, 0.9, 0.8, 0.2, 5)
    rng = np.random.default_rng(5)
    size = int(m["patch_size"][5])
    model = sg.SolidModel(ctx, m, dict(type="linearElastic", E=70e9, nu=0.3),
                          {"zmin": ("fixedDisplacement", np.array([0.0, 1e-5, 0.0]), None),
                           "zmax": ("solidTraction", rng.normal(0.0, 1e6, 3),
                                    rng.uniform(1e5, 1e6, size), 0.5)},
                          solver=solver, outer=dict(nCorrectors=n), precision=precision, **kw)
    D, sig, _ = model.evolve()
    model.close()
    return D, sig


@pytest.mark.parametrize("name", sorted(CASES))
def test_traction_with_pressure_has_the_recorded_bits(ctx, name):
    D, sig = solve(ctx, name)
    with np.load(GOLDEN) as g:
        assert np.array_equal(D.view(np.uint64), g[name + "_D"].view(np.uint64))
        assert np.array_equal(sig.view(np.uint64), g[name + "_sigma"].view(np.uint64))
