"""The processor-local PCG loop in one launch, a CTA per part (kernels_part.cu),
against the part kernels a profiled context launches for every iteration: ragged
and tiny parts, rows with more than three entries of a sweep, levels wider than
the threads that walk them, more parts than the device holds at once (where the
part kernels run in both contexts), repeated solves, a context with a short limit
for bounded waits.

Tolerance: none.  Both compute every row by the same operations, and the sums are
compensated ones whose order does not reach the FP32 alpha and beta.
"""
import numpy as np
import pytest

import solids4foam_gb300 as sg
from oracle import pyoracle
from solids4foam_gb300.cases import block_parts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,kw,one_launch", [
    ((26, 26, 26), dict(blocks=8), True),
    ((39, 34, 33), dict(part_size=512), True),
    ((27, 26, 25), dict(part_size=64), True),
    ((26, 26, 26), dict(blocks=8, shuffle=True), True),
    ((26, 26, 26), dict(part_size=16), True),    # (the resident PCG's launch)
    ((28, 28, 28), dict(part_size=1000), True),  # (the resident PCG's launch)
    ((34, 33, 33), dict(part_size=16), False),
])
def test_one_launch_equals_the_part_kernels(shape, kw, one_launch):
    kw = dict(kw)
    m = sg.box_mesh(*shape, 1.0, 0.9, 0.8, 0.2, 3)
    if "blocks" in kw:
        kw["parts"] = block_parts(*shape, kw.pop("blocks"))
    if kw.pop("shuffle", False):
        order = np.random.default_rng(2).permutation(shape[0] * shape[1] * shape[2])
        m = pyoracle.renumber_mesh(m, order)
        kw["parts"] = kw["parts"][order]
    top = np.tile([1e5, 2e5, -3e5], (int(m["patch_size"][5]), 1))
    bcs = {"zmin": ("fixedDisplacement", None, None), "zmax": ("solidTraction", top, None)}
    out = []
    for opts in (dict(spin_limit=1), dict(profile=True)):
        ctx = sg.Context(0, **opts)
        model = sg.SolidModel(ctx, m, dict(type="linearElastic", E=70e9, nu=0.3), bcs,
                              outer=dict(nCorrectors=3), precision="FP32_REFINE",
                              dic_subdomains=True, **kw)
        first = model.evolve()
        model.set_bc(5, "solidTraction", -0.5 * top)
        out.append((first, model.evolve()))
        model.close()
        ctx.close()
    for (D, sig, perf), (Dp, sp, pp) in zip(*out):
        assert perf["total_lin_iters"] == pp["total_lin_iters"] > 30
        # (total_lin_iters counts the three components; an iteration is two launches)
        assert (3 * perf["kernel_launches"] < 2 * perf["total_lin_iters"]) == one_launch
        assert np.array_equal(D, Dp) and np.array_equal(sig, sp)
