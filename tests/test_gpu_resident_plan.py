"""Plans of the cluster-resident PCG at the sizes where its shared memory runs out:
meshes that fit an SM alone but not twice (batches), exact DIC meshes that do not fit
one CTA's memory with their tables' ring.

Tolerance: none (a batch is the single solves; every form has the general kernels'
bits).
"""
import numpy as np
import pytest

import solids4foam_gb300 as sg

pytestmark = pytest.mark.gpu


def _model(ctx, n, precision, renumber, **kw):
    m = sg.box_mesh(n, n, n, 1.0, 0.9, 0.8, 0.2, 3)
    top = np.tile([1e5, 2e5, -3e5], (int(m["patch_size"][5]), 1))
    return sg.SolidModel(ctx, m, dict(type="linearElastic", E=70e9, nu=0.3),
                         {"zmin": ("fixedDisplacement", None, None),
                          "zmax": ("solidTraction", top, None)},
                         outer=dict(nCorrectors=3), precision=precision, renumber=renumber, **kw)


@pytest.mark.parametrize("precision", ["FP64", "FP32_REFINE"])
def test_batch_of_exact_dic_meshes_equals_the_single_solves(ctx, precision):
    """Exact DIC inside one CTA (16^3-19^3 in the mesh's own order: the rows fit the
    SM's shared memory, not half of it) and across the cluster (26^3)."""
    models = [_model(ctx, n, precision, o) for n, o in
              ((16, "none"), (18, "none"), (19, "none"), (12, "tiled"), (26, "tiled"))]
    batch = sg.solve_batch(models)
    for m, (D, sig, perf) in zip(models, batch):
        D1, s1, p1 = m.evolve()
        assert np.array_equal(D, D1) and np.array_equal(sig, s1)
        assert perf["total_lin_iters"] == p1["total_lin_iters"] > 30
        m.close()
