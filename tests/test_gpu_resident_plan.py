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


@pytest.mark.parametrize("n", [20, 21, 22, 23])
def test_exact_dic_runs_resident_where_one_cta_is_too_small(ctx, n):
    """FP32: up to 20^3 the rows and the ring of the sweep tables fit one CTA, from 23^3
    on not even the rows; 21^3 and 22^3 lie between and run across the cluster: one launch
    per corrector (total_lin_iters counts three components, a general iteration is five
    launches), with the general kernels' results."""
    m = _model(ctx, n, "FP32_REFINE", "none")
    D, sig, perf = m.evolve()
    assert 3 * perf["kernel_launches"] < 2 * perf["total_lin_iters"]
    m.close()
    m = _model(ctx, n, "FP32_REFINE", "none", general_pcg=True)
    D1, s1, p1 = m.evolve()
    assert 3 * p1["kernel_launches"] > 2 * p1["total_lin_iters"] > 0
    assert np.array_equal(D, D1) and np.array_equal(sig, s1)
    m.close()
