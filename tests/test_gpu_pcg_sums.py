"""The global sums of the PCG (w.r, p.Ap) in every form a mesh may run -- the
cluster-resident PCG, the part kernels, the one-launch part loop -- against the
general kernels, and whole runs of some hundred correctors against them.

Tolerance: none.  alpha and beta are rounded to the PCG's value type, so a last bit
of a sum can turn them, and the corrector loop amplifies what follows; every form
adds up in the general kernels' order and precision.
"""
import numpy as np
import pytest

import solids4foam_gb300 as sg
from solids4foam_gb300.cases import block_parts

pytestmark = pytest.mark.gpu

# shape, mesh options, preconditioner: the forms' ranges, ragged parts, ranges of a CTA
# that share a 32-row record, rows a row kernels' grid apart, many tiny parts
FORMS = [
    ((8, 8, 8), dict(renumber="tiled"), "DIC"),
    ((1, 1, 3), dict(renumber="none"), "DIC"),
    ((20, 12, 16), dict(renumber="tiled"), "DIC"),
    ((40, 40, 4), dict(renumber="RCM"), "DIC"),
    ((26, 24, 26), dict(renumber="tiled"), "DIC"),
    ((48, 44, 52), dict(renumber="tiled"), "DIC"),
    ((14, 17, 12), dict(renumber="tiled"), "diagonal"),
    ((25, 24, 26), dict(blocks=8), "diagonal"),
    ((7, 5, 3), dict(part_size=32, dic_subdomains=True), "DIC"),
    ((13, 11, 10), dict(blocks=8), "DIC"),
    ((23, 21, 25), dict(blocks=7), "DIC"),
    ((26, 26, 26), dict(part_size=16, dic_subdomains=True), "DIC"),
    ((28, 28, 28), dict(part_size=1000, dic_subdomains=True), "DIC"),
    ((32, 32, 32), dict(blocks=8), "DIC"),
    ((39, 34, 33), dict(part_size=64, dic_subdomains=True), "DIC"),
    ((41, 39, 37), dict(blocks=8), "DIC"),
    ((61, 59, 57), dict(blocks=8), "DIC"),                            # two rows a lane of p.Ap
    ((34, 33, 33), dict(part_size=16, dic_subdomains=True), "DIC"),   # part kernels
    ((71, 69, 67), dict(part_size=600, dic_subdomains=True), "DIC"),  # three rows a lane
]


def _model(ctx, shape, kw, pre, precision, max_iter=1000, n_corr=1, tol=0.0, scale=1.0, **extra):
    kw = dict(kw)
    if "blocks" in kw:
        kw["parts"] = block_parts(*shape, kw.pop("blocks"))
    m = sg.box_mesh(*shape, 1.0, 0.9, 0.8, 0.2, 3)
    top = scale * np.tile([1e5, 2e5, -3e5], (int(m["patch_size"][5]), 1))
    solver = dict(tolerance=tol, relTol=0.0 if tol == 0.0 else 0.1, maxIter=max_iter)
    if pre == "diagonal":
        solver["preconditioner"] = "diagonal"
    return sg.SolidModel(ctx, m, dict(type="linearElastic", E=70e9, nu=0.3),
                         {"zmin": ("fixedDisplacement", None, None),
                          "zmax": ("solidTraction", top, None)}, solver=solver,
                         outer=dict(nCorrectors=n_corr), precision=precision, **kw, **extra)


@pytest.mark.parametrize("precision", ["FP32_REFINE", "FP64"])
@pytest.mark.parametrize("shape,kw,pre", FORMS)
def test_sums_are_those_of_the_general_kernels(ctx, shape, kw, pre, precision):
    for n_corr, max_iter in ((1, 1), (2, 7), (3, 23)):
        got = []
        for general in (False, True):
            m = _model(ctx, shape, kw, pre, precision, max_iter, n_corr, general_pcg=general)
            D, sig, _ = m.evolve()
            got.append((m.pcg_scalars(), D, sig))
            m.close()
        assert np.isfinite(got[1][0]).all()
        for a, b in zip(*got):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("shape,kw,pre", [
    ((9, 8, 7), dict(renumber="tiled"), "DIC"),
    ((13, 11, 10), dict(blocks=8), "DIC"),
    ((17, 14, 14), dict(part_size=512, dic_subdomains=True), "DIC"),
    ((12, 13, 11), dict(renumber="tiled"), "diagonal"),
    ((27, 26, 28), dict(blocks=8), "DIC"),
])
@pytest.mark.parametrize("precision", ["FP32_REFINE", "FP64"])
def test_long_runs_equal_the_general_kernels(ctx, shape, kw, pre, precision):
    got = []
    for general in (False, True):
        m = _model(ctx, shape, kw, pre, precision, n_corr=200, tol=1e-9, general_pcg=general)
        D, sig, perf = m.evolve()
        got.append((D, sig, np.array([perf["n_correctors"], perf["total_lin_iters"]])))
        m.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("shape,kw,pre", [
    ((26, 24, 26), dict(renumber="tiled"), "DIC"),
    ((24, 24, 24), dict(blocks=8), "DIC"),
    ((24, 24, 24), dict(renumber="tiled"), "diagonal"),
    ((28, 28, 28), dict(blocks=8), "DIC"),
    ((34, 33, 33), dict(part_size=16, dic_subdomains=True), "DIC"),
])
def test_fp32_sums_have_the_range_of_fp64(ctx, shape, kw, pre):
    """A load 2^28 times larger gives 2^28 times the displacement, bit for bit, also
    where w.r and p.Ap exceed what FP32 holds (3.4e38) while the vectors and a
    lane's share of the sum do not: with t = 3e5 2^68 on cells of face area A, a
    loaded cell's r is t A, its term of w.r about 2 (t A)^2 / diag = 2e36, that of
    the 600-1100 loaded cells together 0.8-1.1e39."""
    got = []
    for scale in (2.0 ** 40, 2.0 ** 68):
        m = _model(ctx, shape, kw, pre, "FP32_REFINE", n_corr=3, tol=1e-9, scale=scale)
        D, sig, _ = m.evolve()
        got.append((D / scale, sig / scale))
        m.close()
    m = _model(ctx, shape, kw, pre, "FP32_REFINE", max_iter=1, n_corr=2, scale=scale)
    m.evolve()
    assert np.abs(m.pcg_scalars()[:2]).max() > 3.5e38
    m.close()
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
