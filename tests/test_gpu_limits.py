"""Error paths of the solves, made on the host through a mesh's limits: waits that run
out, tables that cannot be allocated."""
import ctypes as ct
import time

import numpy as np
import pytest

import solids4foam_gb300 as sg
from solids4foam_gb300 import _lib
from solids4foam_gb300.cases import block_parts

pytestmark = pytest.mark.gpu


def _model(ctx, shape, precision, **kw):
    m = sg.box_mesh(*shape, 1.0, 0.9, 0.8, 0.2, 4)
    top = np.tile([1e5, 2e5, -3e5], (int(m["patch_size"][5]), 1))
    return sg.SolidModel(ctx, m, dict(type="linearElastic", E=70e9, nu=0.3),
                         {"zmin": ("fixedDisplacement", None, None),
                          "zmax": ("solidTraction", top, None)},
                         outer=dict(nCorrectors=3), precision=precision, **kw)


def _solve(model):
    """Status, displacement and perf of a solve, whatever its status."""
    n = model.n_cells
    D, sig, perf = np.zeros((n, 3)), np.zeros((n, 6)), _lib.Perf()
    st = model.L.s4g_solve(model.h, _lib.LIN_GEOM_TOTAL_DISP, 1, D.ctypes.data, sig.ctypes.data,
                           ct.byref(perf))
    return st, D, perf.as_dict()


@pytest.mark.parametrize("precision", ["FP64", "FP32_REFINE"])
def test_a_timed_out_sweep_ends_the_loop_with_its_iteration(ctx, precision):
    """The device loop runs several PCG iterations a pass; the iteration whose waits gave
    up is its last (one iteration of three components)."""
    model = _model(ctx, (16, 16, 16), precision, part_size=64, general_pcg=True)
    st, D, p = _solve(model)
    assert st == _lib.NOT_CONVERGED and p["device_loop"] == 1
    model.set_limit(_lib.LIMIT_SWEEP_POLLS, 1)
    st, _, q = _solve(model)
    assert st == _lib.TIMEOUT and q["total_lin_iters"] <= 3
    model.set_limit(_lib.LIMIT_SWEEP_POLLS, 0)
    st, D2, r = _solve(model)
    assert st == _lib.NOT_CONVERGED and r["total_lin_iters"] == p["total_lin_iters"]
    assert np.array_equal(D, D2)
    model.close()


def test_a_timed_out_part_loop_leaves_the_mesh_usable(ctx):
    """The one-launch part loop with a limit of one poll gives up (its CTAs return by
    themselves) and reports S4G_TIMEOUT; the packets it left behind do not reach the
    next launch, which has the first solve's bits."""
    model = _model(ctx, (28, 27, 26), "FP32_REFINE", parts=block_parts(28, 27, 26, 8))
    st, D, p = _solve(model)
    assert st == _lib.NOT_CONVERGED
    assert 3 * p["kernel_launches"] < 2 * p["total_lin_iters"]  # one launch per corrector
    for again in range(5):
        model.set_limit(_lib.LIMIT_PACKET_POLLS, 1)
        st, _, _ = _solve(model)
        assert st == _lib.TIMEOUT
        model.set_limit(_lib.LIMIT_PACKET_POLLS, 0)
        if again % 2:  # (a new matrix before the next solve)
            model.set_law(dict(type="linearElastic", E=70e9, nu=0.3))
        st, D2, q = _solve(model)
        assert st == _lib.NOT_CONVERGED and q["total_lin_iters"] == p["total_lin_iters"]
        assert np.array_equal(D, D2)
    model.close()


@pytest.mark.parametrize("shape,kw,precision", [
    ((12, 11, 10), dict(renumber="tiled"), "FP64"),
    ((12, 11, 10), dict(renumber="tiled"), "FP32_REFINE"),
    ((13, 11, 10), dict(blocks=8), "FP32_REFINE"),
    ((28, 27, 26), dict(blocks=8), "FP32_REFINE"),
    ((28, 27, 26), dict(blocks=8), "FP64"),
    ((34, 33, 33), dict(part_size=16, dic_subdomains=True), "FP32_REFINE"),
])
def test_a_form_whose_tables_do_not_fit_is_not_used(ctx, shape, kw, precision):
    """Tables that cannot be allocated leave the solve to the general kernels, with the
    same results and no memory kept."""
    kw = dict(kw)
    if "blocks" in kw:
        kw["parts"] = block_parts(*shape, kw.pop("blocks"))
    general = _model(ctx, shape, precision, general_pcg=True, **kw)
    st0, D0, p0 = _solve(general)
    for limit in (1, 100_000):  # the first allocation, a later one
        model = _model(ctx, shape, precision, **kw)
        model.set_limit(_lib.LIMIT_TABLE_BYTES, limit)
        st, D, p = _solve(model)
        assert st == st0 == _lib.NOT_CONVERGED and np.array_equal(D, D0)
        assert p["total_lin_iters"] == p0["total_lin_iters"]
        assert p["kernel_launches"] >= 2 * p["total_lin_iters"] // 3  # launches per iteration
        assert model.info()["device_bytes"] == general.info()["device_bytes"]
        model.close()
    general.close()


@pytest.mark.parametrize("precision,general,timed", [
    ("FP64", True, [True, True, True, True, True]),
    ("FP64", False, [False, False, True, True, True]),   # part kernels: the product's forms
    ("FP32_REFINE", False, [False] * 5),
])
def test_the_autotuner_times_what_the_mesh_runs(ctx, precision, general, timed):
    """(general_pcg switches the autotuner off; the general kernels run here because the
    part kernels' tables may not be allocated.)"""
    model = _model(ctx, (13, 11, 10), precision, parts=block_parts(13, 11, 10, 8))
    if general:
        model.set_limit(_lib.LIMIT_TABLE_BYTES, 1)
    st, _, p = _solve(model)
    assert st == _lib.NOT_CONVERGED
    assert [t > 0 for t in p["tune_us"][:5]] == timed
    model.close()


@pytest.mark.parametrize("precision", ["FP64", "FP32_REFINE"])
@pytest.mark.parametrize("n,kw", [
    (24, dict(blocks=8)), (32, dict(blocks=8)), (24, dict(part_size=16, dic_subdomains=True)),
    (20, dict(renumber="tiled")), (24, dict(renumber="tiled", diagonal=True)),
])
def test_a_request_is_booked_with_what_its_mesh_holds(ctx, n, kw, precision):
    """The server's footprint covers the device bytes of the form that runs, and is not
    more than 1.4 times them (and a fixed 16 MB)."""
    kw = dict(kw)
    solver = dict(preconditioner="diagonal") if kw.pop("diagonal", False) else {}
    if "blocks" in kw:
        kw["parts"] = block_parts(n, n, n, kw.pop("blocks"))
    m = sg.box_mesh(n, n, n, 1.0, 0.9, 0.8, 0.2, 4)
    law = dict(type="linearElastic", E=70e9, nu=0.3)
    bcs = {"zmin": ("fixedDisplacement", None, None), "zmax": ("solidTraction", [0, 0, -1e5], None)}
    args = dict(solver=solver, outer=dict(nCorrectors=2), precision=precision)
    model = sg.SolidModel(ctx, m, law, {"zmin": bcs["zmin"]}, **args, **kw)
    _solve(model)
    held = model.info()["device_bytes"]
    model.close()
    srv = sg.Server(max_slots=1, memory_budget=1 << 36, dry_run=True, dry_run_us_per_kcell=2e4)
    rid = srv.submit(m, law, bcs, **args, **kw)
    t0 = time.time()
    while srv.stats()["running"] == 0 and time.time() - t0 < 10:
        time.sleep(0.001)
    booked = srv.stats()["bytes_in_use"]
    assert srv.result(rid)[0] == _lib.OK
    srv.close()
    assert held <= booked <= 1.4 * held + (16 << 20)
