"""The FP32 passes of mixed handles, which IBGB300_DST or refine_sweeps=1 ask for (the solves of other handles run in
fixed point): one and two warps a line, the all-levels Vort2Flux, the predictors, one sweep, the captured CG loop."""
import ctypes
import importlib

import numpy as np
import pytest

from _util import rel
from test_gpu_moving import small_heaving

pytestmark = pytest.mark.gpu


def _steps(ib, lib, wl, n=10, precision="mixed", order=None, **kw):
    """Steps from the workload's start: psi and q of the start, Gamma, forces, and the order in effect."""
    prob = wl.problem()
    st = ib.initstate(prob)
    st._gamma[:] = wl.initial_gamma()
    s = ib.initsolver(prob, st, precision=precision, **kw)
    if order:
        s.set_vort2flux_order(order)
    s.vort2flux(st)
    first = st.qty.psi.copy(), st.qty.q.copy()
    c = []
    for i in range(n):
        ib.advance_(st, s, i * wl.dt)
        c.append([b.CD for b in st.qty.stress] + [b.CL for b in st.qty.stress])
    info = importlib.import_module("ibgb300._lib").IbInfo()
    assert lib.ib_get_info(s.handle, ctypes.byref(info)) == 0
    out = first + (st.qty.gamma.copy(), np.array(c), info.vort2flux_order)
    s.close()
    return out


def _cerr(a, b):
    return np.max(np.abs(a - b) / np.maximum(1.0, np.abs(b)))


def _two_bodies(ib, n=256, L=3):
    return ib.workloads.scaled(ib.workloads.two_body_large(), n, n, nlevels=L)


@pytest.mark.parametrize("order", ["levels", "sequential"])
def test_two_warp_lines_agree_with_one_warp_lines(ib, lib, monkeypatch, order):
    """The same steps to the refinement of their solves, by other kernels (two-warp lines have no all-levels order)."""
    monkeypatch.setenv("IBGB300_DST", "warp")
    monkeypatch.setenv("IBGB300_V2F", order)
    out = {}
    for lanes in ("32", "64"):
        monkeypatch.setenv("IBGB300_LINE_LANES", lanes)
        out[lanes] = _steps(ib, lib, _two_bodies(ib))
    assert out["32"][4] == (1 if order == "levels" else 2) and out["64"][4] == 2
    assert rel(out["64"][2], out["32"][2]) < 1e-9
    assert not np.array_equal(out["64"][2], out["32"][2])


@pytest.mark.parametrize("nx,ny,nl", [(256, 192, 4), (192, 256, 3), (128, 128, 2)])
def test_levels_vort2flux_matches_fp64(ib, lib, monkeypatch, nx, ny, nl):
    wl = ib.workloads.scaled(ib.workloads.cylinder_small(), nx, ny, nlevels=nl)
    want = _steps(ib, lib, wl, 12, "fp64", "sequential")
    monkeypatch.setenv("IBGB300_DST", "warp")
    out = {}
    for order in ("levels", "sequential"):
        out[order] = _steps(ib, lib, wl, 12, order=order)
    lv, sq = out["levels"], out["sequential"]
    assert (lv[4], sq[4]) == (1, 2)
    assert not np.array_equal(lv[0], sq[0])
    for k in range(3):  # psi, q of the initial field; Gamma after 12 steps
        assert rel(lv[k], want[k]) < 1e-10, k
        assert rel(sq[k], want[k]) < 1e-8, k  # (one sweep on the third and coarser levels)
    assert _cerr(lv[3], want[3]) < 1e-8 and _cerr(sq[3], want[3]) < 1e-6


def test_predictors_change_the_solves_not_the_steps(ib, lib, monkeypatch):
    """The trial solve from Gamma_n and the projection from its previous correction, or from zero."""
    monkeypatch.setenv("IBGB300_DST", "warp")
    wl = _two_bodies(ib)
    on = _steps(ib, lib, wl)
    monkeypatch.setenv("IBGB300_CN_PREDICTOR", "0")
    off = _steps(ib, lib, wl)
    assert not np.array_equal(on[2], off[2])
    assert rel(on[2], off[2]) < 1e-9 and _cerr(on[3], off[3]) < 1e-7


@pytest.mark.parametrize("n", [256, 200])
def test_one_sweep(ib, lib, n):
    """refine_sweeps=1, on warp passes and on Stockham passes: C_D and C_L carry about five digits."""
    wl = _two_bodies(ib, n)
    want = _steps(ib, lib, wl, precision="fp64")
    got = _steps(ib, lib, wl, refine_sweeps=1)
    assert not np.array_equal(got[2], _steps(ib, lib, wl)[2])
    assert rel(got[2], want[2]) < 1e-6 and _cerr(got[3], want[3]) < 1e-4


@pytest.mark.parametrize("grid", [(128, 96, 2), (128, 128, 3)])
def test_captured_moving_step_equals_eager(ib, monkeypatch, grid):
    monkeypatch.setenv("IBGB300_DST", "warp")
    wl = small_heaving(ib, nx=grid[0], ny=grid[1], L=grid[2], nsteps=8)
    wl.dt = 0.005
    out = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("IBGB300_NO_GRAPH", mode)
        prob = wl.problem()
        st = ib.initstate(prob)
        st._gamma[:] = wl.initial_gamma()
        s = ib.initsolver(prob, st, precision="mixed")
        s.set_cg_options(tol=1e-10, warm_start="extrapolate")
        s.set_cg_preconditioner("schur_ref")
        s.vort2flux(st)
        for i in range(wl.nsteps):
            ib.advance_(st, s, i * wl.dt)
        out[mode] = (st.qty.gamma.copy(), st.qty.Fb.copy(), s.cg_stats(wl.nsteps)[0])
        s.close()
    for a, b in zip(out["0"], out["1"]):
        np.testing.assert_array_equal(a, b)
