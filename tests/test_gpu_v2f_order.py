"""The order of Vort2Flux asked for by IBGB300_V2F and by ib_set_vort2flux_order: one order, one arithmetic."""
import ctypes
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(ib, lib, nx, ny, L, precision, order=None):
    """psi, q and the order in effect."""
    h = 4.0 / nx
    grid = ib.UniformGrid(h, (-2.0, -2.0 + nx * h), (-0.5 * ny * h, 0.5 * ny * h))
    prob = ib.Problem(ib.StreamFcnFluid(ib.MultiLevel(grid, L), (1.0, 0.0), 100.0), ib.BodyGroup(), ib.SchemeCNAB(0.01))
    st = ib.initstate(prob)
    st._gamma[:] = np.random.default_rng(nx + ny + L).standard_normal(st._gamma.shape)
    s = ib.initsolver(prob, st, precision=precision)
    if order:
        s.set_vort2flux_order(order)
    s.vort2flux(st)
    info = importlib.import_module("ibgb300._lib").IbInfo()
    assert lib.ib_get_info(s.handle, ctypes.byref(info)) == 0
    out = np.array(st.qty.psi), np.array(st.qty.q), info.vort2flux_order
    s.close()
    return out


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("order,code", [("levels", 1), ("sequential", 2)])
def test_variable_and_setter_are_the_same(ib, lib, monkeypatch, precision, order, code):
    by_setter = _run(ib, lib, 128, 192, 3, precision, order)
    monkeypatch.setenv("IBGB300_V2F", order)
    by_variable = _run(ib, lib, 128, 192, 3, precision)
    assert by_setter[2] == by_variable[2] == code
    for a, b in zip(by_setter[:2], by_variable[:2]):
        np.testing.assert_array_equal(a, b)


def test_levels_asked_for_without_one_warp_lines(ib, lib, monkeypatch):
    """200 cells have no one-warp lines: the setter refuses the order on a mixed handle, the variable keeps the rule's."""
    rule = _run(ib, lib, 200, 200, 5, "mixed")
    monkeypatch.setenv("IBGB300_V2F", "levels")
    asked = _run(ib, lib, 200, 200, 5, "mixed")
    assert rule[2] == asked[2] == 1
    np.testing.assert_array_equal(rule[0], asked[0])
    with pytest.raises(ib.IBError):
        _run(ib, lib, 200, 200, 5, "mixed", "levels")


def test_order_may_be_asked_for_whatever_the_tuner_chose(ib, lib, monkeypatch):
    want = _run(ib, lib, 256, 256, 3, "mixed", "levels")
    monkeypatch.setenv("IBGB300_AUTOTUNE", "0")
    got = _run(ib, lib, 256, 256, 3, "mixed", "levels")
    assert want[2] == got[2] == 1
    np.testing.assert_array_equal(want[0], got[0])


def test_ensemble_members_keep_the_all_levels_order(ib, lib):
    """Members in the default order of their sizes (all levels at once, the quarter lines of rectangles on a side
    stream) step in an ensemble as alone."""
    W = ib.workloads

    def start():
        runs = []
        for (nx, ny, L), prec in zip([(128, 96, 4), (192, 128, 4), (64, 64, 5), (200, 160, 3)], ["fp64", "mixed"] * 2):
            wl = W.scaled(W.cylinder_small(), nx, ny, nlevels=L)
            prob = wl.problem()
            st = ib.initstate(prob)
            st._gamma[:] = wl.initial_gamma()
            s = ib.initsolver(prob, st, precision=prec)
            s.vort2flux(st)
            runs.append((st, s))
        return runs

    n, want = 6, []
    for st, s in start():
        for i in range(n):
            ib.advance_(st, s, i * 0.01)
        want.append((st.qty.gamma.copy(), s.force_history(n)))
        s.close()
    runs = start()
    ens = ib.Ensemble([s for _, s in runs])
    ens.advance_n(np.arange(n) * 0.01, states=[st for st, _ in runs])
    info = importlib.import_module("ibgb300._lib").IbInfo()
    for (st, s), (gamma, hist) in zip(runs, want):
        assert lib.ib_get_info(s.handle, ctypes.byref(info)) == 0 and info.vort2flux_order == 1
        np.testing.assert_array_equal(st.qty.gamma, gamma)
        np.testing.assert_array_equal(s.force_history(n), hist)
    ens.close()
    for _, s in runs:
        s.close()
