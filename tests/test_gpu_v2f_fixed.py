"""Vort2Flux of all levels at once in fixed point (csrc/solver.cu, csrc/v2f.cu) against the reference's
coarse-to-fine order, FP64 and float-float state."""
import ctypes
import importlib

import numpy as np
import pytest

from _util import Dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    pytest.importorskip("torch")
    return Dev()


def _solve(ib, lib, dev, nx, ny, L, precision, order):
    h = 4.0 / nx
    grid = ib.UniformGrid(h, (-2.0, -2.0 + nx * h), (-0.5 * ny * h, 0.5 * ny * h))
    prob = ib.Problem(ib.StreamFcnFluid(ib.MultiLevel(grid, L), (1.0, 0.0), 100.0), ib.BodyGroup(), ib.SchemeCNAB(0.01))
    st = ib.initstate(prob)
    st._gamma[:] = np.random.default_rng(nx + ny + L).standard_normal(st._gamma.shape)
    s = ib.initsolver(prob, st, precision=precision)
    s.set_vort2flux_order(order)
    if precision == "fp64":  # the operator entry, on arrays and a ring buffer of its own
        gam = dev.put(np.ascontiguousarray(st._gamma).reshape(-1))
        psi, q = dev.empty(gam.numel()), dev.empty(st.qty.q.size)
        assert lib.ib_op_vort2flux(s.handle, dev.p(gam), dev.p(psi), dev.p(q)) == 0
        out = dev.get(psi).reshape(L, -1), dev.get(q).reshape(L, -1)
    else:
        s.vort2flux(st)
        out = np.array(st.qty.psi).reshape(L, -1), np.array(st.qty.q).reshape(L, -1)
    s.close()
    return out


# the smallest axis, axes with modes cut off and with all kept, both orders of a rectangle's axes, lines of
# one and several warps, one to three rings above a ring; so long and narrow that no mode of one axis is kept
@pytest.mark.parametrize("nx,ny,L", [(8, 8, 2), (8, 12, 4), (12, 8, 3), (36, 60, 5), (64, 48, 3), (200, 192, 5), (96, 300, 4),
                                     (300, 96, 4), (256, 256, 2), (600, 400, 3), (1024, 128, 4), (512, 1200, 3),
                                     (8, 768, 4), (1200, 12, 4)])
def test_all_levels_equal_level_by_level(ib, lib, dev, nx, ny, L):
    want = _solve(ib, lib, dev, nx, ny, L, "fp64", "sequential")
    # four line passes a level, each rounding at 2^-53 of its line's largest value, amplified by at most
    # the axis length (the smallest eigenvalue against the values' spread over the modes); float-float
    # keeps 2^-47 of a value
    tol = 4 * L * max(nx, ny) * 2.0 ** -53
    for got, t in ((_solve(ib, lib, dev, nx, ny, L, "fp64", "levels"), tol),
                   (_solve(ib, lib, dev, nx, ny, L, "mixed", "auto"), tol + 2.0 ** -46)):
        for l in range(L):
            top = np.abs(want[0][l]).max()
            assert np.abs(got[0][l] - want[0][l]).max() < t * top, l
            assert np.abs(got[1][l] - want[1][l]).max() < 2 * t * top, l  # a flux is a difference of two psi


# the rule that chooses the order: levels, and the size of the ring transfer on long, narrow grids
@pytest.mark.parametrize("nx,ny,L,order", [(128, 128, 2, 2), (128, 128, 3, 1), (512, 512, 3, 2), (512, 512, 4, 1), (512, 64, 4, 1),
                                           (1024, 64, 4, 2), (64, 1024, 4, 2), (8, 768, 4, 2)])
def test_order_by_size(ib, lib, nx, ny, L, order):
    h = 4.0 / nx
    grid = ib.UniformGrid(h, (-2.0, -2.0 + nx * h), (-0.5 * ny * h, 0.5 * ny * h))
    prob = ib.Problem(ib.StreamFcnFluid(ib.MultiLevel(grid, L), (1.0, 0.0), 100.0), ib.BodyGroup(), ib.SchemeCNAB(0.01))
    s = ib.initsolver(prob, ib.initstate(prob))
    info = importlib.import_module("ibgb300._lib").IbInfo()
    assert lib.ib_get_info(s.handle, ctypes.byref(info)) == 0
    assert info.vort2flux_order == order  # IB_V2F_LEVELS 1, IB_V2F_SEQUENTIAL 2
    s.close()
