"""ib_info.device_bytes counts the memory a handle takes after its creation too."""
import ctypes
import importlib

import numpy as np
import pytest

from _util import Dev

pytestmark = pytest.mark.gpu


def test_bytes_of_operator_calls_and_of_the_ring_tables(ib, lib):
    nx, ny, L = 64, 48, 2
    h = 4.0 / nx
    grid = ib.UniformGrid(h, (-2.0, 2.0), (-1.5, 1.5))
    prob = ib.Problem(ib.StreamFcnFluid(ib.MultiLevel(grid, L), (1.0, 0.0), 100.0), ib.BodyGroup(), ib.SchemeCNAB(0.01))
    s = ib.initsolver(prob, ib.initstate(prob))

    def held():
        info = importlib.import_module("ibgb300._lib").IbInfo()
        assert lib.ib_get_info(s.handle, ctypes.byref(info)) == 0
        return info.device_bytes

    dev, n = Dev(), (nx - 1) * (ny - 1)
    x, y = dev.put(np.ones(3 * n)), dev.empty(3 * n)
    b0 = held()
    for batch, kept in ((1, 1), (2, 2), (1, 2), (3, 2)):  # up to a field per level stays with the handle
        assert lib.ib_op_laplacian_inv(s.handle, batch, dev.p(x), dev.p(y)) == 0
        assert held() == b0 + 8 * n * kept
    b1 = held()
    s.set_vort2flux_order("levels")
    # at least the ring's response to each mode, and its power for the levels above: 8 bytes a value
    nbc = 2 * (nx + 1) + 2 * (ny + 1)
    assert held() > b1 + 2 * 8 * nbc
    b2 = held()
    s.set_vort2flux_order("sequential")
    s.set_vort2flux_order("levels")
    assert held() == b2
    s.close()
