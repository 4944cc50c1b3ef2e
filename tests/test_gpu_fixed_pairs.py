"""Float-float lines of the fixed-point transforms (csrc/dstfx.cuh) at every accepted axis length: a mixed
solve against the FP64 one of the same field, value by value."""
import numpy as np
import pytest

from test_gpu_fixed_dst import LENGTHS

pytestmark = pytest.mark.gpu


def _psi(ib, gamma, nx, ny, precision):
    h = 4.0 / nx
    grid = ib.UniformGrid(h, (-2.0, -2.0 + nx * h), (-0.5 * ny * h, 0.5 * ny * h))
    prob = ib.Problem(ib.StreamFcnFluid(grid, (1.0, 0.0), 100.0), ib.BodyGroup(), ib.SchemeCNAB(0.01))
    st = ib.initstate(prob)
    st._gamma[:] = gamma.reshape(st._gamma.shape)
    s = ib.initsolver(prob, st, precision=precision)
    s.vort2flux(st)
    psi = np.array(st.qty.psi).reshape(ny - 1, nx - 1)
    s.close()
    return psi


@pytest.mark.parametrize("nx,ny", [(n, 8 if k % 2 else 12) for k, n in enumerate(LENGTHS)])
def test_mixed_solve_is_the_fp64_one_rounded(ib, monkeypatch, nx, ny):
    monkeypatch.setenv("IBGB300_AUTOTUNE", "0")
    rng = np.random.default_rng(nx)
    # psi of small values beside one large one in every row; its Laplacian has 47 bits at most, exact in
    # float-float, so that both solves transform the same integers and differ in the last conversion alone
    psi = rng.integers(-2 ** 18, 2 ** 18, (ny - 1, nx - 1)) * 2.0 ** -44
    psi[np.arange(ny - 1), rng.integers(0, nx - 1, ny - 1)] = 1.25 * (-1.0) ** np.arange(ny - 1)
    p = np.pad(psi, 1)
    gamma = 4 * psi - p[1:-1, :-2] - p[1:-1, 2:] - p[:-2, 1:-1] - p[2:, 1:-1]
    want, got = _psi(ib, gamma, nx, ny, "fp64"), _psi(ib, gamma, nx, ny, "mixed")
    np.testing.assert_allclose(want, psi, rtol=0, atol=1e-12)
    # two 24-bit parts, the second rounded
    np.testing.assert_array_less(np.abs(got - want), np.abs(want) * 2.0 ** -47 + 1e-300)
