"""The FP64 sine transforms (64-bit block fixed point, csrc/dstfx.cu) against scipy's RODFT00 in
extended precision: every accepted axis length, and the ends of the exponent range."""
import numpy as np
import pytest
from scipy import fft as sfft

from _util import Dev

pytestmark = pytest.mark.gpu

# every length has kernels of its own: each is an axis here, beside one of 8 or 12 cells, and a few pairs
# of long axes
LENGTHS = [n for n in range(8, 2049, 4) if not [1 for p in (7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47)
                                                if n % p == 0]
           and max(q for q in range(1, n + 1) if n % q == 0 and all(q % p for p in (2, 3, 5))) == 1]
SHAPES = [(n, 8 if k % 2 else 12) for k, n in enumerate(LENGTHS)] + [(12 if k % 2 else 8, n) for k, n in enumerate(LENGTHS)]
SHAPES += [(200, 192), (600, 400), (1000, 1024), (768, 2048)]


@pytest.fixture(scope="module")
def dev():
    pytest.importorskip("torch")
    return Dev()


def _solver(ib, nx, ny):
    h = 4.0 / nx
    grid = ib.UniformGrid(h, (-2.0, -2.0 + nx * h), (-0.5 * ny * h, 0.5 * ny * h))
    prob = ib.Problem(ib.StreamFcnFluid(grid, (1.0, 0.0), 100.0), ib.BodyGroup(), ib.SchemeCNAB(0.01))
    return ib.initsolver(prob, ib.initstate(prob))


def _dst2(ib, lib, dev, x):
    s = _solver(ib, x.shape[2] + 1, x.shape[1] + 1)
    dx, dy = dev.put(x), dev.empty(x.size)
    assert lib.ib_op_dst2(s.handle, x.shape[0], dev.p(dx), dev.p(dy)) == 0
    out = dev.get(dy).reshape(x.shape)
    s.close()
    return out


@pytest.mark.parametrize("nx,ny", SHAPES)
def test_error_is_that_of_an_fp64_transform(ib, lib, dev, nx, ny):
    rng = np.random.default_rng(nx * 4096 + ny)
    i, j = np.arange(1, nx)[None, :] / nx, np.arange(1, ny)[:, None] / ny
    g = rng.standard_normal((ny - 1, nx - 1))
    spike = np.zeros_like(g)
    spike[(ny - 1) // 3, (nx - 1) // 2] = 1.0
    x = np.stack([g, np.exp(-((i - 0.3) ** 2 + (j - 0.6) ** 2) / 0.01) + 1e-7 * g, spike, np.sin(np.pi * 3 * i) * j,
                  g * np.exp(12 * rng.standard_normal(g.shape)), np.ones_like(g), 1e-9 * g])
    got = _dst2(ib, lib, dev, x)
    want = sfft.dstn(x.astype(np.longdouble), type=1, axes=(-2, -1))
    # a pass rounds its inputs to 2^-56 of the line's largest and each result to a double: at most
    # 2^-55 sqrt(n) of the result's norm when one entry makes up the line, and the prefix sums of the
    # odd outputs add as much again; two passes, with a factor 4 to spare
    tol = 16 * 2.0 ** -55 * np.sqrt(max(nx, ny))
    for a, b in zip(got, want):
        err = float(np.linalg.norm((a - b).astype(np.float64)) / np.linalg.norm(b.astype(np.float64)))
        assert err < tol, (err, tol)


@pytest.mark.parametrize("nx,ny", [(128, 40), (200, 96)])
def test_scaling_by_powers_of_two_is_exact(ib, lib, dev, nx, ny):
    rng = np.random.default_rng(3)
    x = rng.standard_normal((ny - 1, nx - 1))
    scales = [1.0, 2.0 ** -960, 2.0 ** 980, 2.0 ** -300, 0.0]
    got = _dst2(ib, lib, dev, np.stack([x * s for s in scales]))
    for k, s in enumerate(scales[:4]):
        np.testing.assert_array_equal(got[k], got[0] * s)
    np.testing.assert_array_equal(got[4], np.zeros_like(x))
    # subnormal input and output: the same values rounded at the subnormal spacing, once per pass
    tiny = x * 2.0 ** -1060
    out = _dst2(ib, lib, dev, tiny[None])[0]
    np.testing.assert_allclose(out, sfft.dstn(tiny, type=1), rtol=1e-12, atol=4 * nx * 5e-324)


def test_nonfinite_entries_spoil_their_array_only(ib, lib, dev):
    rng = np.random.default_rng(4)
    x = rng.standard_normal((3, 95, 127))
    x[1, 7, 9] = np.nan
    x[2, 0, 0] = -np.inf
    got = _dst2(ib, lib, dev, x)
    assert np.isfinite(got[0]).all()
    assert np.isnan(got[1]).all() and np.isnan(got[2]).all()
    np.testing.assert_array_equal(got[0], _dst2(ib, lib, dev, x[:1])[0])
