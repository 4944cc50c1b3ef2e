"""The lines of the fixed-point kernels (csrc/dstfx.cuh) at every accepted axis length are, bit for bit, those of
the same arithmetic in sequence on the host, whose error test_fixed_point.py measures."""
import numpy as np
import pytest

from _util import Dev
from test_fixed_point import _kinds, _ptr, fx  # noqa: F401 (fixture)
from test_gpu_fixed_dst import SHAPES, _dst2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    pytest.importorskip("torch")
    return Dev()


@pytest.mark.parametrize("nx,ny", SHAPES)
def test_lines_are_the_hosts(ib, lib, dev, fx, nx, ny):  # noqa: F811
    rng = np.random.default_rng(nx * 4096 + ny)
    # kinds of lines along the long axis, one after the other across it
    n, m = max(nx, ny), min(nx, ny)
    lines = [np.asarray(y) * rng.uniform(1, 2) for _, y in _kinds(n, rng)]
    x = []
    for k in range(0, len(lines), m - 1):
        f = np.stack([lines[(k + i) % len(lines)] for i in range(m - 1)])
        x.append(f if nx >= ny else f.T)
    x = np.ascontiguousarray(np.stack(x))
    got, want = _dst2(ib, lib, dev, x), np.empty_like(x)
    for a, b in zip(x, want):
        fx.dst2_fixed(nx, ny, _ptr(a), _ptr(b))
    np.testing.assert_array_equal(got, want)
