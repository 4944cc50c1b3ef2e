"""The fixed-point arithmetic of the sine transforms (csrc/fx.cuh), compiled for the host."""
import ctypes
import shutil
import subprocess
import sys
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "immersedboundary.jl_gb300" / "csrc"


def _build(out, *flags):
    cxx = shutil.which("g++") or shutil.which("c++")
    assert cxx, "no C++ compiler"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-x", "c++", "-I", str(CSRC),
                    *flags, str(HERE / "fx_lines.cpp"), "-o", str(out)], check=True)
    return ctypes.CDLL(str(out))


@pytest.fixture(scope="module")
def fx(tmp_path_factory):
    return _build(tmp_path_factory.mktemp("fx") / "fx_lines.so")


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _integers(rng):
    """Integers of every size up to 63 bits, and about every tie of a 24-bit rounding: halves of a unit in the
    last place, and what is dropped after 32 bits around them."""
    v = [int(x) >> int(s) for x, s in zip(rng.integers(1, 2 ** 63 - 1, 4000), rng.integers(0, 63, 4000))]
    for bits in range(25, 64):
        for _ in range(8):
            top = int(rng.integers(2 ** 23, 2 ** 24)) << (bits - 24)
            tie = top + (1 << (bits - 25))
            low = max(bits - 56, 0)
            v += [tie, tie - 1, tie + 1, tie + (1 << low), tie + (255 << low >> 8), tie - (1 << low)]
    v = [x for x in v if 0 < x < 2 ** 63]
    return np.array(v + [-x for x in v] + [0], dtype=np.int64)


@pytest.mark.parametrize("q", [0, 55, 100, -60])
def test_float_float_is_the_nearest(fx, q):
    v = _integers(np.random.default_rng(q + 1000))
    hi, r, e = np.empty(v.size, np.uint32), np.empty(v.size, np.int32), np.empty(v.size, np.int32)
    fx.to_pair(v.size, _ptr(v), q, _ptr(hi), _ptr(r), _ptr(e))
    first = hi.view(np.float32)
    # the rest as the kernels form it: to FP32, then an exact power of two
    rest = r.astype(np.float32)
    for x, a, b, k in zip(v.tolist(), first.tolist(), rest.tolist(), e.tolist()):
        want = Fraction(x) * Fraction(2) ** -q
        got = Fraction(a) + Fraction(b) * Fraction(2) ** k
        # the first part is nearest: what is left is half a unit of 24 bits at most
        assert abs(want - Fraction(a)) <= abs(want) * Fraction(1, 2 ** 24), x
        # 24 more bits of the rest, of which those below the 56th bit of the value may be cut off
        assert abs(got - want) <= abs(want) * Fraction(1, 2 ** 47), x


def test_doubles_become_the_nearest_integer(fx):
    """Of a line whose largest value is 1.75: values of every size below it, at and about the halves of a unit, and
    far below one."""
    rng = np.random.default_rng(5)
    ex = fx.exponent(ctypes.c_double(1.75))
    q = fx.input_bits() + 1022 - ex
    x = [float(m) * 2.0 ** -k for m, k in zip(rng.uniform(1, 2, 4000), rng.integers(0, 120, 4000))]
    x += [m * 2.0 ** -q for m in (0.25, 0.499, 0.5, 0.501, 0.999, 1.0, 1.499, 1.5, 2.5, 3.5)]
    x += [np.nextafter(0.5, 0.0) * 2.0 ** -q, np.nextafter(0.25, 1.0) * 2.0 ** -q, 1.75, 1e-17, 1e-20, 1e-100, 1e-300,
          2.0 ** -1022, 5e-324, 0.0]
    x = np.array(x + [-v for v in x])
    v = np.empty(x.size, np.int64)
    fx.to_units(x.size, _ptr(x), ex, _ptr(v))
    for a, b in zip(x.tolist(), v.tolist()):
        u = abs(Fraction(a)) * Fraction(2) ** q
        assert abs(b) == int(u + Fraction(1, 2)) and b * a >= 0, (a, b)  # (ties away from zero)


def _kinds(n, rng):
    j = np.arange(1, n)
    x, g = j / n, rng.standard_normal(n - 1)
    spike = np.zeros(n - 1)
    spike[(n - 1) // 3] = 1.0
    yield "normal", g
    yield "smooth", np.exp(-(x - 0.3) ** 2 / 0.01)
    yield "alternating", (-1.0) ** j * (1 + 0.1 * g)
    yield "low mode", np.sin(3 * np.pi * x)
    yield "high mode", np.sin(np.pi * (n - 2) * x)
    yield "spike", spike
    yield "ones", np.ones(n - 1)
    yield "spread", g * np.exp(rng.uniform(-60, 0, n - 1))
    yield "spread far", g * np.exp(12 * rng.standard_normal(n - 1))
    for w in (0.3, 0.5, 1, 2, 5, 20):  # tails of one sign, as the solution beside a body or vortex has them
        yield "tail %g" % w, np.exp(-np.abs(j - n / 4) / w)
        yield "end %g" % w, np.exp(-j / w)
    yield "power", 1.0 / j ** 3
    yield "spike on 1e-17", spike + 1e-17
    yield "spike on 1e-9", spike + 1e-9


@pytest.mark.parametrize("n", [8, 24, 64, 100, 200, 360, 500, 1024, 1500, 2048])
def test_line_error_is_below_an_fp64_transforms(fx, n):
    """Errors (2-norm) of the kernels' steps on integers and of the same steps in FP64 against sums in extended
    precision, root mean squares over lines of one kind."""
    worse = {}
    for seed in range(6):
        rng = np.random.default_rng(seed)
        for kind, y in _kinds(n, rng):
            y = np.ascontiguousarray(y * rng.uniform(1, 2))
            e = (ctypes.c_double * 2)()
            fx.line_errors(n, _ptr(y), ctypes.byref(e, 0), ctypes.byref(e, 8))
            worse.setdefault(kind, []).append((e[0] ** 2, e[1] ** 2))
    for kind, e in worse.items():
        a, b = np.sqrt(np.mean(e, axis=0))
        # (a line whose sums are exact in FP64 leaves nothing to be below: half a unit of the results is)
        assert a <= max(b, 2.0 ** -53), (kind, a, b)


_EXTREME = """
import ctypes, sys
import numpy as np
lib = ctypes.CDLL(sys.argv[1])
ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)
for n in (8, 12, 20, 48, 200, 360, 972, 1000, 1024, 1500, 2048):
    j, rng = np.arange(1, n), np.random.default_rng(n)
    k, e = np.pi * j / n, (ctypes.c_double * 2)()
    top = np.nextafter(2.0, 0.0)  # rounds to the largest integer of a line
    # the largest outputs, and combs whose outputs a and b are the largest of both signs
    lines = [np.ones(n - 1), np.sign(np.sin(k)), np.sign(np.sin((n - 1) * k)), (-1.0) ** j, rng.choice([-1.0, 1.0], n - 1)]
    lines += [(j == i) * 1.0 for i in (1, n // 4, n // 2, n - 1)] + [(j % 8 == 0) * 1.0, (j % 2 == 1) * 1.0]
    for a, b in ((1, 3), (3, 9), (15, 47), (15, 45), (63, 189)):
        f = np.sin(a * k) - np.sin(b * k)
        lines += [np.where(np.abs(f) > t, np.sign(f), 0.0) for t in (0.0, 1.2, 1.8)]
    for y in (y for y in lines if y.any()):
        for s in (top, -top, 1.5):
            lib.line_errors(n, ptr(np.ascontiguousarray(y * s)), ctypes.byref(e, 0), ctypes.byref(e, 8))
            assert e[0] < 1e-14, (n, e[0])
"""


def test_no_signed_overflow_at_extreme_lines(tmp_path):
    """Lines of the largest values, and of the largest outputs of both signs (whose partial sums wrap): no undefined
    operation, and no lost high bit (errors of an FP64 transform's size)."""
    out = tmp_path / "fx_trap.so"
    _build(out, "-fsanitize=signed-integer-overflow,shift", "-fsanitize-undefined-trap-on-error")
    r = subprocess.run([sys.executable, "-c", _EXTREME, str(out)], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stderr[-400:])
