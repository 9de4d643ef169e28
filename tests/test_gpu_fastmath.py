"""The inverse root, root, sine, cosine, arc tangent and quotient that the
kernels use in place of CUDA's (device/rrea_fastmath.cuh,
rrea_exact_quot.cuh), each against extended precision within the bound its
comment states, over the range it covers and at both sides of every hand-over
to CUDA's function; at zeros of both signs, subnormals, infinities and NaN the
result is CUDA's (the sign of a zero sine or quotient aside, which nothing
reads).  tests/cpp/fastmath.cu evaluates them."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

LOG_EXP, TURNS = 1028, 256
L = np.longdouble
PI = L(np.pi) + L(1.2246467991473532e-16)
INF, NAN = np.inf, np.nan
NEG_NAN = np.frombuffer(np.uint64(0xFFF8000000000000).tobytes())[0]


def _neighbours(values):
    v = np.asarray(values, dtype=np.float64)
    return np.concatenate([np.nextafter(v, -INF), v, np.nextafter(v, INF)])


def _logspace(rng, lo, hi, n):
    """n doubles of uniform exponent in [2^lo, 2^hi)."""
    return np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n))


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fastmath") / "fastmath.so")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_103a,code=sm_103a", "-shared", "-Xcompiler",
                    "-fPIC", "-o", so, os.path.join(ROOT, "tests", "cpp", "fastmath.cu")], check=True)
    lib = ctypes.CDLL(so)
    D = ctypes.POINTER(ctypes.c_double)
    lib.fastmath_eval.argtypes = [ctypes.c_int, D, ctypes.c_int, D, D, ctypes.c_int, D, D]
    # sines and cosines of j/256 turns, exact at the quarter turns, as the loader writes them
    j = np.arange(TURNS)
    q, i = j // 64, j % 64
    first = np.minimum(i, 64 - i)
    a, b = np.sin(first * PI / 128), np.cos(first * PI / 128)
    s, c = np.where(i <= 32, a, b), np.where(i <= 32, b, a)
    arena = np.zeros(LOG_EXP + 2 * TURNS)
    arena[LOG_EXP::2] = np.choose(q, [s, c, -s, -c]).astype(np.float64)
    arena[LOG_EXP + 1::2] = np.choose(q, [c, -s, -c, s]).astype(np.float64)

    def run(which, x, y=None):
        x = np.ascontiguousarray(x, dtype=np.float64)
        y = np.zeros_like(x) if y is None else np.ascontiguousarray(y, dtype=np.float64)
        out, out2 = np.zeros_like(x), np.zeros_like(x)
        p = [v.ctypes.data_as(D) for v in (arena, x, y, out, out2)]
        assert lib.fastmath_eval(which, p[0], arena.size, p[1], p[2], x.size, p[3], p[4]) == 0
        return out, out2

    return run


SPECIAL = np.array([0.0, -0.0, 5e-324, -5e-324, 2.2250738585072014e-308, 1e-310, 1e-300, 1e300, 1.7e308, INF, -INF, NAN,
                    NEG_NAN, -1.0, -1e-300])
ROOT_EDGES = _neighbours([2.0 ** -100, 2.0 ** 100, 2.0 ** 101, 2.0 ** -101])


def test_roots(evaluate):
    rng = np.random.default_rng(1)
    x = np.concatenate([_logspace(rng, -100, 100, 200_000), _logspace(rng, -2, 2, 100_000),
                        _neighbours(2.0 ** np.arange(-99, 100))])
    inv, _ = evaluate(0, x)
    ref = 1.0 / np.sqrt(L(x))
    assert (np.abs(inv - ref) <= 0.51 * np.spacing(ref.astype(np.float64))).all()
    root, _ = evaluate(1, x)
    ref = np.sqrt(L(x))
    assert (np.abs(root - ref) <= 0.51 * np.spacing(ref.astype(np.float64))).all()
    y = np.concatenate([SPECIAL, _logspace(rng, -1022, -101, 1000), _logspace(rng, 101, 1023, 1000)])
    inv, cuda = evaluate(0, y)
    np.testing.assert_array_equal(inv, cuda)
    root, cuda = evaluate(1, y)
    np.testing.assert_array_equal(root, cuda)
    edge, _ = evaluate(1, ROOT_EDGES)
    np.testing.assert_allclose(edge, np.sqrt(ROOT_EDGES), rtol=2.0 ** -51, atol=0)
    edge, _ = evaluate(0, ROOT_EDGES)
    np.testing.assert_allclose(edge, 1.0 / np.sqrt(ROOT_EDGES), rtol=2.0 ** -51, atol=0)


def test_sine_and_cosine(evaluate):
    rng = np.random.default_rng(2)
    step = 2.0 * np.pi / TURNS
    k = np.arange(-1024, 1025)
    x = np.concatenate([rng.uniform(-np.pi, np.pi, 300_000), rng.uniform(-1024.0, 1024.0, 100_000),
                        _neighbours(k * step), _neighbours((k + 0.5) * step), _logspace(rng, -1060, 0, 2000),
                        -_logspace(rng, -1060, 0, 2000), [0.0, -0.0, np.nextafter(1024.0, 0.0)]])
    s, c = evaluate(2, x)
    assert np.abs(s - np.sin(L(x))).max() <= 1.1 * 2.0 ** -53
    assert np.abs(c - np.cos(L(x))).max() <= 1.1 * 2.0 ** -53
    far = np.concatenate([[1024.0, -1024.0, 1e6, 1e22, -1e300, INF, -INF, NAN, NEG_NAN], _logspace(rng, 10, 1023, 1000)])
    np.testing.assert_array_equal(evaluate(2, far), evaluate(3, far))
    u = np.concatenate([rng.uniform(0.0, 1.0, 200_000), np.clip(_neighbours(np.arange(512) / 512.0), 0.0, 1.0)])
    s, c = evaluate(4, u)
    assert np.abs(s - np.sin(2.0 * PI * L(u))).max() <= 1.1 * 2.0 ** -53
    assert np.abs(c - np.cos(2.0 * PI * L(u))).max() <= 1.1 * 2.0 ** -53


def _check_angle(evaluate, x, y):
    """CUDA's angle where the larger coordinate is outside [2^-100, 2^100], else
    within two ulps of the exact one; the sign (of a zero too) always."""
    a, cuda = evaluate(5, x, y)
    m = np.maximum(np.abs(x), np.abs(y))   # NaN if either is
    near = (m >= 2.0 ** -100) & (m <= 2.0 ** 100)
    np.testing.assert_array_equal(a[~near], cuda[~near])
    ref = np.arctan2(L(y[near]), L(x[near]))
    ulp = np.spacing(np.maximum(np.abs(ref), 2.3e-308).astype(np.float64))
    assert (np.abs(a[near] - ref) <= 2.0 * ulp).all()
    number = ~np.isnan(cuda)
    np.testing.assert_array_equal(np.signbit(a[number]), np.signbit(cuda[number]))


def test_arc_tangent(evaluate):
    rng = np.random.default_rng(3)
    step = 2.0 * np.pi / TURNS
    k = np.arange(-TURNS // 2, TURNS // 2 + 1)
    th = np.concatenate([rng.uniform(-np.pi, np.pi, 200_000), rng.uniform(-0.05, 0.05, 100_000),
                         _neighbours(k * step), _neighbours((k + 0.5) * step)])
    r = _logspace(rng, -98, 98, th.size)
    x, y = r * np.cos(th), r * np.sin(th)
    # beside the axes, down to coordinates past the seed's range
    big, small = _logspace(rng, -90, 99, 4000), _logspace(rng, -1000, -91, 4000)
    sx, sy = rng.choice([-1.0, 1.0], (2, 4000))
    x = np.concatenate([x, sx * big, sx * small, sx * big, sx * 0.0, sx * big])
    y = np.concatenate([y, sy * small, sy * big, sy * 0.0, sy * big, sy * big])
    _check_angle(evaluate, x, y)
    v = np.concatenate([SPECIAL, -SPECIAL, [2.0 ** -101, 2.0 ** 101, 2.0 ** 127, 2.0 ** 128, 2.0 ** 130, 2.0 ** 200,
                                            -2.0 ** 130]])
    _check_angle(evaluate, *(g.ravel() for g in np.meshgrid(v, v)))
    # one coordinate far beyond the other's, in and out of range
    one = rng.choice([-1.0, 1.0], 2000) * rng.uniform(0.5, 2.0, 2000)
    huge = rng.choice([-1.0, 1.0], 2000) * _logspace(rng, 101, 1023, 2000)
    for x, y in ((huge, one), (one, huge), (huge, 2.0 ** 60 * one), (huge, huge[::-1].copy())):
        _check_angle(evaluate, x, y)


def test_quotient(evaluate):
    rng = np.random.default_rng(4)
    n = 200_000
    a = rng.choice([-1.0, 1.0], n) * _logspace(rng, -500, 500, n)
    b = rng.choice([-1.0, 1.0], n) * _logspace(rng, -400, 400, n)
    b[:1000] = np.nextafter(2.0 ** rng.integers(-40, 40, 1000), 0.0)   # mantissas of all ones
    a[-4000:], b[-4000:] = rng.integers(-50, 50, 4000), rng.integers(1, 50, 4000)
    q, ref = evaluate(6, a, b)
    np.testing.assert_array_equal(q, ref)
    a = np.array([0.0, -0.0, INF, -INF, NAN, 1.7e308, -1.7e308])
    q, ref = evaluate(6, a, np.full(a.size, 0.3))
    np.testing.assert_array_equal(q, ref)
