"""The wave pass's reciprocal square root and the pivots' reciprocals, each one
step from the hardware's approximation, by themselves: against 80-bit results
over the exponent range and next to powers of two, and against the bounds that
their steps give (u = 2^-53, or 2^-24 in single precision; an approximation of
20 bits, in single precision of 22).

Square root: y (1 + h / 2 + 3 h^2 / 8) with h = 1 - x y^2. The series' remainder is
5 / 16 h^3 <= 2^-58, h carries the rounding of x y (u, of which half enters) and
the last operation rounds by u: 1.6 u in all, in units of the last place half of
one by the rounding, at most half of one by h and 0.03 by the remainder; CUDA
documents one unit for its own rsqrt.

Reciprocal: conj(p) / |p|^2. The sum of squares carries 2 u, its reciprocal the
remainder h^3 <= 2^-57 (single precision: h^2 <= 2^-42, with h = 1 - d r) and one
rounding, the product one: 4.1 u of each component."""
import ctypes

import numpy as np
import pytest

import nemoh_b200 as nb

pytestmark = pytest.mark.gpu


def _run(x, p, q):
    f = nb.load_library().nemoh_b200_diag_reciprocals
    d, s = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_float)
    f.argtypes = [ctypes.c_int, ctypes.c_int, d, d, d, d, s, s]
    rs, rp, rq = np.zeros_like(x), np.zeros_like(p), np.zeros_like(q)
    st = f(0, len(x), *[a.ctypes.data_as(d) for a in (x, rs, p, rp)], *[a.ctypes.data_as(s) for a in (q, rq)])
    assert st == 0
    return rs, rp, rq


def _values(rng, n, lo, hi, dtype):
    """Magnitudes over 2^lo .. 2^hi, a third of them within 50 units of a power of two."""
    x = np.exp2(rng.uniform(lo, hi, n)).astype(dtype)
    near = np.exp2(np.floor(rng.uniform(lo, hi, n // 3))).astype(dtype)
    for _ in range(50):
        step = rng.random(len(near)) < 0.5
        near[step] = np.nextafter(near[step], np.where(rng.random(step.sum()) < 0.5, 0, np.inf).astype(dtype))
    x[:len(near)] = near
    return x


def _pivots(rng, n, lo, hi, dtype):
    a, b = _values(rng, n, lo, hi, dtype), _values(rng, n, lo, hi, dtype)
    b[::2] = (a[::2] * rng.uniform(0, 1, len(a[::2]))).astype(dtype)   # components of like size
    a[5::97], b[7::101] = 0, 0
    a[(a == 0) & (b == 0)] = 1
    sign = lambda: rng.choice([-1, 1], n).astype(dtype)  # noqa: E731
    v = np.stack([a * sign(), b * sign()], axis=1)
    swap = rng.random(n) < 0.5
    v[swap] = v[swap][:, ::-1]
    return np.ascontiguousarray(v)


def _componentwise(v, r, u, tiny):
    x = v.astype(np.longdouble)
    s = np.exp2(-np.frexp(np.abs(x).max(axis=1))[1].astype(np.longdouble))[:, None]
    y = x * s
    ref = y * np.array([1, -1]) / (y * y).sum(axis=1, keepdims=True) * s
    big = np.abs(ref) > tiny   # results in the normal range
    assert np.isfinite(r).all()
    err = np.abs(r - ref)[big] / np.abs(ref)[big]
    assert (np.abs(r - ref)[~big] <= 2 * tiny).all()
    assert err.max() <= 4.1 * u, float(err.max() / u)


def test_reciprocals():
    rng = np.random.default_rng(0)
    n = 300000
    x = _values(rng, n, -1000, 1000, np.float64)
    x[:n // 2] = _values(rng, n // 2, -27, 45, np.float64)   # squared distances: 1e-8 to 3e13 m^2
    p, q = _pivots(rng, n, -60, 60, np.float64), _pivots(rng, n, -60, 60, np.float32)
    wide = slice(n // 2, None)
    p[wide] = _pivots(rng, n - n // 2, -1000, 1000, np.float64)
    q[wide] = _pivots(rng, n - n // 2, -120, 120, np.float32)
    rs, rp, rq = _run(x, p, q)
    xl = x.astype(np.longdouble)
    err = np.abs(rs * np.sqrt(xl) - 1)
    assert err.max() <= 1.6 * 2.0 ** -53, float(err.max() * 2 ** 53)
    ulp = np.abs(rs - 1 / np.sqrt(xl)) / np.spacing(rs)
    assert ulp.max() <= 1.03, float(ulp.max())
    _componentwise(p, rp, 2.0 ** -53, 1e-307)
    _componentwise(q, rq, 2.0 ** -24, 1e-37)
    # an ordinary quotient, where its own squares neither overflow nor underflow
    mid = slice(0, n // 2)
    c = 1 / (p[mid, 0] + 1j * p[mid, 1])
    got = rp[mid, 0] + 1j * rp[mid, 1]
    assert (np.abs(got - c) <= 8 * 2.0 ** -53 * np.abs(c)).all()
