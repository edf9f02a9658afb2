"""The f32 arithmetic of the pair loops: the quotient and the root against CUDA's own
division and square root and against 64 bits, the gradient factor of pass A on close
pairs.

Bounds: the approximate reciprocal and reciprocal root are within 2^-23 and 2^-22.4;
one Newton (Heron) step leaves 2^-45 (2^-43) before the last rounding, that is
2^-21 (2^-19) ulp: half an ulp and that much against 64 bits, and another float than
the rounded result only that near a tie, an ulp away, in one of 2^20 (2^18) values.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _math(op, a, b):
    from sphgpu import _capi
    lib = _capi.load()
    a = np.ascontiguousarray(np.broadcast_to(a, np.broadcast(a, b).shape), np.float32)
    b = np.ascontiguousarray(np.broadcast_to(b, a.shape), np.float32)
    out = np.empty_like(a)
    f = lib.sph_test_pair_math
    f.argtypes = [C.c_int, C.c_size_t, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int]
    f.restype = C.c_int
    _capi.check(f(op, a.size, a.ctypes.data, b.ctypes.data, out.ctypes.data, 0))
    return out


def _values(rng, lo, hi, n):
    return np.exp(rng.uniform(np.log(lo), np.log(hi), n)).astype(np.float32)


def _check(got, cuda, exact, near):
    ulp = np.spacing(np.abs(exact.astype(np.float32))).astype(np.float64)
    assert np.max(np.abs(got - exact) / ulp) <= 0.5 + near
    other = got != cuda
    assert np.max(np.abs(got[other].astype(np.float64) - cuda[other]) / ulp[other], initial=0) <= 1.0 + near
    assert other.mean() <= 4 * near


@pytest.mark.parametrize("a,b", [((1e-12, 1e12), (1e-12, 1e6)), ((1.0, 2.0), (1.0, 2.0)), ((1e-6, 1e-5), (1e-9, 1e-3))])
def test_quotient(a, b):
    rng = np.random.default_rng(5)
    n = 1 << 22
    x, y = _values(rng, *a, n) * rng.choice([-1, 1], n).astype(np.float32), _values(rng, *b, n)
    _check(_math(0, x, y), _math(1, x, y), x.astype(np.float64) / y.astype(np.float64), 2.0 ** -20)


def test_quotient_of_zero_is_zero():
    assert not np.any(_math(0, np.zeros(64), _values(np.random.default_rng(1), 1e-12, 1e6, 64)))


@pytest.mark.parametrize("lo,hi", [(1e-30, 1e6), (1.0, 4.0), (1e-6, 1e-2)])
def test_root(lo, hi):
    x = _values(np.random.default_rng(6), lo, hi, 1 << 22)
    _check(_math(2, x, np.float32(1.0)), _math(3, x, np.float32(1.0)), np.sqrt(x.astype(np.float64)), 2.0 ** -18)


# Pass A's factor (2 - 3q) / h for q < 1/2, (1-q)^2 / |r| beyond, against 64 bits: the rms
# relative error of (2 - 3q) / h, from an f32 q with an error of 1.5 ulp, is below
# 2^-24 (1 + 3 q 1.5 / (2 - 3q)); half as much again for the constants.
@pytest.mark.parametrize("lo,hi", [(1e-3, 1e-2), (0.01, 0.1), (0.1, 0.2), (0.2, 0.3), (0.3, 0.4), (0.4, 0.5)])
@pytest.mark.parametrize("h", [0.04, 0.13, 2.7])
def test_gradient_factor_of_close_pairs(lo, hi, h):
    ih = np.float32(1.0 / h)
    x = (np.random.default_rng(7).uniform(lo, hi, 1 << 20) * h).astype(np.float32)
    q = x.astype(np.float64) * np.float64(ih)
    exact = (2.0 - 3.0 * q) * np.float64(ih)
    rms = np.sqrt(np.mean((_math(5, x, ih) / exact - 1.0) ** 2))
    assert rms < 1.5 * 2.0 ** -24 * (1.0 + 4.5 * hi / (2.0 - 3.0 * hi))
