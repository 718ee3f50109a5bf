"""The square root, reciprocal and quotients of the double segment law and the
reciprocals of the LU's pivots against long double (quadruple) arithmetic, over
random mantissas, both ends of a binade, and the exponents that they meet:
squared lengths 1e-20 to 1e24, denominators 1e-40 to 1e60, pivots and their
reciprocals normal.  Bars, relative to the exact value: 2 x 2^-52 and 4 x 2^-52 as
their comments state (a start of 20 bits with one plain Newton step only would be
off by 2^-40), an ulp for the pivots."""
import ctypes as C

import numpy as np
import pytest
import torch

from tinyvlm_gb300 import _lib

pytestmark = pytest.mark.gpu
N = 1 << 16
L = np.longdouble


def _values(rng, lo, hi, n=N):
    m = rng.uniform(1.0, 2.0, n)
    m[:64] = 1.0 + np.arange(64) * 2.0 ** -52
    m[64:128] = 2.0 - np.arange(1, 65) * 2.0 ** -52
    return m * 2.0 ** rng.integers(int(np.ceil(np.log2(lo))), int(np.log2(hi)), n)


def _walk(kind, a, b=None):
    d = lambda z: None if z is None else torch.from_numpy(z).cuda()
    ptr = lambda t: None if t is None else C.c_void_p(t.data_ptr())
    ta, tb = d(a), d(b)
    out = torch.empty_like(ta)
    n = len(a) // (2 if kind == 2 else 1)
    assert _lib.lib().gbvlm_test_walk_math(kind, n, ptr(ta), ptr(tb), ptr(out), None) == 0
    return out.cpu().numpy().astype(L)


def _off(got, exact):
    return float(np.abs((got - exact) / exact).max())


def test_length(cuda):
    a = _values(np.random.default_rng(1), 1e-20, 1e24)
    assert _off(_walk(0, a), np.sqrt(a.astype(L))) <= 2 * 2.0 ** -52
    assert float(_walk(0, np.zeros(4)).max()) < 1e-140


def test_reciprocal(cuda):
    a = _values(np.random.default_rng(2), 1e-80, 1e120)
    assert _off(_walk(1, a), 1 / a.astype(L)) <= 2 * 2.0 ** -52


def test_quotients(cuda):
    rng = np.random.default_rng(3)
    a, b = _values(rng, 1e-20, 1e20), _values(rng, 1e-40, 1e60)
    assert _off(_walk(2, a, b), a.astype(L) / b.astype(L)) <= 4 * 2.0 ** -52


def test_pivots(cuda):
    rng = np.random.default_rng(4)
    sign = np.where(rng.uniform(size=N) < 0.5, -1.0, 1.0)
    a64 = sign * _values(rng, 1e-307, 1e306)
    a32 = (sign * _values(rng, 1.3e-38, 8e36)).astype(np.float32)
    a32 = np.where(np.abs(a32) > 1e37, np.float32(1e37), a32)
    t32, t64 = torch.from_numpy(a32).cuda(), torch.from_numpy(a64).cuda()
    o32, o64 = torch.empty_like(t32), torch.empty_like(t64)
    ptr = lambda t: C.c_void_p(t.data_ptr())
    assert _lib.lib().gbvlm_test_pivot_rcp(N, ptr(t32), ptr(o32), ptr(t64), ptr(o64), None) == 0
    assert _off(o32.cpu().numpy().astype(L), 1 / a32.astype(L)) <= 2.0 ** -23
    assert _off(o64.cpu().numpy().astype(L), 1 / a64.astype(L)) <= 2.0 ** -52
