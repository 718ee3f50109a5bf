"""The refinement residual's arithmetic, to the bit: every product exact as a pair
of floats, the running sum compensated, one column after the other.  numpy's
float32 does the same operations (a fused multiply-add by way of long double).  At the
edges of chunks (8 columns), right-hand sides (8) and rows (128), with columns
and solutions of widely different magnitude within a chunk, and its error
against long double (or quadruple) arithmetic: the median over rows at most twice
the 3.4e-15 of the sum of |a x| that this arithmetic has for 512 random terms."""
import ctypes as C

import numpy as np
import pytest
import torch

from tinyvlm_gb300 import _lib

pytestmark = pytest.mark.gpu
f32 = np.float32


def _fma(a, b, c):
    """a * b + c rounded once: the product of floats is exact in double, the sum in quadruple precision."""
    L = np.longdouble
    return (a.astype(np.float64) * b.astype(np.float64)).astype(L).__add__(c.astype(L)).astype(f32)


def _emulate(A, Alo, X, B, x_lo):
    n, m = X.shape
    sh, sl = np.zeros((n, m), f32), np.zeros((n, m), f32)
    for j in range(n):
        a = np.repeat(A[:, j:j + 1], m, 1)
        xh = X[j].astype(f32)
        xl = (X[j] - xh.astype(np.float64)).astype(f32)
        xh, xl = np.repeat(xh[None], n, 0), np.repeat(xl[None], n, 0)
        p = a * xh
        pe = (a.astype(np.float64) * xh.astype(np.float64) - p.astype(np.float64)).astype(f32)
        s = sh + p
        bb = s - sh
        e = (sh - (s - bb)) + (p - bb)
        sh = s
        sl = sl + (e + pe)
        if x_lo:
            sl = _fma(a, xl, sl)
        if Alo is not None:
            sl = _fma(np.repeat(Alo[:, j:j + 1], m, 1), xh, sl)
    return B - (sh.astype(np.float64) + sl.astype(np.float64))


def _gpu(A, Alo, X, B, x_lo):
    n, m = X.shape
    d = lambda z: torch.from_numpy(np.ascontiguousarray(z.T)).cuda()
    a, x, b = d(A), d(X), d(B)
    al = None if Alo is None else d(Alo)
    r = torch.empty((m, n), dtype=torch.float64, device="cuda")
    ptr = lambda t: None if t is None else C.c_void_p(t.data_ptr())
    rc = _lib.lib().gbvlm_test_batch_residual(n, m, ptr(a), ptr(al), ptr(x), ptr(b), ptr(r), int(x_lo), None)
    assert rc == 0
    return r.cpu().numpy().T


@pytest.mark.parametrize("n,m", [(1, 1), (7, 8), (8, 9), (9, 1), (127, 3), (129, 7), (257, 17)])
@pytest.mark.parametrize("lo", [False, True])
@pytest.mark.parametrize("x_lo", [False, True])
@pytest.mark.parametrize("spread", [0, 6])
def test_bits(cuda, n, m, lo, x_lo, spread):
    rng = np.random.default_rng(n + 1000 * m)
    A = (rng.standard_normal((n, n)) * 10.0 ** rng.uniform(-spread, spread, (1, n))).astype(f32)
    X = rng.standard_normal((n, m)) * 10.0 ** rng.uniform(-spread, spread, (n, m))
    if not x_lo:
        X = X.astype(f32).astype(np.float64)
    Alo = (A.astype(np.float64) * rng.uniform(-1, 1, (n, n)) * 2.0 ** -25).astype(f32) if lo else None
    B = rng.standard_normal((n, m))
    assert (_gpu(A, Alo, X, B, x_lo) == _emulate(A, Alo, X, B, x_lo)).all()


def test_error(cuda):
    n = 512
    rng = np.random.default_rng(3)
    A = rng.standard_normal((n, n)).astype(f32)
    X = rng.standard_normal((n, 8))
    L = np.longdouble
    exact = -sum(A[:, j:j + 1].astype(L) * X[j][None].astype(L) for j in range(n))
    scale = np.abs(A).astype(np.float64) @ np.abs(X)
    err = np.abs((_gpu(A, None, X, np.zeros((n, 8)), True).astype(L) - exact).astype(np.float64)) / scale
    assert np.median(err) <= 6.8e-15, np.median(err)
