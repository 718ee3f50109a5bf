"""Matrices that need row interchanges, through the LU operators, with a leading
dimension above n as well: seen before the factorisation (an entry below the
diagonal larger than it, in the first, a middle and the last columns), found on
the way (no such entry, but a pivot that cancels), and none at all.  P A = L U
with dgetrf's permutation to n u |L| |U| (Higham, theorem 9.3; u 2^-21 in float,
where three TF32 passes keep 21 bits), |L| <= 1, the rows between n and the
leading dimension untouched, and a solve to 12 n u |A| |x|.

What the attempt costs a matrix that needs interchanges: it is seen first, so
next to nothing.  Factoring it in vain took 1.09 to 1.5 times the pivoting
launches alone."""
import ctypes as C
import os
import time

import numpy as np
import pytest
import torch
from scipy.linalg import lapack

from tinyvlm_gb300 import _lib

pytestmark = pytest.mark.gpu

KINDS = ("none", "first", "middle", "last", "cancels", "cancels_late", "random", "drops", "drops_late")


def _matrix(n, kind, npd):
    rng = np.random.default_rng(n + 10 * KINDS.index(kind))
    if kind == "random":
        return rng.standard_normal((n, n)).astype(npd)
    A = (0.01 * rng.uniform(-1, 1, (n, n)) + np.diag(rng.uniform(8, 10, n))).astype(npd)
    if kind in ("first", "middle", "last"):
        j = {"first": 0, "middle": n // 2, "last": n - 2}[kind]
        A[n - 1, j] = 100.0
    if kind.startswith("cancels"):  # pivot k + 1 becomes 1e-3 against 0.9 below it
        k = 1 if kind == "cancels" else n - 4
        A[k:k + 3, k:k + 3] = [[1, 1, 0], [1, 1.001, 0], [0, 0.9, 5]]
        A[k + 3:, k:k + 3] *= 0.01
        A[k:k + 3, :k] *= 0.001
    if kind.startswith("drops"):  # the same without the tie in column k
        k = 1 if kind == "drops" else n - 4
        A[k:k + 3, k:k + 3] = [[1, 1, 0], [0.5, 0.501, 0], [0, 0.4, 5]]
        A[k + 3:, k:k + 3] *= 0.01
        A[k:k + 3, :k] *= 0.001
    return A


class _Lu:
    def __init__(self, npd):
        self.L, self.sfx = _lib.lib(), "f32" if npd == np.float32 else "f64"
        self.h = C.c_void_p()
        assert self.L.gbvlm_lu_create(C.byref(self.h)) == 0

    def factor(self, M, n, ld):
        rc = getattr(self.L, "gbvlm_lu_factor_" + self.sfx)(self.h, C.c_void_p(M.data_ptr()), C.c_int64(n),
                                                           C.c_int64(ld), None)
        assert rc == 0, self.L.gbvlm_last_error()

    def solve(self, M, n, ld, X):
        rc = getattr(self.L, "gbvlm_lu_solve_" + self.sfx)(self.h, C.c_void_p(M.data_ptr()), C.c_int64(n),
                                                          C.c_int64(ld), C.c_void_p(X.data_ptr()), C.c_int64(n),
                                                          C.c_int64(1), None)
        assert rc == 0, self.L.gbvlm_last_error()

    def close(self):
        self.L.gbvlm_lu_destroy(self.h)


@pytest.mark.parametrize("npd", [np.float32, np.float64])
@pytest.mark.parametrize("n,pad", [(33, 0), (40, 7), (128, 4), (129, 3), (200, 0), (300, 21), (517, 11)])
@pytest.mark.parametrize("kind", KINDS)
def test_factor_and_solve(cuda, npd, n, pad, kind):
    ld = n + pad
    A = _matrix(n, kind, npd)
    A64 = A.astype(np.float64)
    _, piv, info = lapack.dgetrf(A64)
    assert info == 0
    moved = (piv != np.arange(n)).any()
    assert moved == (kind != "none"), kind
    low = (np.abs(np.tril(A64, -1)) > np.abs(np.diag(A64))).any()
    assert low == (kind in ("first", "middle", "last", "random"))
    M = np.full((n, ld), 7.0, npd)  # column-major: row c is column c
    M[:, :n] = A.T
    lu = _Lu(npd)
    b = np.random.default_rng(1).standard_normal(n).astype(npd)
    for _ in range(2):  # the handle's second factorisation, too
        T = torch.from_numpy(M.copy()).cuda()
        X = torch.from_numpy(b.copy()).cuda()
        lu.factor(T, n, ld)
        lu.solve(T, n, ld, X)
        torch.cuda.synchronize()
    out, x = T.cpu().numpy(), X.cpu().numpy().astype(np.float64)
    lu.close()
    assert (out[:, n:] == 7.0).all()
    F = out[:, :n].T.astype(np.float64)
    L, U = np.tril(F, -1) + np.eye(n), np.triu(F)
    p = np.arange(n)
    for k, q in enumerate(piv):
        p[[k, q]] = p[[q, k]]
    u = 2.0 ** -21 if npd == np.float32 else 2.0 ** -53
    # (float decides near ties otherwise: a random matrix's, the one between the rows k and k + 1 of "cancels")
    if npd == np.float64 or not (kind == "random" or kind.startswith("cancels")):
        assert (np.abs(L) <= 1.0 + 4 * u).all()
        assert (np.abs(A64[p] - L @ U) <= n * u * (np.abs(L) @ np.abs(U))).all()
    assert (np.abs(b - A64 @ x) <= 12 * n * u * (np.abs(A64) @ np.abs(x)) * (1 if kind != "random" else n)).all()


@pytest.mark.parametrize("npd,n", [(np.float32, 500), (np.float64, 200), (np.float32, 4096)])
def test_what_the_look_costs(cuda, npd, n):
    gen = torch.Generator("cuda").manual_seed(1)
    A = torch.rand((n, n), dtype=torch.float32 if npd == np.float32 else torch.float64, device="cuda", generator=gen)
    W = torch.empty_like(A)
    best = {}
    old = os.environ.get("GBVLM_LU_FAST")
    try:
        for fast in ("1", "0"):
            os.environ["GBVLM_LU_FAST"] = fast
            lu = _Lu(npd)
            for _ in range(12):
                W.copy_(A)
                torch.cuda.synchronize()
                t = time.perf_counter()
                lu.factor(W, n, n)
                best[fast] = min(best.get(fast, 1e9), time.perf_counter() - t)
            lu.close()
    finally:
        os.environ.pop("GBVLM_LU_FAST") if old is None else os.environ.update(GBVLM_LU_FAST=old)
    assert best["1"] <= 1.06 * best["0"], best
