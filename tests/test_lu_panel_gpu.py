"""The register panel's attempt without interchanges against LAPACK's pivots.

Diagonally dominant matrices keep every row in place; a planted entry larger
than the diagonal must send its panel (and the one after it) through the
pivoting loop, wherever the entry's row lives: the diagonal block, the same
CTA, another CTA of the cluster, the last ragged panel.  An entry of exactly
the diagonal's magnitude must not (LAPACK takes the first of equals).

The pivots are dgetrf's on the same matrix (the planted entries make them
unambiguous), so with L and U read back, P A = L U must hold to the backward
error of elimination: |PA - LU| <= n u |L||U| (Higham, Accuracy and Stability,
theorem 9.3), u = 2^-53 in double and 2^-21 in float, where a product
of the tensor cores' three TF32 passes keeps 21 bits.  Another pivot
order fails by many orders of magnitude."""
import numpy as np
import pytest
import torch
from scipy.linalg import lapack

from tinyvlm_gb300 import backend as B

pytestmark = pytest.mark.gpu


def _dominant(n, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((n, n)) + 4.0 * np.sqrt(n) * np.eye(n)


def _check(A, npd):
    n = A.shape[0]
    A = A.astype(npd)
    At = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    be = B.Backend(torch.float32 if npd == np.float32 else torch.float64)
    lu = be.create_lu_solver()
    lu.init(At)
    lu.factorize(At)
    torch.cuda.synchronize()
    F = At.cpu().numpy().T.astype(np.float64)
    _, piv, info = lapack.dgetrf(A.astype(np.float64))
    assert info == 0
    PA = A.astype(np.float64)
    for r, p in enumerate(piv):
        PA[[r, p]] = PA[[p, r]]
    L, U = np.tril(F, -1) + np.eye(n), np.triu(F)
    u = 2.0 ** -21 if npd == np.float32 else 2.0 ** -53
    bound = n * u * (np.abs(L) @ np.abs(U))
    assert (np.abs(PA - L @ U) <= bound).all()
    return piv


@pytest.mark.parametrize("npd", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 65, 300, 1057])
def test_rows_stay(cuda, npd, n):
    piv = _check(_dominant(n, n), npd)
    assert (piv == np.arange(n)).all()


@pytest.mark.parametrize("npd", [np.float32, np.float64])
@pytest.mark.parametrize("n,row,col", [
    (40, 5, 3),        # inside the diagonal block
    (40, 39, 33),      # the last, narrow panel
    (300, 299, 0),     # the first column, the last row
    (300, 150, 64),    # a later panel
    (1057, 1050, 7),   # a row of the cluster's last CTA
    (1300, 1299, 200),
])
def test_planted_pivot_moves_rows(cuda, npd, n, row, col):
    A = _dominant(n, n + row)
    A[row, col] = 3.0 * A[col, col]
    piv = _check(A, npd)
    assert piv[col] == row


@pytest.mark.parametrize("npd", [np.float32, np.float64])
@pytest.mark.parametrize("n,row", [(33, 20), (300, 299)])
def test_equal_magnitude_keeps_the_first(cuda, npd, n, row):
    A = _dominant(n, 7).astype(npd).astype(np.float64)
    A[row, 0] = -A[0, 0]
    piv = _check(A, npd)
    assert piv[0] == 0
