"""One right-hand side through the single-column dataflow solve, at the edges
of its blocks (128 rows in float, 64 in double) and of the size from which it
is used, with row interchanges, twice on the same factors, and on a matrix
with a leading dimension.  Bar: the backward error of two triangular solves,
|b - A x| <= 3 n u (|A| |x|) with a factor 4 for the factorisation's growth
(Higham, theorem 9.4), u the unit roundoff (2^-21 in float: the trailing
updates' three TF32 passes)."""
import numpy as np
import pytest
import torch

from tinyvlm_gb300 import backend as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npd", [np.float32, np.float64])
@pytest.mark.parametrize("n", [64, 65, 96, 127, 128, 129, 192, 193, 257, 513, 900])
def test_one_column(cuda, npd, n):
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 0.5 * np.sqrt(n) * np.eye(n)).astype(npd)
    be = B.Backend(torch.float32 if npd == np.float32 else torch.float64)
    At = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    lu = be.create_lu_solver()
    lu.init(At)
    lu.factorize(At)
    A64 = A.astype(np.float64)
    u = 2.0 ** -21 if npd == np.float32 else 2.0 ** -53
    for k in range(2):
        b = rng.standard_normal(n).astype(npd)
        X = torch.from_numpy(b.copy()).cuda()
        lu.solve(At, X)
        torch.cuda.synchronize()
        x = X.cpu().numpy().astype(np.float64)
        r = np.abs(b.astype(np.float64) - A64 @ x)
        assert (r <= 12 * n * u * (np.abs(A64) @ np.abs(x))).all(), (k, r.max())
    lu.factorize(torch.from_numpy(np.ascontiguousarray(A.T)).cuda())  # reports a wait that ran out
