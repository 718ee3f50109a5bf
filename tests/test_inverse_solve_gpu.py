"""The solve of a long unsteady run's steps (the inverse, refined once) against the
triangular solve that it takes the place of, on AICs of wings whose panel
counts lie off the tiles of 32, off the 16-byte rows and beyond the sizes from
which the identity is solved for by the dataflow launch (256 in float), and on
matrices with row interchanges.  Bar: its error is no larger than the solve's, in
the 2-norm of the error against 64 bits (in double: of the residual, formed in
long double; the bits of a double solution leave its error no exact yardstick).
The product with the inverse alone has 1.04 to 1.25 times the solve's error."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import oracle as O
from tinyvlm_gb300 import _lib
from tinyvlm_gb300 import backend as B
from tinyvlm_gb300 import mesh as M

pytestmark = pytest.mark.gpu


def _wing(nc, ns):
    v = M.trapezoid(nc, ns, 7.0, 0.5, 15.0)
    M.quarter_chord(v)
    return np.asarray(O.vlm_run([v.astype(np.float64)], 0.0, dtype=np.float64, return_state=True)["lhs"])


def _both(A, b):
    """x by the triangular solve and by the inverse, in the type of A."""
    n = len(b)
    td = torch.float32 if A.dtype == np.float32 else torch.float64
    F = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    At, bt = F.clone(), torch.from_numpy(b).cuda()
    lu = B.Backend(td).create_lu_solver()
    lu.init(F)
    lu.factorize(F)
    x = bt.clone()
    lu.solve(F, x)
    y = torch.empty_like(bt)
    ptr = lambda t: C.c_void_p(t.data_ptr())
    sfx = "f32" if A.dtype == np.float32 else "f64"
    assert getattr(_lib.lib(), "gbvlm_test_inverse_solve_" + sfx)(ptr(At), n, ptr(bt), ptr(y), None) == 0
    torch.cuda.synchronize()
    return x.cpu().numpy(), y.cpu().numpy()


SIZES = [(1, 1), (1, 31), (3, 11), (5, 13), (1, 127), (4, 33), (1, 257), (3, 171), (9, 65), (20, 45)]


@pytest.mark.parametrize("nc,ns", SIZES)
@pytest.mark.parametrize("kind", ["wing", "interchanges"])
def test_float(cuda, nc, ns, kind):
    A = _wing(nc, ns).astype(np.float32)
    n = len(A)
    rng = np.random.default_rng(n)
    if kind == "interchanges":
        A = A[rng.permutation(n)]
    ex = ey = 0.0
    for _ in range(4):
        b = rng.standard_normal(n).astype(np.float32)
        t = np.linalg.solve(A.astype(np.float64), b.astype(np.float64))
        x, y = _both(A, b)
        ex += np.linalg.norm(x - t) / np.linalg.norm(t)
        ey += np.linalg.norm(y - t) / np.linalg.norm(t)
    assert ey <= ex or ey <= 4 * 4 * 2.0 ** -24  # (or within some units of the result's own rounding)


@pytest.mark.parametrize("nc,ns", SIZES)
def test_double(cuda, nc, ns):
    A = _wing(nc, ns)
    n = len(A)
    rng = np.random.default_rng(n)
    L = np.longdouble
    ex = ey = 0.0
    for _ in range(4):
        b = rng.standard_normal(n)
        for k, z in enumerate(_both(A, b)):
            z = z.astype(L)
            r = b.astype(L) - np.array([(A[i].astype(L) * z).sum() for i in range(n)])
            e = float(np.sqrt((r * r).sum())) / np.linalg.norm(b)
            ex, ey = (ex + e, ey) if k == 0 else (ex, ey + e)
    assert ey <= ex or ey <= 4 * 4 * 2.0 ** -53
