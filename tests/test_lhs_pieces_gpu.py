"""AIC assembly at the edges of its pieces (two or four ring rows, 8 to 32
rings, 64 points): one ring, remainders of each, sizes on both sides of the
switch to larger pieces, several wake rows, core smoothing, and accumulation
into what the matrix held.  Bars of the operator's own test: float against the
double oracle on the same inputs 2e-4 of the entry plus 2e-5 of the largest,
double 1e-9 and 1e-12."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.helpers import close, synthetic_wake, wing
from tinyvlm_gb300 import backend as B

pytestmark = pytest.mark.gpu


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("npd,td", [(np.float32, torch.float32), (np.float64, torch.float64)])
@pytest.mark.parametrize("nc,ns,iteration,sigma", [(1, 1, 0, 0.0), (1, 1, 1, 0.0), (2, 7, 2, 0.0), (3, 9, 1, 0.05),
                                                   (5, 33, 1, 0.0), (4, 64, 3, 0.0), (9, 65, 1, 0.0), (30, 70, 1, 0.0)])
def test_lhs_pieces(cuda, npd, td, nc, ns, iteration, sigma):
    v = wing("trap", nc, ns, npd)
    w = synthetic_wake(v, iteration + 2, dtype=npd)
    col, nor, _ = O.mesh_metrics(0.0, [v], npd)
    n = nc * ns
    d = lambda x: x.astype(np.float64)
    base = np.random.default_rng(n).standard_normal((n, n)).astype(npd)
    ref = np.asfortranarray(d(base))
    O.lhs_assemble(ref, [d(col[0])], [d(nor[0])], [d(v)], [d(w)], iteration, sigma)
    be = B.Backend(td)
    be.sigma_vatistas = sigma
    lhs = T(base.T)
    be.lhs_assemble(lhs, [T(col[0])], [T(nor[0])], [T(v)], [T(w)], iteration)
    close(lhs.cpu().numpy().T, ref, *((2e-4, 2e-5) if npd == np.float32 else (1e-9, 1e-12)), "lhs")
