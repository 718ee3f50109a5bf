"""The refinement residual at the edges of its chunks (8 columns, 8 right-hand
sides, 128 rows), and a lone system whose geometry is shared by several blocks:
two sweeps against the FP64 system.  Bars: those of the batched solver's own
test, 3e-7 of the circulations' norm and 5e-7 of CL and CM."""
import numpy as np
import pytest

from oracle import oracle as O
from tinyvlm_gb300 import mesh as M
from tinyvlm_gb300.batch import BatchSolver, pack_alphas, pack_verts

pytestmark = pytest.mark.gpu
REF = (0.25, 0.0, 0.0)


@pytest.mark.parametrize("nc,ns,angles", [(1, 7, 1), (3, 3, 8), (1, 15, 9), (1, 127, 2), (4, 32, 8), (3, 43, 7),
                                          (5, 51, 17), (1, 257, 3), (9, 33, 1)])
def test_against_double(cuda, nc, ns, angles):
    case = M.batch_cases(1, seed=2, n_alpha=angles, nc_range=(nc, nc), ns_range=(ns, ns))[0]
    bs = BatchSolver([case], mode="shared", refine=2, fp64_residual=True)
    bs.set_inputs(pack_verts([case]), pack_alphas([case]), ref_pt=REF)
    bs.run(want_gamma=True)
    co, gam = bs.results(gamma=True)
    for k, r in enumerate(O.vlm_shared([case.verts.astype(np.float64)], case.alphas, ref_pt=REF)):
        g = np.concatenate([x.ravel() for x in r["gamma"]])
        assert np.linalg.norm(gam[k] - g) <= 3e-7 * np.linalg.norm(g)
        assert abs(co[k, 0] - r["cl"]) <= 5e-7 * max(abs(r["cl"]), 1e-3)
        assert np.abs(co[k, 2:5] - r["cm"]).max() <= 5e-7 * max(np.abs(r["cm"]).max(), 1e-6)
