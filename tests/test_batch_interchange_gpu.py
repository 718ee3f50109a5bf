"""A batch factors without row interchanges first and repeats the systems that
need them.  A mesh with shuffled vertices has an AIC that is not dominated by
its diagonal (checked with LAPACK's pivots): its results must be, bit for bit,
those of a plan that pivots from the start (GBVLM_LU_FAST=0), and its mates'
those they have alone.  The same when the inputs of the next run are set
before the results of this one are read."""
import os

import numpy as np
import pytest
from scipy.linalg import lapack

from oracle import oracle as O
from tinyvlm_gb300 import mesh as M
from tinyvlm_gb300.batch import BatchSolver, pack_alphas, pack_verts

pytestmark = pytest.mark.gpu


def _cases(nc, ns):
    cases = M.batch_cases(3, seed=5, n_alpha=2, nc_range=(nc, nc), ns_range=(ns, ns))
    rng = np.random.default_rng(1)
    v = cases[1].verts
    v[:3, 1:-1, 1:-1] += rng.normal(0.0, 0.4, v[:3, 1:-1, 1:-1].shape).astype(np.float32)
    s = O.vlm_run([v.astype(np.float64)], 0.0, dtype=np.float64, return_state=True)
    _, piv, _ = lapack.dgetrf(s["lhs"])
    assert (piv != np.arange(len(piv))).any()
    return cases


def _solve(cases, mode, fast=True, graph=True):
    old = os.environ.get("GBVLM_LU_FAST")
    os.environ["GBVLM_LU_FAST"] = "1" if fast else "0"
    try:
        bs = BatchSolver(cases, mode=mode)
        bs.set_inputs(pack_verts(cases), pack_alphas(cases))
        bs.run(want_gamma=True, graph=graph)
        return bs, bs.results(gamma=True)
    finally:
        if old is None:
            del os.environ["GBVLM_LU_FAST"]
        else:
            os.environ["GBVLM_LU_FAST"] = old


@pytest.mark.parametrize("nc,ns", [(4, 9), (12, 20), (20, 70)])
@pytest.mark.parametrize("mode,graph", [("shared", True), ("exact", True), ("shared", False)])
def test_interchanges_in_a_batch(cuda, nc, ns, mode, graph):
    cases = _cases(nc, ns)
    _, (co, g) = _solve(cases, mode, graph=graph)
    _, (cp, gp) = _solve(cases, mode, fast=False, graph=graph)
    assert np.isfinite(co).all()
    assert (co[2:4] == cp[2:4]).all() and all((a == b).all() for a, b in zip(g[2:4], gp[2:4]))
    for k in (0, 2):
        _, (ca, ga) = _solve(cases[k:k + 1], mode, graph=graph)
        assert (co[2 * k:2 * k + 2] == ca).all() and all((a == b).all() for a, b in zip(g[2 * k:2 * k + 2], ga))


def test_inputs_replaced_before_results(cuda):
    cases = _cases(12, 20)
    bs, (co, g) = _solve(cases, "shared")
    bs.set_inputs(pack_verts(cases), pack_alphas(cases))
    bs.run(want_gamma=True)
    other = [M.Case(c.verts, 2.0 * c.alphas, {}) for c in cases]
    bs.set_inputs(pack_verts(other), pack_alphas(other))
    c2, g2 = bs.results(gamma=True)
    assert (c2 == co).all() and all((a == b).all() for a, b in zip(g2, g))
    bs.run(want_gamma=True)
    c3, _ = bs.results(gamma=True)
    _, (cr, _) = _solve(other, "shared")
    assert (c3 == cr).all()
