"""A plan is used again after a run that failed: a wing so small that every
segment lies inside the cut-off has a zero AIC (a zero pivot in its first
column, reported), and the next inputs of the same plan must give, bit for
bit, the results of a plan that never saw it."""
import numpy as np
import pytest

from tinyvlm_gb300 import mesh as M
from tinyvlm_gb300.batch import BatchSolver, pack_alphas, pack_verts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["shared", "exact"])
@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("refine", [0, 1])
def test_plan_after_a_singular_system(cuda, mode, graph, refine):
    cases = M.batch_cases(3, seed=7, n_alpha=2, nc_range=(4, 9), ns_range=(6, 30))
    good = pack_verts(cases)
    small = [M.Case(c.verts.copy(), c.alphas, {}) for c in cases]
    small[1].verts[:3] *= 1e-12
    bs = BatchSolver(cases, mode=mode, refine=refine)
    bs.set_inputs(pack_verts(small), pack_alphas(cases))
    bs.run(graph=graph)
    with pytest.raises(RuntimeError, match="zero pivot"):
        bs.results()
    bs.set_inputs(good, pack_alphas(cases))
    bs.run(want_gamma=True, graph=graph)
    co, g = bs.results(gamma=True)
    fresh = BatchSolver(cases, mode=mode, refine=refine)
    fresh.set_inputs(good, pack_alphas(cases))
    fresh.run(want_gamma=True, graph=graph)
    cf, gf = fresh.results(gamma=True)
    assert (co == cf).all() and all((a == b).all() for a, b in zip(g, gf))
