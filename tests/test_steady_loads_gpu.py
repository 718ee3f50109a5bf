"""The steady drivers' fused launches at the edges of their blocks (128 panels,
127 strips of chords, 32 strips of the nonlinear correction), one surface and
two, in double against the oracle.  Bars: those of the drivers' own tests, 1e-8
for the linear one, 5e-8 and 1e-6 (strip angles, returned as float) for the
nonlinear one; each run twice on one state."""
import math

import numpy as np
import pytest

from oracle import oracle as O
from tests.test_nlvlm_gpu import CURVES, _db
from tinyvlm_gb300 import mesh as M
from tinyvlm_gb300.vlm import NLVLM, VLM, FlowData

pytestmark = pytest.mark.gpu
SIZES = [[(1, 1)], [(1, 127)], [(1, 128)], [(1, 129)], [(2, 64)], [(3, 43)], [(1, 255)], [(2, 63), (1, 130)],
         [(3, 33), (2, 31)], [(4, 32)]]


def _wings(sizes):
    out = []
    for k, (nc, ns) in enumerate(sizes):
        v = M.rectangular(nc, ns, 1.0, 4.0 + 0.02 * ns).astype(np.float32)
        v[0] += 1.2 * k
        M.quarter_chord(v)
        out.append(v)
    return out


@pytest.mark.parametrize("sizes", SIZES, ids=str)
def test_linear(cuda, sizes):
    wings = _wings(sizes)
    sim = VLM("gb300", wings, precision=64)
    for adeg in (3.0, 7.0):
        al = math.radians(adeg)
        ref = O.vlm_run([v.astype(np.float64) for v in wings], al, dtype=np.float64, ref_pt=(0.25, 0.0, 0.0))
        got, g = sim.run(FlowData(al), ref_pt=(0.25, 0.0, 0.0), return_gamma=True)
        rg = np.concatenate([x.ravel() for x in ref["gamma"]])
        assert abs(got.cl - ref["cl"]) <= 1e-8 * abs(ref["cl"])
        assert np.linalg.norm(g - rg) <= 1e-8 * np.linalg.norm(rg)
        assert abs(got.cd - ref["cdi"]) <= 1e-8 * abs(ref["cdi"]) + 1e-9
        assert np.abs(np.array(got.cm) - ref["cm"]).max() <= 1e-8 * np.abs(ref["cm"]).max()


@pytest.mark.parametrize("sizes", SIZES, ids=str)
def test_nonlinear(cuda, sizes):
    wings = _wings(sizes)
    db, a, cl = _db(CURVES["spallart2"])
    sim = NLVLM("gb300", wings, precision=64)
    for adeg in (6.0, 17.0):
        al = math.radians(adeg)
        ref = O.nlvlm_run(wings, al, a, cl, dtype=np.float64, beta=math.radians(1.0))
        got = sim.run(FlowData(al, beta=math.radians(1.0)), db)
        assert sim.iters == ref["iters"]
        assert abs(got.cl - ref["cl"]) <= 5e-8 * abs(ref["cl"])
        for g, r in zip(sim.strip_alpha, ref["strip_alpha"]):
            np.testing.assert_allclose(g, r, rtol=0, atol=1e-6)
