"""The lattice sums (wake influence and roll-up) at the edges of their pieces
of 4 ring rows x 32 rings: one ring, remainders of both, several pieces, two
surfaces of which one does not lift, the core smoothing, and a wake longer
than the active rows.  Bars: those of the operators' own tests -- float
against the double oracle on the same inputs 2e-4 of the entry plus 2e-5 of
the largest, double 1e-9 and 1e-12; positions moved by a roll-up 1e-5 and
1e-6, 1e-12 and 1e-13.  The roll-up is checked in float with the core smoothing
only: the newest wake row lies within 1e-3 of the wing's trailing edge, where
the unsmoothed law in float has no digits to compare (an entry in a thousand
is off by up to 1e-4 with any order of evaluation)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.helpers import close, synthetic_wake, wing
from tinyvlm_gb300 import backend as B

pytestmark = pytest.mark.gpu

DT = [(np.float32, torch.float32), (np.float64, torch.float64)]
SHAPES = [(1, 1, 1), (2, 31, 3), (3, 32, 4), (5, 33, 5), (4, 65, 9), (3, 7, 40)]


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _d(xs):
    return [x.astype(np.float64) for x in xs]


def _case(shapes, npd, spare):
    rng = np.random.default_rng(len(shapes) + shapes[0][1])
    surf = [wing("trap", nc, ns, npd) for nc, ns, _ in shapes]
    for k, s in enumerate(surf):
        s[1] += npd(9.0 * k)  # side by side
    it = min(r for _, _, r in shapes)
    wakes = [synthetic_wake(s, r + 1 + spare, seed=k, dtype=npd) for k, (s, (_, _, r)) in enumerate(zip(surf, shapes))]
    gw = [rng.standard_normal((w.shape[1] - 1, w.shape[2] - 1)).astype(npd) for w in wakes]
    gs = [rng.standard_normal((s.shape[1] - 1, s.shape[2] - 1)).astype(npd) for s in surf]
    return surf, wakes, gw, gs, it


CASES = [([s], [True], spare, sigma) for s in SHAPES for spare, sigma in ((0, 0.0), (3, 0.05))]
CASES += [([SHAPES[3], SHAPES[1]], [True, False], 2, 0.0), ([SHAPES[1], SHAPES[3]], [True, True], 0, 0.05)]


@pytest.mark.parametrize("npd,td", DT)
@pytest.mark.parametrize("shapes,lifting,spare,sigma", CASES)
def test_wake_influence(cuda, npd, td, shapes, lifting, spare, sigma):
    surf, wakes, gw, _, it = _case(shapes, npd, spare)
    col, nor, _ = O.mesh_metrics(0.0, surf, npd)
    n = sum(c.shape[1] * c.shape[2] for c in col)
    rhs0 = np.linspace(-1, 1, n)
    ref = rhs0.copy()
    O.rhs_assemble_wake_influence(ref, _d(gw), _d(col), _d(nor), _d(wakes), lifting, it, sigma)
    be = B.Backend(td)
    be.sigma_vatistas = sigma
    got = T(rhs0.astype(npd))
    be.rhs_assemble_wake_influence(got, [T(g) for g in gw], [T(c) for c in col], [T(x) for x in nor],
                                   [T(w) for w in wakes], lifting, it)
    close(got.cpu().numpy(), ref, *((2e-4, 2e-5) if npd == np.float32 else (1e-9, 1e-12)), "wake influence")


@pytest.mark.parametrize("npd,td", DT)
@pytest.mark.parametrize("shapes,lifting,spare,sigma", CASES)
def test_rollup(cuda, npd, td, shapes, lifting, spare, sigma):
    if npd == np.float32 and sigma == 0.0:
        pytest.skip("ill-conditioned in float")
    surf, wakes, gw, gs, it = _case(shapes, npd, spare)
    ref = _d(wakes)
    O.wake_rollup(ref, _d(surf), _d(gs), _d(gw), lifting, 0.01, it, sigma)
    be = B.Backend(td)
    be.sigma_vatistas = sigma
    got = [T(w) for w in wakes]
    be.wake_rollup(got, [T(s) for s in surf], [T(g) for g in gs], [T(g) for g in gw], lifting, 0.01, it)
    for g, r in zip(got, ref):
        close(g.cpu().numpy(), r, *((1e-5, 1e-6) if npd == np.float32 else (1e-12, 1e-13)), "rollup")
