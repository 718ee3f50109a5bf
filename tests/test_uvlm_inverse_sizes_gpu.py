"""A resident run with room for many steps multiplies by the AIC's inverse, one with
room for few solves: after the same steps both hold the same circulations.  Panel
counts beyond 256, where the identity is solved for by the dataflow launch with
many groups of right-hand sides (float), odd ones, so that the inverse's leading
dimension is not the panel count, and more than five tiles of the transposition.
Bar: each solve's forward error, at most cond(A) times its backward error (measured
up to 5 units of rounding, 2^-21 in float, where a product of three TF32 passes
keeps 21 bits, 2^-53 in double; 8 units here), for either of the two."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from tests.test_uvlm_graph_gpu import DT, Stepper
from tests.test_uvlm_gpu import pitch_plunge
from tinyvlm_gb300 import mesh as M
from tinyvlm_gb300._lib import call
from tinyvlm_gb300.uvlm import kinematics_arrays

pytestmark = pytest.mark.gpu


def _gamma(v, capacity, precision, steps):
    T, Td, fs, ref = kinematics_arrays(pitch_plunge(), capacity, DT)
    s = Stepper(v, T, Td, fs, ref, capacity, precision)
    for _ in range(steps):
        s.step()
    n = (v.shape[1] - 1) * (v.shape[2] - 1)
    cl, cm, g = np.zeros(capacity), np.zeros((capacity, 3)), np.zeros(n)
    call("gbvlm_uvlm_results", s.h, *[ctypes.c_void_p(x.ctypes.data) for x in (cl, cm, g)], None)
    return g


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("nc,ns", [(1, 257), (3, 171), (9, 65), (20, 45)])
def test_inverse_equals_solve(cuda, precision, nc, ns):
    v = M.rectangular(nc, ns, 1.0, 4.0).astype(np.float32)
    M.quarter_chord(v)
    A = O.vlm_run([v.astype(np.float64)], 0.0, dtype=np.float64, return_state=True)["lhs"]
    bar = 2 * 8 * np.linalg.cond(np.asarray(A)) * (2.0 ** -21 if precision == 32 else 2.0 ** -53)
    many, few = _gamma(v, 64, precision, 3), _gamma(v, 6, precision, 3)
    assert np.linalg.norm(many - few) <= bar * np.linalg.norm(few)
    assert (many != few).any()  # the two are not the same path
