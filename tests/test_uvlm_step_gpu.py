"""The time step's three elementwise launches at the edges of their blocks (128
panels; 127 strips of chords), one surface and two: CL(t), CM(t) and the last
circulation in double against the oracle's time loop.  Bar: that of the UVLM
driver's own tests, 1e-9 of the value (a wing of up to 255 panels: n times the
condition of its AIC, some 1e3, times 2^-53 is 3e-11).  A run over two records
of kinematics checks that the block counter is back at zero after each step."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.test_uvlm_gpu import pitch_plunge
from tinyvlm_gb300 import mesh as M
from tinyvlm_gb300.kinematics import Assembly
from tinyvlm_gb300.uvlm import UVLM, kinematics_arrays

pytestmark = pytest.mark.gpu


def _wings(sizes):
    out = []
    for k, (nc, ns) in enumerate(sizes):
        v = M.rectangular(nc, ns, 1.0, 4.0 + 0.02 * ns).astype(np.float32)
        v[0] += 1.2 * k
        M.quarter_chord(v)
        out.append(v)
    return out


@pytest.mark.parametrize("sizes", [[(1, 1)], [(1, 127)], [(1, 128)], [(1, 129)], [(2, 64)], [(3, 43)], [(1, 254)],
                                   [(1, 255)], [(2, 63), (1, 130)], [(3, 3), (2, 127)]], ids=str)
def test_step(cuda, sizes):
    wings = _wings(sizes)
    base = pitch_plunge()
    asm = Assembly(base.kinematics())
    for k in range(len(wings)):
        asm.add("s%d" % k, base.surface_kinematics()[0])
    sim = UVLM("gb300", wings, precision=64)
    steps, dt = 7, 0.05
    T, Td, fs, ref = kinematics_arrays(asm, steps, dt)
    o = O.uvlm_run(wings, [True] * len(wings), T, Td, fs, ref, steps, dt, dtype=np.float64)
    for _ in range(2):
        r = sim.run(asm, t_steps=steps, dt=dt, return_gamma=True)
        np.testing.assert_allclose(r["cl"][1:-1], o["cl"][1:-1], rtol=1e-9, atol=1e-11)
        np.testing.assert_allclose(r["cm"][1:-1], o["cm"][1:-1], rtol=1e-9, atol=1e-11)
        np.testing.assert_allclose(r["gamma"], np.concatenate([x.ravel() for x in o["gamma"]]), rtol=1e-9, atol=1e-12)
