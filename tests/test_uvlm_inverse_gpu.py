"""Long runs, whose steps multiply by the AIC's inverse instead of solving: sizes
off the tiles of 32 and off the 16-byte rows, against the oracle's time loop
(bars of the UVLM driver's own tests: 1e-9 of the value in double, 2e-3 of the
largest CL in float), and against a run too short for the inverse (the same
steps; in double n cond u, about 1e2 x 1e3 x 1e-16, with a factor ten)."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.test_uvlm_gpu import pitch_plunge
from tinyvlm_gb300 import mesh as M
from tinyvlm_gb300.uvlm import UVLM, kinematics_arrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("nc,ns", [(1, 1), (1, 31), (3, 11), (5, 13), (1, 127), (4, 33)])
def test_long_run(cuda, precision, nc, ns):
    v = M.rectangular(nc, ns, 1.0, 4.0).astype(np.float32)
    M.quarter_chord(v)
    asm, dt, steps, few = pitch_plunge(), 0.06, 24, 12
    sim = UVLM("gb300", [v], precision=precision)
    r = sim.run(asm, t_steps=steps, dt=dt, return_gamma=True)
    T, Td, fs, ref = kinematics_arrays(asm, steps, dt)
    o = O.uvlm_run([v], [True], T, Td, fs, ref, steps, dt, dtype=np.float64)
    s = UVLM("gb300", [v], precision=precision).run(asm, t_steps=few, dt=dt)
    if precision == 64:
        np.testing.assert_allclose(r["cl"][1:-1], o["cl"][1:-1], rtol=1e-9, atol=1e-11)
        np.testing.assert_allclose(r["gamma"], np.concatenate([x.ravel() for x in o["gamma"]]), rtol=1e-9, atol=1e-12)
        np.testing.assert_allclose(r["cl"][1:few - 1], s["cl"][1:-1], rtol=1e-10, atol=1e-12)
    else:
        scale = np.abs(o["cl"][1:-1]).max()
        assert np.abs(r["cl"][1:-1] - o["cl"][1:-1]).max() <= 2e-3 * scale
        assert np.abs(r["cl"][1:few - 1] - s["cl"][1:-1]).max() <= 2e-3 * scale
