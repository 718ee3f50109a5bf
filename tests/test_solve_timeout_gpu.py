"""A single-column solve whose wait runs out (its first block withheld: the
dispatch counter is one ahead, so nothing ever finishes that block; two
seconds) is reported by whoever hands out its results: the LU handle, the
strip-corrected solver, the coupled 2-DOF time loop, the unsteady driver step by
step and in its request loop.  The verdict sets the counters back, so the next
run gives, bit for bit, what a handle that never failed gives."""
import ctypes as C

import numpy as np
import pytest
import torch

from tests.test_uvlm_gpu import pitch_plunge
from tests.test_uvlm_graph_gpu import DT, Stepper
from tinyvlm_gb300 import _lib
from tinyvlm_gb300 import mesh as M
from tinyvlm_gb300._lib import call
from tinyvlm_gb300.aeroelastic import UVLM_2DOF, reference_vars
from tinyvlm_gb300.serve import UvlmLoop
from tinyvlm_gb300.uvlm import kinematics_arrays
from tinyvlm_gb300.vlm import NLVLM, Database, FlowData, WingProfile

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sfx,td", [("f32", torch.float32), ("f64", torch.float64)])
@pytest.mark.parametrize("n", [65, 128, 129, 300])
def test_lu_handle(cuda, sfx, td, n):
    L = _lib.lib()
    A = torch.randn((n, n), dtype=td, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    A += 2 * n * torch.eye(n, dtype=td, device="cuda")
    b = torch.ones(n, dtype=td, device="cuda")
    h = C.c_void_p()
    assert L.gbvlm_lu_create(C.byref(h)) == 0
    ptr = lambda t: C.c_void_p(t.data_ptr())

    def factor():
        F = A.clone()
        return F, getattr(L, "gbvlm_lu_factor_" + sfx)(h, ptr(F), n, n, None)

    def solve(F):
        x = b.clone()
        assert getattr(L, "gbvlm_lu_solve_" + sfx)(h, ptr(F), n, n, ptr(x), n, 1, None) == 0
        return x

    F, rc = factor()
    assert rc == 0
    x = solve(F)
    assert L.gbvlm_test_lu_solve_check(h, None) == 0
    for reader in ("check", "factor"):
        assert L.gbvlm_test_lu_withhold(h, None) == 0
        solve(F)
        solve(F)  # returns at once: the error word is set
        rc = L.gbvlm_test_lu_solve_check(h, None) if reader == "check" else factor()[1]
        assert rc == 2 and b"timed out" in L.gbvlm_last_error()
        assert (solve(F) == x).all() and L.gbvlm_test_lu_solve_check(h, None) == 0
    L.gbvlm_lu_destroy(h)


def _polar():
    a = np.linspace(0.0, 0.35, 40).astype(np.float32)
    db = Database()
    db.profiles.append(WingProfile(a, (5.0 * a).astype(np.float32)))
    return db


@pytest.mark.parametrize("precision", [32, 64])
def test_strip_corrected_solver(cuda, precision):
    L = _lib.lib()
    v = M.rectangular(5, 30, 1.0, 8.0).astype(np.float32)
    M.quarter_chord(v)
    sim = NLVLM("gb300", [v], precision=precision)
    want = sim.run(FlowData(0.1), _polar()).cl
    assert L.gbvlm_test_nlvlm_withhold(sim.h, None) == 0
    with pytest.raises(RuntimeError, match="timed out"):
        sim.run(FlowData(0.1), _polar())
    assert sim.run(FlowData(0.1), _polar()).cl == want


def test_coupled_time_loop(cuda):
    L = _lib.lib()
    v = M.rectangular(8, 10, 1.0, 40000.0).astype(np.float32)
    M.quarter_chord(v)
    sim = UVLM_2DOF([v], [1])
    sim.start(reference_vars(), 40.0)
    sim.advance(3)
    assert L.gbvlm_test_aero2dof_withhold(sim.h, None) == 0
    with pytest.raises(RuntimeError, match="timed out"):
        sim.advance(2, max_iter=3)
    fresh, again = UVLM_2DOF([v], [1]), sim
    again.start(reference_vars(), 40.0)
    again.advance(5)
    np.testing.assert_array_equal(again.results()["u"], fresh.run(reference_vars(), 40.0, steps=5)["u"])


@pytest.mark.parametrize("kind", ["step", "graph", "loop"])
def test_unsteady_steps(cuda, kind):
    L = _lib.lib()
    v = M.rectangular(4, 24, 1.0, 4.0).astype(np.float32)
    M.quarter_chord(v)
    steps = 8  # too few for the inverse: the steps solve
    T, Td, fs, ref = kinematics_arrays(pitch_plunge(), steps, DT)
    a = Stepper(v, T, Td, fs, ref, steps)
    want = [a.step(), a.step(graph=kind != "step"), a.step(graph=kind != "step")]
    b = Stepper(v, T, Td, fs, ref, steps)
    b.step()
    if kind == "loop":
        class Sim:
            h = b.h
        lp = UvlmLoop(Sim, 0.2)
        assert lp.wait(lp.submit(), 20.0)[1] == want[1][1]
        assert L.gbvlm_test_uvlm_withhold(b.h, None) == 0
        with pytest.raises(RuntimeError, match="timed out"):
            lp.wait(lp.submit(), 20.0)
        lp.close()
        with pytest.raises(RuntimeError, match="timed out"):  # the word is still set: the next factorisation reads it
            call("gbvlm_uvlm_begin", b.h, DT, 0, 0.0, None)
    else:
        assert L.gbvlm_test_uvlm_withhold(b.h, None) == 0
        with pytest.raises(RuntimeError, match="timed out"):
            b.step(graph=kind == "graph")
    call("gbvlm_uvlm_begin", b.h, DT, 0, 0.0, None)
    got = [b.step(), b.step(graph=kind != "step"), b.step(graph=kind != "step")]
    assert [x[1] for x in got] == [x[1] for x in want]
