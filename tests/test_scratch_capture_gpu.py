"""A wake sum and a roll-up captured into a graph after calls with fewer wake rows,
by a thread whose scratch those calls made: growing it for the larger sum would
need an allocation, which a capture does not allow.  The replay gives, bit for
bit, what the call gives outside."""
import threading

import numpy as np
import pytest
import torch

from tinyvlm_gb300 import backend as B
from tinyvlm_gb300 import mesh as M

pytestmark = pytest.mark.gpu


def _in_thread(f):
    err = []

    def g():
        try:
            f()
        except BaseException as e:
            err.append(e)
    t = threading.Thread(target=g)
    t.start()
    t.join()
    if err:
        raise err[0]


@pytest.mark.parametrize("td", [torch.float32, torch.float64])
@pytest.mark.parametrize("first", ["few rows", "another operator"])
@pytest.mark.parametrize("kind", ["wake", "rollup"])
def test_more_rows_under_capture(cuda, td, first, kind):
    nc, ns, rows, few = 20, 80, 150, 2
    rng = np.random.default_rng(1)
    wing = M.rectangular(nc, ns, 1.0, 4.0)
    wake = np.zeros((4, rows + 1, ns + 1))
    wake[0] = wing[0, -1] + 0.05 * np.arange(rows + 1)[::-1, None]
    wake[1], wake[3] = wing[1, -1], 1.0
    wake[2] = 0.01 * rng.standard_normal((rows + 1, ns + 1))
    d = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(td).cuda()
    w, k0, gk, gw = d(wing), d(wake), d(rng.uniform(0, 0.1, (rows, ns))), d(rng.uniform(0, 0.1, (nc, ns)))
    col, nor, ar = (torch.zeros(s, dtype=td, device="cuda") for s in ((3, nc, ns), (3, nc, ns), (nc, ns)))
    k, rhs = k0.clone(), torch.zeros(nc * ns, dtype=td, device="cuda")

    def work():
        st = torch.cuda.Stream()
        be = B.Backend(td, stream=st.cuda_stream)

        def call(n):
            if kind == "wake":
                be.rhs_assemble_wake_influence(rhs, [gk], [col], [nor], [k], [True], n)
            else:
                be.wake_rollup([k], [w], [gw], [gk], [True], 0.01, n)
        be.mesh_metrics(0.0, [w], [col], [nor], [ar])
        if first == "few rows":
            call(few)
        else:
            be.sum(ar)
        st.synchronize()
        k.copy_(k0)
        rhs.zero_()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            call(rows)
        g.replay()
        torch.cuda.synchronize()
        got = (k.clone(), rhs.clone())
        k.copy_(k0)
        rhs.zero_()
        torch.cuda.synchronize()
        call(rows)
        torch.cuda.synchronize()
        assert (got[0] == k).all() and (got[1] == rhs).all()
        assert bool((k != k0).any()) == (kind == "rollup") and bool((rhs != 0).any()) == (kind == "wake")
    _in_thread(work)
