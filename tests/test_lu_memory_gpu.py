"""Device memory that the factorisation without interchanges holds on to.  The copy
of a large matrix is given back with the factorisation's end (64 MB of it may
stay with the handle), and a plan of systems of up to 128 unknowns, which have no
rows or columns past their one block, holds no block workspace for them (131 KB
each before)."""
import numpy as np
import torch
import pytest

from tinyvlm_gb300 import backend as B
from tinyvlm_gb300 import mesh as M
from tinyvlm_gb300.batch import BatchSolver

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_the_copy_is_given_back(cuda):
    n = 12288  # 576 MB
    A = torch.full((n, n), 0.001, device="cuda")
    A.diagonal().fill_(10.0)
    be = B.Backend(torch.float32)
    lu = be.create_lu_solver()
    lu.init(A)
    W = A[:512, :512].contiguous()
    lu2 = be.create_lu_solver()
    lu2.factorize(W)  # modules loaded, the thread's scratch made
    before = _free()
    lu.factorize(A)
    held = before - _free()
    assert held <= 100 * MB, held / MB
    A[5, 5] = 0.0005  # needs an interchange, so the copy is looked at as well
    lu.factorize(A)
    assert before - _free() <= 100 * MB


def test_small_systems_have_no_block_workspace(cuda):
    warm = BatchSolver([M.Case(M.trapezoid(8, 12, 5.0, 0.5, 10.0).astype(np.float32), np.radians([1.0, 2.0]), {})])
    cases = [M.Case(M.trapezoid(8, 12, 4.0 + 0.001 * k, 0.5, 10.0).astype(np.float32), np.radians([1.0, 2.0]), {})
             for k in range(4096)]
    before = _free()
    bs = BatchSolver(cases)
    held = before - _free()
    # two float AICs, a double Trefftz matrix, and per panel and right-hand side some 200 bytes
    own = 4096 * (2 * 96 * 96 * 4 + 12 * 12 * 8 + 96 * 200 * 2)
    assert held <= own + 128 * MB, (held / MB, own / MB)
    del warm, bs
