"""Which kernels a CG solve takes: the one launch on the row partition wherever
a block's window fits in shared memory, the batched kernels where it does not,
told apart by the library's profile counters.  A mesh numbered at random fits in
the order of its graph.

The graph that does not fit is random with 80 neighbours per node: a block of
the 152 (264 rows) sees about 16,000 other nodes, which with 16 bytes each (4
values in FP32) are more than the 227 KB of a block.

Tolerance: as in test_gpu_wcg.py.
"""
import ctypes as C

import numpy as np
import pytest

from svfsi_gb300 import _lib, fsils
from test_gpu_wcg import CASES, _graph, _system

pytestmark = pytest.mark.gpu


def _solve(gsls, torch, lhs, d, R0, V0, mixed, tol, itr):
    ls = fsils.FSILS_LS_CREATE(fsils.LS_TYPE_CG, relTol=tol, maxItr=itr)
    dR = torch.tensor(R0, dtype=torch.float64, device="cuda")
    dV = torch.tensor(V0, dtype=torch.float32 if mixed else torch.float64, device="cuda")
    torch.cuda.synchronize()
    gsls.gsls_profile_enable(1)
    gsls.gsls_profile_reset()
    _lib.check(gsls.gsls_solve_dev(lhs.h, C.byref(ls), d, C.c_void_p(dR.data_ptr()),
                                   C.c_void_p(dV.data_ptr()),
                                   _lib.PREC_MIXED if mixed else _lib.PREC_FP64,
                                   fsils.PRECOND_FSILS, None, None), "gsls_solve_dev")
    n, ms = C.c_longlong(), C.c_double()
    ran = []
    for name in (b"cg_persistent", b"cg_spmv"):
        gsls.gsls_profile_read(name, C.byref(n), C.byref(ms))
        ran.append(n.value > 0)
    gsls.gsls_profile_enable(0)
    return dR.cpu().numpy(), ran


def _lhs(rp, cp):
    n = rp.size - 1
    return fsils.FSILS_LHS_CREATE(n, n, cp.size, np.arange(1, n + 1, dtype=np.int32),
                                  rp.astype(np.int32) + 1, cp.astype(np.int32) + 1, 1)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("kind,d", CASES)
def test_windows_that_fit(gsls, kind, d, mixed):
    torch = pytest.importorskip("torch")
    rp, cp = _graph(kind)
    V0, R0 = _system(rp, cp, d, 7)
    lhs = _lhs(rp, cp)
    _, ran = _solve(gsls, torch, lhs, d, R0, V0, mixed, 1e-3, 3)
    assert ran == [True, False]
    lhs.free()


def test_windows_that_do_not_fit(gsls, orc):
    torch = pytest.importorskip("torch")
    rp, cp = _graph(("random", 40000, 1600000))
    n, d = rp.size - 1, 4
    own = n // 152
    seen = np.unique(cp[rp[own * 70]:rp[own * 71]])
    assert 16 * (seen.size + own) > 232448  # the kernel's window and products, of a middle block
    V0, R0 = _system(rp, cp, d, 7)
    s = orc.OracleSolver(n, rp.astype(np.int32), cp.astype(np.int32), 1)
    Ro, Vo = R0.copy(), V0.copy()
    s.solve(orc.ls_create(orc.LS_TYPE_CG, relTol=1e-10, mItr=500), d, Ro, Vo, orc.PRECOND_FSILS)
    for mixed in (False, True):
        lhs = _lhs(rp, cp)
        held = gsls.gsls_alloc_bytes()
        _, ran = _solve(gsls, torch, lhs, d, R0, V0, mixed, 1e-3, 1)
        assert ran == [False, True]
        # the workspaces (76 bytes per unknown), not the tables of a partition
        # that nothing uses (6 bytes per matrix block)
        assert gsls.gsls_alloc_bytes() - held < 80 * n * d + 3 * cp.size
        tol = 1e-5 if mixed else 1e-10
        x, ran = _solve(gsls, torch, lhs, d, R0, V0, mixed, tol, 500)
        assert ran == [False, True]
        assert np.linalg.norm(x - Ro) <= 10 * tol * np.linalg.norm(Ro)
        lhs.free()


@pytest.mark.parametrize("mixed", [False, True])
def test_scattered_numbering_takes_the_order_of_the_graph(gsls, orc, mixed):
    """120 x 100 x 20 hexes numbered at random: windows of 25,000 entries, which
    do not fit with 3 values each, and of 3,500 in the order of the graph."""
    torch = pytest.importorskip("torch")
    rp, cp = _graph(("shuffled", 120, 100, 20))
    n, d = rp.size - 1, 3
    own = n // 152
    seen = np.unique(cp[rp[own * 70]:rp[own * 71]])
    assert 4 * d * (seen.size + own) > 232448
    V0, R0 = _system(rp, cp, d, 7)
    s = orc.OracleSolver(n, rp.astype(np.int32), cp.astype(np.int32), 1)
    Ro, Vo = R0.copy(), V0.copy()
    s.solve(orc.ls_create(orc.LS_TYPE_CG, relTol=1e-10, mItr=500), d, Ro, Vo, orc.PRECOND_FSILS)
    lhs = _lhs(rp, cp)
    tol = 1e-5 if mixed else 1e-10
    x, ran = _solve(gsls, torch, lhs, d, R0, V0, mixed, tol, 500)
    assert ran == [True, False]
    assert np.linalg.norm(x - Ro) <= 10 * tol * np.linalg.norm(Ro)
    lhs.free()
