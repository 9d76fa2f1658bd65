"""Host threads that solve on systems of different size at the same time: they
launch the same kernels with different amounts of shared memory, and no launch
is refused for another thread's amount.  Afterwards a solve has the bits of the
one before.
"""
import ctypes as C
import sys
import threading

import numpy as np
import pytest

from svfsi_gb300 import _lib, fsils, problems
from test_gpu_wcg import _graph, _system

pytestmark = pytest.mark.gpu


class _Cg:
    """Solves on one system: of two iterations, or over and over with a zero
    right-hand side, whose solution is zero again."""

    def __init__(self, gsls, torch, kind, d):
        rp, cp = _graph(kind)
        n = rp.size - 1
        V0, R0 = _system(rp, cp, d, 7)
        self.lhs = fsils.FSILS_LHS_CREATE(n, n, cp.size, np.arange(1, n + 1, dtype=np.int32),
                                          rp.astype(np.int32) + 1, cp.astype(np.int32) + 1, 1)
        self.V0, self.R0 = (torch.tensor(a, dtype=torch.float64, device="cuda") for a in (V0, R0))
        self.V, self.R = self.V0.clone(), self.R0.clone()
        self.ls = fsils.FSILS_LS_CREATE(fsils.LS_TYPE_CG, relTol=1e-6, maxItr=2)
        self.args = (self.lhs.h, C.byref(self.ls), d, C.c_void_p(self.R.data_ptr()),
                     C.c_void_p(self.V.data_ptr()), _lib.PREC_FP64, fsils.PRECOND_FSILS, None, None)
        self.call, self.torch = gsls.gsls_solve_dev, torch

    def again(self):
        _lib.check(self.call(*self.args), "gsls_solve_dev")

    def fresh(self):
        self.V.copy_(self.V0)
        self.R.copy_(self.R0)
        self.torch.cuda.synchronize()
        self.again()
        x = self.R.cpu().numpy()
        self.R.zero_()
        self.torch.cuda.synchronize()
        return x


class _Step:
    """Steps of a few Newton iterations from the same state."""

    def __init__(self, h, itr):
        p = problems.fluid_cylinder(h=h)
        p.maxItr = itr
        self.lhs, self.mesh, self.eq = problems.build_equation(p)
        self.old = p.initial_state()

    def again(self):
        self.eq.set_state(*self.old)
        self.eq.step()

    def fresh(self):
        self.again()
        return self.eq.get_state()[1]


def _together(small, big, n):
    """`big` n times while the other threads run their small ones over and over."""
    errors, end = [], threading.Event()

    def work(x, more):
        try:
            while more():
                x.again()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)

    want = [x.fresh().copy() for x in [big] + small]
    left = iter(range(n))
    th = [threading.Thread(target=work, args=(x, lambda: not end.is_set())) for x in small]
    last = threading.Thread(target=work, args=(big, lambda: next(left, None) is not None))
    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-5)
    try:
        for t in th + [last]:
            t.start()
        last.join()
    finally:
        end.set()
        for t in th:
            t.join()
        sys.setswitchinterval(interval)
    assert not errors, errors
    for x, w in zip([big] + small, want):
        assert np.array_equal(x.fresh(), w)


def test_cg_solves_of_several_threads(gsls):
    torch = pytest.importorskip("torch")
    # 2 KB of shared memory a block, and more than the 48 KB that need no attribute
    small = [_Cg(gsls, torch, ("box", 4, 3, 3), 3) for _ in range(3)]
    _together(small, _Cg(gsls, torch, ("box", 100, 25, 25), 3), 3000)


def test_schur_solves_of_several_threads(gsls):
    _together([_Step(0.25, 1) for _ in range(2)], _Step(0.04, 2), 12)
