"""A VMS fluid step on the cylinder with its nodes numbered at random gives the
step of the mesh as it was, and runs its Schur CG in one launch per call: in
FP64 the windows of 97,000 scattered nodes do not fit in shared memory, those in
the order of the graph do.

Tolerance: both converge to 1e-10 of the first residual (Newton, with inexact
inner solves that start from different roundings), so that the states differ by
1e-8 at most relative to their norm.
"""
import ctypes as C
import dataclasses

import numpy as np
import pytest

from svfsi_gb300 import fsils, meshgen, problems

pytestmark = pytest.mark.gpu


def _shuffled(p, seed):
    new = np.random.default_rng(seed).permutation(p.nNo)
    old = np.argsort(new)
    ien = new[p.ien].astype(p.ien.dtype)
    rp, cp = meshgen.csr_from_ien(p.nNo, ien)
    # a profile goes with its nodes, in the order in which they are given
    dirichlet = [dataclasses.replace(b, nodes=new[b.nodes].astype(b.nodes.dtype)) for b in p.dirichlet]
    neumann = [dataclasses.replace(b, faces=new[b.faces].astype(b.faces.dtype)) for b in p.neumann]
    return dataclasses.replace(p, x=np.ascontiguousarray(p.x[old]), ien=ien, rowPtr=rp, colPtr=cp,
                               dirichlet=dirichlet, neumann=neumann), new


def test_fluid_step_on_scattered_nodes(gsls):
    p = problems.fluid_cylinder(h=0.035)
    q, new = _shuffled(p, 3)
    own = p.nNo // 152
    rows = slice(q.rowPtr[own * 70], q.rowPtr[own * 71])
    assert 8 * (4 * (np.unique(q.colPtr[rows]).size + own) + 3 * own) > 232448
    Y = []
    n, ms = C.c_longlong(), C.c_double()
    gsls.gsls_profile_enable(1)
    for prob in (p, q):
        lhs, mesh, eq = problems.build_equation(prob, fsils.PREC_FP64)
        gsls.gsls_profile_reset()
        eq.step()
        gsls.gsls_profile_read(b"schur", C.byref(n), C.byref(ms))
        assert n.value > 0
        Y.append(eq.get_state()[1])
        del eq
        mesh.free()
        lhs.free()
    gsls.gsls_profile_enable(0)
    assert np.linalg.norm(Y[1][new] - Y[0]) <= 1e-8 * np.linalg.norm(Y[0])
