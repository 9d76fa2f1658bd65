"""FP32 tangents of a flat element: the node with the smallest shape gradient
has its own digits.

A needle of height 4000 on a base of size 1: the gradient of the apex is
1/4000, those of the base nodes about 1.  Its tangents in the mixed precision
are compared with those in FP64, row by row and column by column of the apex,
each relative to the largest entry of that row or column.  The time step is so
large that the inertia, which hides the gradients, is below 1e-3 of the rest.

Tolerance: an entry is formed by at most 40 roundings of 6e-8, of terms that
add up to at most twice the largest entry of the row or column (1.6 times, by
the elements' formulas with absolute values): 40 x 6e-8 x 2 = 4.8e-6.
A gradient that is minus the sum of three rounded ones is off by 6e-8 x 4000 =
2.4e-4.
"""
import ctypes as C
import dataclasses

import numpy as np
import pytest

from svfsi_gb300 import _lib, fsils, problems

H = 4000.0
TOL = 40 * 6e-8 * 2


def needle(phys, apex):
    """One-element problem with the needle's apex at place `apex` of the element."""
    base = np.array([[0.0, 0.0, 0.0], [1.1, 0.1, 0.0], [0.2, 0.9, 0.0]])
    x = np.zeros((4, 3))
    others = [k for k in range(4) if k != apex]
    x[others] = base
    x[apex] = [0.3, 0.4, H]
    ien = np.arange(4, dtype=np.int32)[None]
    if np.linalg.det(x[ien[0, :3]] - x[ien[0, 3]]) < 0:
        x[others[:2]] = x[others[1::-1]]
    p = {"struct": lambda: problems.struct_beam(1, 1, 1), "lelas": lambda: problems.lelas_beam(1, 1, 1),
         "fluid": lambda: problems.fluid_cylinder(h=0.5), "heatf": lambda: problems.heatf_cylinder(h=0.5)}[phys]()
    rp = np.arange(0, 17, 4, dtype=np.int32)
    cp = np.tile(np.arange(4, dtype=np.int32), 4)
    dt = 1e3 if phys in ("struct", "lelas") else 1e6
    return dataclasses.replace(p, x=x, ien=ien, rowPtr=rp, colPtr=cp, dirichlet=[], traction=[],
                               neumann=[], Y0=None, params=dict(p.params, dt=dt))


def state(phys, p):
    rng = np.random.default_rng(5)
    A, Y, D = (np.zeros((4, p.tDof)) for _ in range(3))
    if phys in ("fluid", "heatf"):
        Y[:, :3] = [1.0, 0.7, 0.9]
        Y[:, 3] = 0.1 * rng.standard_normal(4)
        if phys == "heatf":
            Y[:, 4] = rng.standard_normal(4)
    else:
        D[:, :] = 1e-3 * rng.standard_normal((4, 3))
        D[:, 2] = 0.0
    return A, Y, D


def parts(phys, V):
    """The tangent as (4, 4, r, c) blocks of one kind each."""
    d = {"fluid": 4, "heatf": 1}.get(phys, 3)
    K = V.reshape(4, 4, d, d)
    return [K] if d < 4 else [K[..., :3, :3], K[..., :3, 3:], K[..., 3:, :3], K[..., 3:, 3:]]


@pytest.mark.gpu
@pytest.mark.parametrize("apex", [0, 1, 2, 3])
@pytest.mark.parametrize("phys", ["struct", "lelas", "fluid", "heatf"])
def test_smallest_gradient_keeps_its_digits(gsls, phys, apex):
    torch = pytest.importorskip("torch")
    p = needle(phys, apex)
    g, rp1, cp1 = problems.make_lhs_arrays(p)
    lhs = fsils.FSILS_LHS_CREATE(p.nNo, p.nNo, p.nnz, g, rp1, cp1, 1)
    mesh = fsils.Mesh(lhs, p.ien, p.x)
    t = [torch.tensor(a, dtype=torch.float64, device="cuda") for a in state(phys, p)]
    prm = p.eq_params()
    out = []
    for prec, vt in ((fsils.PREC_FP64, torch.float64), (fsils.PREC_MIXED, torch.float32)):
        dR = torch.zeros(p.nNo * p.dof, dtype=torch.float64, device="cuda")
        dV = torch.zeros(p.nnz * p.dof ** 2, dtype=vt, device="cuda")
        torch.cuda.synchronize()
        _lib.check(gsls.gsls_assemble_dev(mesh.h, C.byref(prm), *(C.c_void_p(q.data_ptr()) for q in t),
                                          C.c_void_p(dR.data_ptr()), C.c_void_p(dV.data_ptr()), prec))
        out.append(parts(phys, dV.cpu().numpy().astype(np.float64)))
    for K, K32 in zip(*out):
        for k, k32 in ((K[apex], K32[apex]), (K[:, apex], K32[:, apex])):
            assert np.abs(k32 - k).max() <= TOL * np.abs(k).max()
    mesh.free()
    lhs.free()
