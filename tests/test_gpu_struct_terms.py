"""STRUCT assembly with every term of the element in use: solid viscosity
(which has a kernel of its own), damping, body forces and a penalty of zero,
alone and together, against the oracle; and every gathered physics on meshes of
exactly 1, 31, 32, 33, 128 and 129 elements, the edges of a warp and a block.

Tolerances, relative to the largest entry: a block sums at most ~30 element
blocks, each formed by at most 200 roundings of 1.1e-16 (FP64, 7e-13) or 40 of
6e-8 (FP32 tangents, 7e-5).
"""
import ctypes as C
import dataclasses

import numpy as np
import pytest

from svfsi_gb300 import _lib, fsils, meshgen, problems

pytestmark = pytest.mark.gpu


def _check(gsls, orc, p, mixed):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(1)
    A, Y, D = p.initial_state()
    A = A + rng.standard_normal(A.shape)
    Y = Y + 0.1 * rng.standard_normal(Y.shape)
    D = D + 1e-3 * rng.standard_normal(D.shape)
    R0, V0 = orc.assemble(p, A, Y, D)
    g, rp1, cp1 = problems.make_lhs_arrays(p)
    lhs = fsils.FSILS_LHS_CREATE(p.nNo, p.nNo, p.nnz, g, rp1, cp1, 1)
    mesh = fsils.Mesh(lhs, p.ien, p.x)
    t = [torch.tensor(a, dtype=torch.float64, device="cuda") for a in (A, Y, D)]
    dR = torch.full((p.nNo * p.dof,), 7.0, dtype=torch.float64, device="cuda")
    dV = torch.full((p.nnz * p.dof ** 2,), 7.0, device="cuda",
                    dtype=torch.float32 if mixed else torch.float64)
    torch.cuda.synchronize()
    _lib.check(gsls.gsls_assemble_dev(mesh.h, C.byref(p.eq_params()),
                                      *(C.c_void_p(q.data_ptr()) for q in t),
                                      C.c_void_p(dR.data_ptr()), C.c_void_p(dV.data_ptr()),
                                      fsils.PREC_MIXED if mixed else fsils.PREC_FP64))
    R, V = dR.cpu().numpy(), dV.cpu().numpy().astype(np.float64)
    assert np.abs(R - R0.ravel()).max() <= 1e-12 * np.abs(R0).max()
    assert np.abs(V - V0.ravel()).max() <= (7e-5 if mixed else 1e-12) * np.abs(V0).max()
    mesh.free()
    lhs.free()


TERMS = [dict(visc=40.0), dict(dmp=900.0), dict(fb=(30.0, -2e4, 4e4)), dict(Kpen=0.0),
         dict(visc=40.0, dmp=900.0, fb=(30.0, -2e4, 4e4)),
         dict(visc=40.0, Kpen=0.0), dict(dmp=900.0, fb=(30.0, -2e4, 4e4), Kpen=0.0)]


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("terms", TERMS, ids=lambda t: "-".join(t))
def test_struct_terms(gsls, orc, terms, mixed):
    p = problems.struct_beam(7, 4, 3)
    _check(gsls, orc, dataclasses.replace(p, params=dict(p.params, **terms)), mixed)


def _truncated(phys, n):
    """The first n elements of a box, and their nodes alone."""
    x, ien = meshgen.kuhn_box(6, 2, 2, 4.0, 1.0, 1.0)
    nodes, ien = np.unique(ien[:n], return_inverse=True)
    ien = np.ascontiguousarray(ien.reshape(n, 4).astype(np.int32))
    x = np.ascontiguousarray(x[nodes])
    rp, cp = meshgen.csr_from_ien(x.shape[0], ien)
    p = {"struct": lambda: problems.struct_beam(1, 1, 1), "lelas": lambda: problems.lelas_beam(1, 1, 1),
         "fluid": lambda: problems.fluid_cylinder(h=0.5), "heatf": lambda: problems.heatf_cylinder(h=0.5)}[phys]()
    return dataclasses.replace(p, x=x, ien=ien, rowPtr=rp, colPtr=cp, dirichlet=[], traction=[],
                               neumann=[], Y0=None)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 128, 129])
@pytest.mark.parametrize("phys", ["struct", "lelas", "fluid", "heatf"])
def test_element_counts(gsls, orc, phys, n, mixed):
    _check(gsls, orc, _truncated(phys, n), mixed)
