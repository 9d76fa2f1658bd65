"""Assembly through the element buffer, SpMV lane groups and the GMRES column
rotation at the sizes where their work splits: meshes of one element, fewer
elements than a warp, one more than a block of 128, and one whose FP64 element
matrices (4.4 GB) take the buffer twice; SpMV systems on both
sides of the lane-group rule; Krylov spaces on both sides of the 32 rotations
that one turn takes.

Tolerances.  Assembly, relative to the largest entry: a block sums at most ~30
element blocks, each formed by at most 200 roundings of 1.1e-16 (FP64, 7e-13)
or 40 of 6e-8 (FP32 tangents, 7e-5).  SpMV: sums of at most 60 products, 60 x 1.1e-16
(FP64) or 60 x 6e-8 (FP32) of sum |K||x|.  GMRES: both sides stop at 1e-8 |r0|
on a system with condition number < 10.
"""
import ctypes as C
import dataclasses

import numpy as np
import pytest

from svfsi_gb300 import _lib, fsils, meshgen, problems

pytestmark = pytest.mark.gpu


def _problem(phys, nx, ny, nz):
    if phys == "fluid" and nx:
        x, ien = meshgen.kuhn_box(nx, ny, nz, 4.0, 1.0, 1.0)
        rp, cp = meshgen.csr_from_ien(x.shape[0], ien)
        return dataclasses.replace(_problem("fluid", 0, 0, 0), x=x, ien=ien, rowPtr=rp, colPtr=cp,
                                   dirichlet=[], traction=[], neumann=[], Y0=None)
    build = {"struct": problems.struct_beam, "lelas": problems.lelas_beam}.get(phys)
    if build:
        return build(nx, ny, nz)
    q = (problems.fluid_cylinder if phys == "fluid" else problems.heatf_cylinder)(h=0.25, nsteps=1)
    return q


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("phys,n", [("struct", (1, 1, 1)), ("struct", (3, 1, 1)),
                                    ("struct", (11, 1, 2)), ("struct", (7, 3, 3)),
                                    ("lelas", (1, 1, 1)), ("lelas", (5, 2, 2)),
                                    ("fluid", None), ("heatf", None),
                                    ("fluid", (176, 44, 44))])
def test_gathered_assembly_matches_oracle(gsls, orc, phys, n, mixed):
    torch = pytest.importorskip("torch")
    p = _problem(phys, *(n or (0, 0, 0)))
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
    nv = p.nnz * p.dof ** 2
    dV = torch.full((nv + 1,), 7.0, device="cuda",
                    dtype=torch.float32 if mixed else torch.float64)
    prm = p.eq_params()
    torch.cuda.synchronize()
    for o in (0, 1):  # the second matrix starts off a 16-byte boundary
        dst = dV[o:o + nv]
        _lib.check(gsls.gsls_assemble_dev(mesh.h, C.byref(prm), *(C.c_void_p(q.data_ptr()) for q in t),
                                          C.c_void_p(dR.data_ptr()), C.c_void_p(dst.data_ptr()),
                                          fsils.PREC_MIXED if mixed else fsils.PREC_FP64))
        torch.cuda.synchronize()
        R, V = dR.cpu().numpy(), dst.cpu().numpy().astype(np.float64)
        assert np.abs(R - R0.ravel()).max() <= 1e-12 * np.abs(R0).max()
        assert np.abs(V - V0.ravel()).max() <= (7e-5 if mixed else 1e-12) * np.abs(V0).max()
    mesh.free()
    lhs.free()


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("d,n", [(1, (3, 2, 2)), (1, (20, 20, 20)), (1, (45, 44, 43)),
                                 (2, (5, 4, 3)), (2, (30, 29, 28)), (2, (40, 40, 40)),
                                 (3, (4, 3, 3)), (3, (33, 32, 31)), (4, (4, 4, 3)),
                                 (4, (24, 23, 22)), (4, (40, 33, 30))])
def test_spmv_lane_groups(gsls, d, n, mixed):
    torch = pytest.importorskip("torch")
    x, ien = meshgen.kuhn_box(*n)
    rp, cp = (np.asarray(a) for a in meshgen.csr_from_ien(x.shape[0], ien))
    nn = x.shape[0]
    lhs = fsils.FSILS_LHS_CREATE(nn, nn, cp.size, np.arange(1, nn + 1, dtype=np.int32),
                                 (rp + 1).astype(np.int32), (cp + 1).astype(np.int32), 1)
    rng = np.random.default_rng(d)
    V = rng.standard_normal((cp.size, d, d))
    v = rng.standard_normal((nn, d))
    if mixed:
        V, v = V.astype(np.float32).astype(float), v.astype(np.float32).astype(float)
    rows = np.repeat(np.arange(nn), np.diff(rp))
    ref, mag = np.zeros((nn, d)), np.zeros((nn, d))
    np.add.at(ref, rows, np.einsum("jrc,jc->jr", V, v[cp]))
    np.add.at(mag, rows, np.einsum("jrc,jc->jr", np.abs(V), np.abs(v[cp])))
    dV = torch.tensor(np.concatenate([V.ravel(), np.zeros(8)]), device="cuda",
                      dtype=torch.float32 if mixed else torch.float64)
    dx = torch.tensor(v, dtype=torch.float64, device="cuda")
    dy = torch.full_like(dx, 7.0)
    torch.cuda.synchronize()
    _lib.check(gsls.gsls_spmv_dev(lhs.h, d, C.c_void_p(dV.data_ptr()),
                                  fsils.PREC_MIXED if mixed else fsils.PREC_FP64,
                                  C.c_void_p(dx.data_ptr()), C.c_void_p(dy.data_ptr())))
    err = np.abs(dy.cpu().numpy() - ref)
    assert (err <= 60 * (6e-8 if mixed else 1.2e-16) * mag).all()
    lhs.free()


@pytest.mark.parametrize("dim", [1, 2, 31, 33, 70])
def test_gmres_rotation_sizes(gsls, orc, dim):
    p = problems.heats_cube(7)
    rp, cp = np.asarray(p.rowPtr), np.asarray(p.colPtr)
    rows = np.repeat(np.arange(p.nNo), np.diff(rp))
    rng = np.random.default_rng(dim)
    V0 = np.where(rows == cp, 28.0, -1.0 + 0.3 * rng.standard_normal(cp.size))[:, None]
    R0 = rng.standard_normal((p.nNo, 1))
    g, rp1, cp1 = problems.make_lhs_arrays(p)
    lhs = fsils.FSILS_LHS_CREATE(p.nNo, p.nNo, p.nnz, g, rp1, cp1, 1)
    ls = fsils.FSILS_LS_CREATE(fsils.LS_TYPE_GMRES, relTol=1e-8, maxItr=400, dimKry=dim)
    R, Val = R0.copy(), V0.copy()
    fsils.FSILS_SOLVE(lhs, ls, 1, R, Val, fsils.PRECOND_FSILS)
    s = orc.OracleSolver(p.nNo, p.rowPtr, p.colPtr, 1)
    ols = orc.ls_create(orc.LS_TYPE_GMRES, relTol=1e-8, mItr=400, sD=dim)
    Ro, Vo = R0.copy(), V0.copy()
    s.solve(ols, 1, Ro, Vo, orc.PRECOND_FSILS)
    assert ls.RI.suc == ols.RI.suc == 1
    assert np.linalg.norm(R - Ro) <= 2e-7 * np.linalg.norm(Ro)
    lhs.free()
