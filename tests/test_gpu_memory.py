"""Device memory that cannot be had: solves and assemblies that fitted without
a second copy of the matrix, or without a whole element buffer, still run, and
do not ask for the same memory again on every call.

The library is given a budget (gsls_set_alloc_budget) in place of a full
device.  Tolerances: the solves stop at 1e-10 |r0| on systems with a condition
number below 5 (as in test_gpu_wcg.py); an assembly in parts has the bits of
the whole one, since a block's sum keeps its order; sums of ones are exact; steps of the NS solver
on either Schur CG stop at 1e-10 of the first residual.
"""
import ctypes as C

import numpy as np
import pytest

from svfsi_gb300 import _lib, fsils, problems
from test_gpu_wcg import _graph, _system

pytestmark = pytest.mark.gpu


@pytest.fixture
def budget(gsls):
    yield gsls.gsls_set_alloc_budget
    gsls.gsls_set_alloc_budget(-1)


def _profile(gsls, name):
    n, ms = C.c_longlong(), C.c_double()
    gsls.gsls_profile_read(name, C.byref(n), C.byref(ms))
    return n.value


@pytest.mark.parametrize("mixed", [False, True])
def test_cg_without_memory_for_the_stream(gsls, orc, budget, mixed):
    torch = pytest.importorskip("torch")
    rp, cp = _graph(("box", 40, 20, 17))
    n, d = rp.size - 1, 3
    V0, R0 = _system(rp, cp, d, 7)
    s = orc.OracleSolver(n, rp.astype(np.int32), cp.astype(np.int32), 1)
    Ro, Vo = R0.copy(), V0.copy()
    s.solve(orc.ls_create(orc.LS_TYPE_CG, relTol=1e-10, mItr=500), d, Ro, Vo, orc.PRECOND_FSILS)
    matrix = V0.size * (4 if mixed else 8)
    paths = set()
    gsls.gsls_profile_enable(1)
    # the workspaces of the batched kernels take less than 3 vectors of 64
    # bytes per unknown; the partition's stream takes a matrix and more
    for more in (0.0, 0.2, 0.6, 0.9, 1.3, 3.0):
        lhs = fsils.FSILS_LHS_CREATE(n, n, cp.size, np.arange(1, n + 1, dtype=np.int32),
                                     rp.astype(np.int32) + 1, cp.astype(np.int32) + 1, 1)
        budget(int(3 * 64 * n * d + more * matrix))
        for call in range(2):
            ls = fsils.FSILS_LS_CREATE(fsils.LS_TYPE_CG, relTol=1e-5 if mixed else 1e-10, maxItr=500)
            dR = torch.tensor(R0, dtype=torch.float64, device="cuda")
            dV = torch.tensor(V0, dtype=torch.float32 if mixed else torch.float64, device="cuda")
            torch.cuda.synchronize()
            gsls.gsls_profile_reset()
            a0 = gsls.gsls_alloc_count()
            _lib.check(gsls.gsls_solve_dev(lhs.h, C.byref(ls), d, C.c_void_p(dR.data_ptr()),
                                           C.c_void_p(dV.data_ptr()),
                                           _lib.PREC_MIXED if mixed else _lib.PREC_FP64,
                                           fsils.PRECOND_FSILS, None, None), "gsls_solve_dev")
            assert ls.RI.suc == 1
            assert np.linalg.norm(dR.cpu().numpy() - Ro) <= (1e-4 if mixed else 1e-9) * np.linalg.norm(Ro)
            if call:
                assert gsls.gsls_alloc_count() == a0
        one, many = (_profile(gsls, k) > 0 for k in (b"cg_persistent", b"cg_spmv"))
        assert one != many
        paths.add(one)
        budget(-1)
        lhs.free()
    gsls.gsls_profile_enable(0)
    assert paths == {False, True}


def _assemble(gsls, mesh, p):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(1)
    t = [torch.tensor(a + 1e-3 * rng.standard_normal(a.shape), device="cuda")
         for a in p.initial_state()]
    dR = torch.zeros(p.nNo * p.dof, dtype=torch.float64, device="cuda")
    dV = torch.zeros(p.nnz * p.dof ** 2, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    _lib.check(gsls.gsls_assemble_dev(mesh.h, C.byref(p.eq_params()),
                                      *(C.c_void_p(q.data_ptr()) for q in t),
                                      C.c_void_p(dR.data_ptr()), C.c_void_p(dV.data_ptr()),
                                      fsils.PREC_FP64))
    return dR.cpu().numpy(), dV.cpu().numpy()


def test_schur_cg_without_memory_for_the_streams(gsls, budget):
    p = problems.fluid_cylinder(h=0.1)
    p.ls_sD = 10
    paths, Y, need = set(), [], None
    gsls.gsls_profile_enable(1)
    # a step takes the NS solver's blocks, then the streams (7 values of 8 bytes
    # per CSR block and more), then a basis of 11 vectors (a quarter of them)
    for short in (None, 0.6, 0.8):
        lhs, mesh, eq = problems.build_equation(p)
        _assemble(gsls, mesh, p)  # the element buffer is there
        before = gsls.gsls_alloc_bytes()
        if short is not None:
            budget(int(need - short * 56 * p.nnz))
        for call in range(2):
            eq.set_state(*p.initial_state())
            gsls.gsls_profile_reset()
            a0 = gsls.gsls_alloc_count()
            eq.step()
            if call:
                assert gsls.gsls_alloc_count() == a0
        if need is None:
            need = gsls.gsls_alloc_bytes() - before
        Y.append(eq.get_state()[1])
        paths.add(_profile(gsls, b"schur") > 0)
        budget(-1)
        del eq
        mesh.free()
        lhs.free()
    gsls.gsls_profile_enable(0)
    assert paths == {False, True}
    # both stop at 1e-10 of the first residual
    for y in Y[1:]:
        assert np.linalg.norm(y - Y[0]) <= 1e-7 * np.linalg.norm(Y[0])


@pytest.mark.parametrize("d", [1, 3, 4])
def test_spmv_asks_for_no_memory(gsls, d):
    """The room for an FP32 copy of the vector comes with the lhs."""
    torch = pytest.importorskip("torch")
    rp, cp = _graph(("box", 100, 25, 25) if d < 4 else ("box", 60, 15, 15))
    n = rp.size - 1
    lhs = fsils.FSILS_LHS_CREATE(n, n, cp.size, np.arange(1, n + 1, dtype=np.int32),
                                 rp.astype(np.int32) + 1, cp.astype(np.int32) + 1, 1)
    dV = torch.ones(cp.size * d * d + 8, dtype=torch.float32, device="cuda")
    dx = torch.ones(n * d, dtype=torch.float64, device="cuda")
    dy = torch.empty_like(dx)
    torch.cuda.synchronize()
    a0 = gsls.gsls_alloc_count()
    _lib.check(gsls.gsls_spmv_dev(lhs.h, d, C.c_void_p(dV.data_ptr()), fsils.PREC_MIXED,
                                  C.c_void_p(dx.data_ptr()), C.c_void_p(dy.data_ptr())))
    assert gsls.gsls_alloc_count() == a0
    assert np.array_equal(dy.cpu().numpy().reshape(n, d)[:, 0], np.diff(rp) * d)
    lhs.free()


@pytest.mark.parametrize("phys", ["struct", "fluid"])
def test_assembly_in_the_parts_that_memory_allows(gsls, budget, phys):
    p = problems.struct_beam(40, 10, 10) if phys == "struct" else problems.fluid_cylinder(h=0.12)
    per = 16 * p.dof ** 2 * 8 + 32 * p.dof
    whole = per * p.nEl
    out = []
    for left in (None, 6.0, 2.2, 1.1, 0.3):
        g, rp1, cp1 = problems.make_lhs_arrays(p)
        lhs = fsils.FSILS_LHS_CREATE(p.nNo, p.nNo, p.nnz, g, rp1, cp1, 1)
        mesh = fsils.Mesh(lhs, p.ien, p.x)
        if left is not None:
            # the inverse map, 64 bytes per element and 12 per CSR block in all
            budget(int(64 * p.nEl + 12 * p.nnz + 4096 + max(left * whole, 4096 * per)))
        for call in range(2):
            a0 = gsls.gsls_alloc_count()
            res = _assemble(gsls, mesh, p)
            if call:
                assert gsls.gsls_alloc_count() == a0
        out.append(res)
        budget(-1)
        mesh.free()
        lhs.free()
    for R, V in out[1:]:
        assert np.array_equal(R, out[0][0]) and np.array_equal(V, out[0][1])
