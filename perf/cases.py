"""Workloads of the implicit-step engine, measured one pass at a time.

A case is a dict: ``kind`` names the entry point, the other values its sizes
and options.  Kinds:

* ``spmv``     y = K x on device arrays (gsls_spmv_dev);
* ``assemble`` residual and tangent of one Newton iteration on device arrays
               (gsls_assemble_dev / gsls_assemble_ustruct_dev);
* ``solve``    one preconditioned Krylov solve, on host arrays
               (FSILS_SOLVE, the drop-in of a Fortran driver) or on device
               arrays (gsls_solve_dev);
* ``step``     one implicit time step (gsls_eq_step) from a given old state
               held on the device, as a sub-iterating or restarted program
               takes it: copy the old state in, step, read the new state;
* ``adjoint``  forward steps with checkpoints and the backward pass to the
               gradient with respect to the per-element parameter.

Meshes are those of ``svfsi_gb300.problems`` (Kuhn-split boxes and the
seeded cylinder).  The seed sets the matrices, states and material
parameters.
"""
from __future__ import annotations

import ctypes as C
import dataclasses
import functools
import math

import numpy as np
import torch

from svfsi_gb300 import _lib, fsils, meshgen, problems

DEV = "cuda"
F64 = torch.float64


# ---------------------------------------------------------------------------
# the cases
def listed():
    return [
        # y = K x of the heat cube (20^3 hexes, 48,000 tets): the smallest call
        dict(name="spmv_cube", kind="spmv", nx=20, ny=20, nz=20, d=1, prec="fp64"),
        # the same on the 2,044,416-tet beam, 3x3 blocks in FP32: the largest
        # matrix of the mixed path
        dict(name="spmv_beam", kind="spmv", nx=176, ny=44, nz=44, d=3, prec="mixed"),
        # drop-in solve on host arrays as the reference's driver calls it:
        # 3x3 blocks, CG + diagonal preconditioner, a small solid
        dict(name="solve_host_cg", kind="solve", where="host", ls="cg", nx=43, ny=11, nz=11, d=3),
        # nonsymmetric 4x4 blocks, restarted GMRES on device arrays, ragged box
        dict(name="solve_gmres", kind="solve", where="dev", ls="gmres", nx=61, ny=29, nz=17, d=4),
        # neo-Hookean beam, mixed precision: the assembly of the default run
        dict(name="assemble_struct", kind="assemble", phys="struct", prec="mixed", nx=176, ny=44,
             nz=44),
        # VMS Navier-Stokes in the cylinder, plain FP64
        dict(name="assemble_fluid", kind="assemble", phys="fluid", prec="fp64", h=0.04),
        # unsteady heat on the 48,000-tet cube, plain FP64: the small step
        dict(name="step_heats", kind="step", phys="heats", prec="fp64", nx=20, ny=20, nz=20),
        # monodomain slab, 2,952,450 tets, mixed: thousands of short steps
        dict(name="step_cep", kind="step", phys="cep", prec="mixed", nx=135, ny=135, nz=27),
        # heat carried by a flow, 1,225,440 tets, mixed, GMRES
        dict(name="step_heatf", kind="step", phys="heatf", prec="mixed", h=0.027),
        # neo-Hookean beam, 2,044,416 tets, mixed: the default run's step
        dict(name="step_struct", kind="step", phys="struct", prec="mixed", nx=176, ny=44, nz=44),
        # VMS Navier-Stokes, 1,225,440 tets, mixed, RCS + NS solver
        dict(name="step_fluid", kind="step", phys="fluid", prec="mixed", h=0.027),
        # discrete adjoint of the beam, plain FP64: forward and backward
        dict(name="adjoint_struct", kind="adjoint", prec="fp64", nx=60, ny=15, nz=15, steps=2),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _beam(rng, lo, hi):
    """nx x ny x nz of a beam of lo..hi hexes, odd sizes among them."""
    n = _log(rng, lo, hi)
    ny = max(2, round((n / 4.0) ** (1.0 / 3.0) * rng.uniform(0.8, 1.25)))
    nz = max(2, round((n / 4.0) ** (1.0 / 3.0) * rng.uniform(0.8, 1.25)))
    return dict(nx=max(2, round(n / (ny * nz))), ny=ny, nz=nz)


def draw(rng):
    """One more case of the ranges that the listed ones stand for."""
    kind = rng.choice(["spmv", "solve", "assemble", "step", "step", "step", "adjoint"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "spmv":
        return dict(kind=kind, d=rng.randint(1, 4), prec=prec, **_beam(rng, 500, 340000))
    if kind == "solve":
        ls = rng.choice(["cg", "gmres", "bicgs"])
        where = rng.choice(["host", "dev"])
        return dict(kind=kind, where=where, ls=ls, d=rng.randint(1, 4),
                    **_beam(rng, 500, 20000 if where == "host" else 60000))
    if kind == "assemble":
        phys = rng.choice(["struct", "lelas", "ustruct", "fluid", "heatf"])
        if phys in ("fluid", "heatf"):
            return dict(kind=kind, phys=phys, prec=prec, h=round(_log(rng, 0.027, 0.12), 4))
        return dict(kind=kind, phys=phys, prec=prec, **_beam(rng, 500, 340000))
    if kind == "adjoint":
        return dict(kind=kind, prec=prec, steps=rng.randint(1, 3), **_beam(rng, 300, 14000))
    phys = rng.choice(["heats", "cep", "struct", "lelas", "fluid", "heatf"])
    if phys == "heats":
        n = round(_log(rng, 6, 60))
        return dict(kind=kind, phys=phys, prec=prec, nx=n, ny=n, nz=max(3, n + rng.randint(-3, 3)))
    if phys == "cep":
        n = round(_log(rng, 24, 135))
        return dict(kind=kind, phys=phys, prec=prec, nx=n, ny=n, nz=max(4, n // 5),
                    ode=rng.randint(0, 1))
    if phys == "fluid":
        return dict(kind=kind, phys=phys, prec=prec, h=round(_log(rng, 0.04, 0.12), 4))
    if phys == "heatf":
        return dict(kind=kind, phys=phys, prec=prec, h=round(_log(rng, 0.027, 0.12), 4))
    return dict(kind=kind, phys=phys, prec=prec, **_beam(rng, 500, 340000 if prec == "mixed" else 100000))


# ---------------------------------------------------------------------------
# meshes and states
@functools.lru_cache(maxsize=4)
def _problem(phys, ode, nx, ny, nz, h):
    """Mesh, CSR, boundary conditions and solver settings of a case."""
    if phys == "heats":
        p = problems.heats_cube(nx) if nx == ny == nz else _heats_box(nx, ny, nz)
    elif phys == "cep":
        p = problems.cep_slab(nx, ny, nz, A=52.0, ode=ode)
    elif phys == "fluid":
        p = problems.fluid_cylinder(h=h)
    elif phys == "heatf":
        p = problems.heatf_cylinder(h=h)
    else:
        build = dict(struct=problems.struct_beam, lelas=problems.lelas_beam,
                     ustruct=problems.ustruct_beam)[phys]
        p = build(nx, ny, nz)
    return p


def _heats_box(nx, ny, nz):
    """The heat cube's problem on nx x ny x nz hexes."""
    x, ien = meshgen.kuhn_box(nx, ny, nz)
    rp, cp = meshgen.csr_from_ien(x.shape[0], ien)
    base = problems.heats_cube(2)
    faces = [problems.DirBC(meshgen.nodes_on_plane(x, 0, 0.0), 1.0),
             problems.DirBC(meshgen.nodes_on_plane(x, 0, 1.0), 0.0)]
    return dataclasses.replace(base, name=f"heats_box_{nx}x{ny}x{nz}", x=x, ien=ien, rowPtr=rp,
                               colPtr=cp, dirichlet=faces)


def _prob(case, phys=None):
    return _problem(phys or case["phys"], case.get("ode", 0), case.get("nx", 0),
                    case.get("ny", 0), case.get("nz", 0), case.get("h", 0.0))


@functools.lru_cache(maxsize=4)
def _graph(nx, ny, nz):
    """CSR of the beam's node graph (0-based, numpy)."""
    x, ien = meshgen.kuhn_box(nx, ny, nz, 4.0, 1.0, 1.0)
    rp, cp = meshgen.csr_from_ien(x.shape[0], ien)
    return x, rp, cp


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _smooth(x, seed, ncomp, modes=4):
    """Smooth random field (nNo, ncomp) of unit amplitude: a few sine modes."""
    rng = np.random.default_rng(seed)
    span = np.maximum(x.max(axis=0) - x.min(axis=0), 1e-12)
    z = (x - x.min(axis=0)) / span
    out = np.zeros((x.shape[0], ncomp))
    for c in range(ncomp):
        for _ in range(modes):
            k = rng.integers(1, 4, 3)
            out[:, c] += rng.standard_normal() / modes * np.prod(
                np.sin(np.pi * k * z + rng.uniform(0, np.pi, 3)), axis=1)
    return out


def _old_state(case, p, seed):
    """Old-step state (A, Y, D) of a running simulation, (nNo, tDof) each."""
    phys = case["phys"]
    A, Y, D = p.initial_state()
    if phys == "heats":
        Y[:, 0] = 1.0 - p.x[:, 0] + 0.2 * _smooth(p.x, seed, 1)[:, 0]
    elif phys == "cep":
        # a front part of the way through the slab and an uneven resting state
        rng = np.random.default_rng(seed)
        s = p.x[:, 0] + 0.3 * p.x[:, 1] - rng.uniform(2.0, 9.0)
        Y[:, 0] = -80.0 + 95.0 / (1.0 + np.exp(s / 0.25)) + 0.5 * _smooth(p.x, seed, 1)[:, 0]
    elif phys == "fluid":
        # part of the inflow's Poiseuille profile, disturbed off the wall
        rng = np.random.default_rng(seed)
        w = np.clip(1.0 - 4.0 * (p.x[:, 0] ** 2 + p.x[:, 1] ** 2), 0.0, None)
        Y[:, :3] = 1.5 * _smooth(p.x, seed, 3) * w[:, None]
        Y[:, 2] += 30.0 * rng.uniform(0.85, 0.95) * w
    elif phys == "heatf":
        Y[:, 4] = 1.0 - p.x[:, 2] / 5.0 + 0.1 * _smooth(p.x, seed, 1)[:, 0]
    else:
        # a beam in motion, at rest on the clamped face
        ramp = (p.x[:, 0] / 4.0)[:, None]
        D[:, :3] = 2e-3 * _smooth(p.x, seed, 3) * ramp
        Y[:, :3] = 0.2 * _smooth(p.x, seed + 1, 3) * ramp
        A[:, :3] = 10.0 * _smooth(p.x, seed + 2, 3) * ramp
    return A, Y, D


def _eparam(case, p, seed):
    """Per-element material parameter, log-normal around the nominal one."""
    name = dict(struct="C10", heats="cond", cep="Diso").get(case.get("phys", "struct"))
    if name is None:
        return None
    return p.params[name] * np.exp(0.2 * np.random.default_rng(seed + 3).standard_normal(p.nEl))


class _Ptr:
    """Device pointer of the library as a CUDA array; the tensor made of it
    holds this object and with it the equation that owns the memory."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(ptr, False),
                                             version=3, strides=None)


def _prec(case):
    return fsils.PREC_MIXED if case.get("prec") == "mixed" else fsils.PREC_FP64


def _own_stream(lhs):
    """A torch stream that the library's calls on this lhs share."""
    st = torch.cuda.Stream()
    _lib.check(_lib.load().gsls_set_stream(lhs.h, C.c_void_p(st.cuda_stream)), "gsls_set_stream")
    return st


# ---------------------------------------------------------------------------
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, int(seed))


def run(state):
    return state["run"](state)


# ---- y = K x
def _prepare_spmv(case, seed):
    x, rp, cp = _graph(case["nx"], case["ny"], case["nz"])
    d, n = case["d"], x.shape[0]
    lhs = fsils.FSILS_LHS_CREATE(n, n, cp.size, np.arange(1, n + 1), rp + 1, cp + 1, 1)
    g = _gen(seed)
    vt = torch.float32 if case["prec"] == "mixed" else F64
    val = torch.randn(cp.size, d, d, generator=g, device=DEV, dtype=F64).to(vt)
    v = torch.randn(n, d, generator=g, device=DEV, dtype=F64)
    # 16 bytes of slack after the values, as the engine's own matrices have
    buf = torch.zeros(val.numel() + 8, device=DEV, dtype=vt)
    buf[: val.numel()] = val.reshape(-1)
    return dict(run=_run_spmv, lhs=lhs, d=d, prec=_prec(case), val=buf, x=v,
                y=torch.empty_like(v), L=_lib.load())


def _run_spmv(s):
    _lib.check(s["L"].gsls_spmv_dev(s["lhs"].h, s["d"], s["val"].data_ptr(), s["prec"],
                                    s["x"].data_ptr(), s["y"].data_ptr()), "gsls_spmv_dev")
    return s["y"]


def _rows_cols(rp, cp):
    rp = torch.from_numpy(rp.astype(np.int64)).to(DEV)
    cols = torch.from_numpy(cp.astype(np.int64)).to(DEV)
    rows = torch.repeat_interleave(torch.arange(rp.numel() - 1, device=DEV), rp[1:] - rp[:-1])
    return rows, cols


def _matvec(rows, cols, val, x):
    y = torch.zeros_like(x)
    step = 1 << 20
    for k in range(0, rows.numel(), step):
        s = slice(k, k + step)
        y.index_add_(0, rows[s], torch.einsum("jrc,jc->jr", val[s], x[cols[s]]))
    return y


def _exact_spmv(case, seed):
    s = _prepare_spmv(case, seed)
    _, rp, cp = _graph(case["nx"], case["ny"], case["nz"])
    rows, cols = _rows_cols(rp, cp)
    d = case["d"]
    return _matvec(rows, cols, s["val"][: cp.size * d * d].double().reshape(-1, d, d), s["x"])


# ---- one Krylov solve
def _system(case, seed):
    """Block matrix of a diffusion on the mesh graph (CG) or an
    advection-diffusion (GMRES, BiCGStab), with a lumped mass; its solution
    and right-hand side."""
    x, rp, cp = _graph(case["nx"], case["ny"], case["nz"])
    d, n = case["d"], x.shape[0]
    rows, cols = _rows_cols(rp, cp)
    g = _gen(seed)
    # edge weights that are equal for (i, j) and (j, i): products of node values
    s = torch.exp(0.3 * torch.randn(n, generator=g, device=DEV, dtype=F64))
    off = rows != cols
    w = torch.where(off, s[rows] * s[cols], torch.zeros_like(s[rows]))
    mix = torch.randn(d, d, generator=g, device=DEV, dtype=F64)
    mix = torch.eye(d, device=DEV, dtype=F64) + 0.1 * (mix + mix.T) / d
    val = -w[:, None, None] * mix
    if case["ls"] != "cg":
        xs = torch.from_numpy(x).to(DEV)
        flow = torch.tensor([1.0, 0.3, 0.2], device=DEV, dtype=F64)
        edge = xs[cols] - xs[rows]
        adv = (edge @ flow) / edge.norm(dim=1).clamp_min(1e-12)
        val = val + (0.4 * w * adv)[:, None, None] * torch.eye(d, device=DEV, dtype=F64)
    diag = torch.zeros(n, device=DEV, dtype=F64).index_add_(0, rows, w)
    val = torch.where(off[:, None, None], val, ((1.05 * diag)[rows])[:, None, None] * mix)
    sol = torch.randn(n, d, generator=g, device=DEV, dtype=F64)
    return rows, cols, val, sol, _matvec(rows, cols, val, sol)


def _prepare_solve(case, seed):
    _, rp, cp = _graph(case["nx"], case["ny"], case["nz"])
    n = rp.size - 1
    lhs = fsils.FSILS_LHS_CREATE(n, n, cp.size, np.arange(1, n + 1), rp + 1, cp + 1, 1)
    _, _, val, _, rhs = _system(case, seed)
    typ = dict(cg=fsils.LS_TYPE_CG, gmres=fsils.LS_TYPE_GMRES, bicgs=fsils.LS_TYPE_BICGS)[case["ls"]]
    ls = fsils.FSILS_LS_CREATE(typ, relTol=1e-11, maxItr=40 if case["ls"] == "gmres" else 1000,
                               dimKry=50)
    if case["where"] == "host":
        val0, r0 = val.cpu().numpy(), rhs.cpu().numpy()
        return dict(run=_run_solve_host, lhs=lhs, ls=ls, d=case["d"], val0=val0, r0=r0,
                    val=np.empty_like(val0), r=np.empty_like(r0))
    return dict(run=_run_solve_dev, lhs=lhs, ls=ls, d=case["d"], stream=_own_stream(lhs),
                val0=val.contiguous(), r0=rhs, val=torch.empty_like(val).contiguous(),
                r=torch.empty_like(rhs), L=_lib.load())


def _run_solve_host(s):
    # the driver's assembly leaves a fresh Val and Ri before every call
    np.copyto(s["val"], s["val0"])
    np.copyto(s["r"], s["r0"])
    fsils.FSILS_SOLVE(s["lhs"], s["ls"], s["d"], s["r"], s["val"], fsils.PRECOND_FSILS)
    return {"x": s["r"], "val": s["val"]}


def _run_solve_dev(s):
    with torch.cuda.stream(s["stream"]):
        s["val"].copy_(s["val0"])
        s["r"].copy_(s["r0"])
        _lib.check(s["L"].gsls_solve_dev(s["lhs"].h, C.byref(s["ls"]), s["d"], s["r"].data_ptr(),
                                         s["val"].data_ptr(), fsils.PREC_FP64,
                                         fsils.PRECOND_FSILS, None, None), "gsls_solve_dev")
    return {"x": s["r"], "val": s["val"]}


def _exact_solve(case, seed):
    rows, cols, val, sol, _ = _system(case, seed)
    dg = val[rows == cols].diagonal(dim1=1, dim2=2)
    w = dg.abs().rsqrt()
    return {"x": sol, "val": w[rows][:, :, None] * val * w[cols][:, None, :]}


# ---- assembly
def _prepare_assemble(case, seed):
    p = _prob(case)
    g, rp1, cp1 = problems.make_lhs_arrays(p)
    lhs = fsils.FSILS_LHS_CREATE(p.nNo, p.nNo, p.nnz, g, rp1, cp1, 1)
    mesh = fsils.Mesh(lhs, p.ien, p.x)
    state = [torch.from_numpy(np.ascontiguousarray(a)).to(DEV) for a in _old_state(case, p, seed)]
    vt = torch.float32 if case["prec"] == "mixed" else F64
    out = dict(R=torch.empty(p.nNo, p.dof, device=DEV, dtype=F64),
               Val=torch.empty(p.nnz, p.dof * p.dof, device=DEV, dtype=vt))
    if case["phys"] == "ustruct":
        out["Kd"] = torch.empty(p.nnz, 12, device=DEV, dtype=F64)
    return dict(run=_run_assemble, lhs=lhs, mesh=mesh, params=p.eq_params(), state=state, out=out,
                prec=_prec(case), L=_lib.load())


def _run_assemble(s):
    a, y, d = (t.data_ptr() for t in s["state"])
    o = s["out"]
    if "Kd" in o:
        rc = s["L"].gsls_assemble_ustruct_dev(s["mesh"].h, C.byref(s["params"]), a, y, d,
                                              o["R"].data_ptr(), o["Val"].data_ptr(),
                                              o["Kd"].data_ptr(), s["prec"])
    else:
        rc = s["L"].gsls_assemble_dev(s["mesh"].h, C.byref(s["params"]), a, y, d,
                                      o["R"].data_ptr(), o["Val"].data_ptr(), s["prec"])
    _lib.check(rc, "gsls_assemble_dev")
    return o


def _exact_assemble(case, seed):
    """Neo-Hookean + ST91 element in closed form; the tangent from the
    derivative of the first Piola-Kirchhoff stress by automatic
    differentiation.  Other physics: none."""
    if case["phys"] != "struct":
        return None
    p = _prob(case)
    q = p.params
    A, Y, D = (torch.from_numpy(np.ascontiguousarray(a)).to(DEV) for a in _old_state(case, p, seed))
    xs = torch.from_numpy(p.x).to(DEV)
    ien = torch.from_numpy(p.ien.astype(np.int64)).to(DEV)
    rp = torch.from_numpy(p.rowPtr.astype(np.int64)).to(DEV)
    cp = torch.from_numpy(p.colPtr.astype(np.int64)).to(DEV)
    n = p.nNo
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), rp[1:] - rp[:-1])
    key = rows * n + cp
    s_, t_ = (5.0 + 3.0 * 5.0 ** 0.5) / 20.0, (5.0 - 5.0 ** 0.5) / 20.0
    N = torch.full((4, 4), t_, device=DEV, dtype=F64)
    N.fill_diagonal_(s_)
    M = N.T @ N
    R = torch.zeros(n, 3, device=DEV, dtype=F64)
    Val = torch.zeros(p.nnz, 9, device=DEV, dtype=F64)
    afu = q["af"] * q["beta"] * q["dt"] ** 2
    amd = q["am"] * q["rho"] + q["af"] * q["gam"] * q["dt"] * q["dmp"]
    eye = torch.eye(3, device=DEV, dtype=F64)

    def stress(F):
        J = torch.linalg.det(F)
        Ci = torch.linalg.inv(F.T @ F)
        S = J ** (-2.0 / 3.0) * 2.0 * q["C10"] * (eye - (F * F).sum() / 3.0 * Ci)
        return F @ (S + 0.5 * q["Kpen"] * (J - 1.0 / J) * J * Ci)

    tangent = torch.func.vmap(torch.func.jacfwd(stress))
    values = torch.func.vmap(stress)
    for e in range(0, p.nEl, 1 << 17):
        nd = ien[e: e + (1 << 17)]
        X = (xs[nd[:, :3]] - xs[nd[:, 3:]]).transpose(1, 2)
        Jac = torch.linalg.det(X)
        Xi = torch.linalg.inv(X)                       # rows: gradients of N_1..N_3
        Nx = torch.cat([Xi, -Xi.sum(1, keepdim=True)], 1)  # (e, a, i)
        w = Jac / 24.0
        F = eye + torch.einsum("eac,eam->ecm", D[nd], Nx)
        P, T = values(F), tangent(F)
        inert = q["rho"] * A[nd] + q["dmp"] * Y[nd]
        lR = 4.0 * w[:, None, None] * torch.einsum("eam,ecm->eac", Nx, P) + \
            w[:, None, None] * torch.einsum("ab,ebc->eac", M, inert)
        R.index_add_(0, nd.reshape(-1), lR.reshape(-1, 3))
        K = torch.einsum("eam,ermcl,ebl->eabrc", Nx, T, Nx)
        K = (4.0 * afu) * w[:, None, None, None, None] * K
        K = K + (amd * w)[:, None, None, None, None] * (M[:, :, None, None] * eye)
        pos = torch.searchsorted(key, (nd[:, :, None] * n + nd[:, None, :]).reshape(-1))
        Val.index_add_(0, pos, K.reshape(-1, 9))
    return {"R": R, "Val": Val}


# ---- one implicit step
def _prepare_step(case, seed):
    p = dataclasses.replace(_prob(case))
    p.eparam = _eparam(case, p, seed)
    lhs, mesh, eq = problems.build_equation(p, _prec(case))
    if case["phys"] == "cep":
        # CEPINTEG's first pass starts from the resting potential: take it
        # here, so that every pass starts from the state that is set
        eq.step()
    eq.set_state(*_old_state(case, p, seed))
    s = dict(run=_run_step, eq=eq, mesh=mesh, lhs=lhs, stream=_own_stream(lhs), ptrs={},
             shape=(p.nNo, p.tDof), L=_lib.load(),
             fields=3 if case["phys"] in ("struct", "lelas") else 2,
             pp=[C.c_void_p() for _ in range(3)])
    s["old"] = [t.clone() for t in _state_views(s)]
    torch.cuda.synchronize()
    return s


def _state_views(s):
    """The engine's resident (A, Y, D) as tensors (the buffers alternate)."""
    _lib.check(s["L"].gsls_eq_state_dev(s["eq"].h, *(C.byref(q) for q in s["pp"])),
               "gsls_eq_state_dev")
    out = []
    for q in s["pp"][: s["fields"]]:
        if q.value not in s["ptrs"]:
            s["ptrs"][q.value] = torch.as_tensor(_Ptr(s["eq"], q.value, s["shape"]), device=DEV)
        out.append(s["ptrs"][q.value])
    return out


def _run_step(s):
    with torch.cuda.stream(s["stream"]):
        for dst, src in zip(_state_views(s), s["old"]):
            dst.copy_(src)
    s["eq"].step()
    return dict(zip("AYD", _state_views(s)))


def _exact_step(case, seed):
    """Heat on up to 12,000 nodes: the step is linear, solved densely."""
    p = _prob(case)
    if case["phys"] != "heats" or p.nNo > 12000:
        return None
    q = p.params
    kap = torch.from_numpy(_eparam(case, p, seed)).to(DEV)
    Ao, Yo, _ = (torch.from_numpy(a[:, 0].copy()).to(DEV) for a in _old_state(case, p, seed))
    xs = torch.from_numpy(p.x).to(DEV)
    nd = torch.from_numpy(p.ien.astype(np.int64)).to(DEV)
    X = (xs[nd[:, :3]] - xs[nd[:, 3:]]).transpose(1, 2)
    Xi = torch.linalg.inv(X)
    Nx = torch.cat([Xi, -Xi.sum(1, keepdim=True)], 1)
    vol = torch.linalg.det(X) / 6.0
    me = (vol / 20.0)[:, None, None] * (1.0 + torch.eye(4, device=DEV, dtype=F64))
    ke = (vol * kap)[:, None, None] * torch.einsum("eai,ebi->eab", Nx, Nx)
    n = p.nNo
    flat = (nd[:, :, None] * n + nd[:, None, :]).reshape(-1)
    M = torch.zeros(n * n, device=DEV, dtype=F64).index_add_(0, flat, me.reshape(-1)).view(n, n)
    K = torch.zeros(n * n, device=DEV, dtype=F64).index_add_(0, flat, ke.reshape(-1)).view(n, n)
    dt, am, af, gam = q["dt"], q["am"], q["af"], q["gam"]
    An = Ao * (gam - 1.0) / gam
    Yn = Yo.clone()
    free = torch.ones(n, device=DEV, dtype=F64)
    for d in p.dirichlet:
        k = torch.from_numpy(d.nodes.astype(np.int64)).to(DEV)
        An[k], Yn[k], free[k] = 0.0, d.g, 0.0
    # dYn = gam dt dAn
    R = M @ (Ao + am * (An - Ao)) * q["rho"] + K @ (Yo + af * (Yn - Yo))
    T = am * q["rho"] * M + af * gam * dt * K
    T = free[:, None] * T * free + torch.diag(1.0 - free)
    dA = torch.linalg.solve(T, -free * R)
    return {"A": (An + dA)[:, None], "Y": (Yn + gam * dt * dA)[:, None]}


# ---- adjoint
def _prepare_adjoint(case, seed):
    p = dataclasses.replace(_prob(case, "struct"), tol=1e-12, maxItr=20, ls_relTol=1e-8)
    c = dict(case, phys="struct")
    p.eparam = _eparam(c, p, seed)
    lhs, mesh, eq = problems.build_equation(p, _prec(case))
    A, Y, D = _old_state(c, p, seed)
    target = D + 1e-3 * _smooth(p.x, seed + 5, 3)
    return dict(run=_run_adjoint, eq=eq, mesh=mesh, lhs=lhs, start=(A, Y, D), target=target,
                steps=case["steps"])


def _run_adjoint(s):
    eq = s["eq"]
    eq.set_state(*s["start"])
    tape = eq.adjoint_forward(s["steps"], every=2)
    D = eq.get_state()[2]
    grad = tape.backward(Dbar=D - s["target"])  # J = |D - target|^2 / 2
    tape.free()
    return {"D": D, "grad": grad}


# ---------------------------------------------------------------------------
def _sizes(case):
    """Nodes, elements, CSR blocks (from the mesh's regular structure)."""
    if case.get("h"):
        h, R, Lz = case["h"], 0.5, 5.0
        nr, nz = max(1, round(R / h)), max(1, round(Lz / h))
        n2 = 1 + sum(max(6, round(2 * math.pi * R * k / nr / h)) for k in range(1, nr + 1))
        nel = 3 * nz * (2 * n2 - 2 - round(2 * math.pi * R / h))
        return n2 * (nz + 1), nel, int(14.55 * n2 * (nz + 1))
    a, b, c = case["nx"], case["ny"], case["nz"]
    n = (a + 1) * (b + 1) * (c + 1)
    edges = a * (b + 1) * (c + 1) + (a + 1) * b * (c + 1) + (a + 1) * (b + 1) * c + \
        a * b * (c + 1) + a * (b + 1) * c + (a + 1) * b * c + a * b * c
    return n, 6 * a * b * c, n + 2 * edges


#: phys: (dof, state values per node, Newton iterations of a step, Krylov
#: iterations of a Newton iteration at the listed sizes)
_PHYS = dict(heats=(1, 1, 2, 45), cep=(1, 1, 4, 3), struct=(3, 3, 5, 380), lelas=(3, 3, 4, 380),
             ustruct=(4, 4, 10, 250), fluid=(4, 4, 7, 900), heatf=(1, 5, 10, 4))


def work(case):
    """Bytes and operations of one pass: matrix and vectors once per product
    that the method takes, state and mesh once per assembly."""
    n, nel, nnz = _sizes(case)
    sa = 4 if case.get("prec") == "mixed" else 8
    kind = case["kind"]
    if kind in ("spmv", "solve"):
        d = case["d"]
        mat = nnz * (d * d * sa + 4) + 4 * n
        if kind == "spmv":
            return dict(bytes=mat + 16 * n * d, flops=2 * nnz * d * d)
        its = dict(cg=90, gmres=60, bicgs=90)[case["ls"]]
        return dict(bytes=its * (mat + 16 * n * d), flops=its * 2 * nnz * d * d)
    d, td, newton, its = _PHYS[case.get("phys", "struct")]
    asm = 16 * nel + 24 * n + 3 * 8 * n * td + nnz * d * d * sa + 8 * n * d
    fl = dict(heats=100, cep=100, struct=1500, lelas=900, ustruct=4000, fluid=6000, heatf=1200)
    asm_fl = nel * fl[case.get("phys", "struct")]
    if kind == "assemble":
        return dict(bytes=asm + (96 * nnz if d == 4 and case["phys"] == "ustruct" else 0),
                    flops=asm_fl)
    it_b = nnz * (d * d * sa + 4) + 4 * n + 2 * n * d * sa
    b, f = newton * (asm + its * it_b), newton * (asm_fl + its * 2 * nnz * d * d)
    if kind == "adjoint":
        b, f = 3 * case["steps"] * b, 3 * case["steps"] * f
    return dict(bytes=b, flops=f)


def exact(case, seed):
    fn = globals().get("_exact_" + case["kind"])
    return fn(case, int(seed)) if fn else None
