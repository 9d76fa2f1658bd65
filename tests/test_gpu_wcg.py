"""The CG that runs as one cooperative launch on a row partition: block
sizes, precisions and mesh sizes at which the partition changes shape, against
the oracle's CG on the same system.

Edges: fewer rows than one block takes (32), one row more; a few rows per
block (several lanes per row); a slice more than the warps of a block; more
than 512 rows per block, where the rows are cut into strips; a random
numbering, whose halos are many times the own rows; a row without neighbours;
and a matrix whose windows do not fit in shared memory, which takes the
batched kernels.

Tolerance: both sides stop at |r| <= 1e-10 |r0| (FP64) on systems whose
diagonal exceeds the off-diagonal sum by a factor 1.5, so that the condition
number is below 5 and the two solutions differ by at most twice 5e-10.  The
FP32 solve (1e-5 on |r|) is held to twice 5e-5.
"""
import ctypes as C

import numpy as np
import pytest

from svfsi_gb300 import _lib, fsils, meshgen

pytestmark = pytest.mark.gpu


def _graph(kind):
    if kind[0] == "box":
        x, ien = meshgen.kuhn_box(*kind[1:])
        rp, cp = meshgen.csr_from_ien(x.shape[0], ien)
        return np.asarray(rp, np.int64), np.asarray(cp, np.int64)
    if kind[0] == "shuffled":
        rp, cp = _graph(("box",) + kind[1:])
        n = rp.size - 1
        new = np.random.default_rng(3).permutation(n)
        rows = new[np.repeat(np.arange(n), np.diff(rp))]
        cols = new[cp]
        o = np.lexsort((cols, rows))
        return np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]), cols[o]
    if kind[0] == "lonely":
        # a path of k nodes, then one node without neighbours
        k = kind[1]
        rows = np.concatenate([np.arange(k + 1), np.arange(k - 1), np.arange(1, k)])
        cols = np.concatenate([np.arange(k + 1), np.arange(1, k), np.arange(k - 1)])
    else:
        # random symmetric graph: every window holds most of the nodes
        n, m = kind[1], kind[2]
        rng = np.random.default_rng(4)
        a, b = rng.integers(0, n, m), rng.integers(0, n, m)
        rows = np.concatenate([np.arange(n), a, b])
        cols = np.concatenate([np.arange(n), b, a])
    key = np.unique(rows.astype(np.int64) * (cols.max() + 1) + cols)
    n = int(cols.max()) + 1
    rows, cols = key // n, key % n
    return np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]), cols


def _system(rp, cp, d, seed):
    """Symmetric block matrix, diagonally dominant by 1.5, and a right-hand side."""
    n = rp.size - 1
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(n), np.diff(rp))
    s = rng.uniform(0.5, 1.0, n)
    mix = np.eye(d) + 0.1 * np.ones((d, d)) / d
    w = s[rows] * s[cp]
    off = rows != cp
    val = -w[:, None, None] * mix
    deg = np.bincount(rows, weights=np.where(off, w, 0.0), minlength=n)
    val[~off] = (1.5 * deg + 0.1)[rows[~off], None, None] * mix
    return val.reshape(-1, d * d), rng.standard_normal((n, d))


CASES = [
    (("box", 2, 2, 2), 1), (("box", 2, 2, 2), 4),
    (("lonely", 31), 3), (("lonely", 32), 1),
    (("box", 7, 5, 3), 2), (("box", 13, 11, 9), 3), (("shuffled", 13, 11, 9), 3),
    (("box", 29, 24, 23), 1), (("box", 29, 24, 23), 4), (("box", 40, 20, 17), 2),
    (("box", 60, 38, 37), 1), (("box", 60, 38, 37), 3), (("shuffled", 30, 29, 28), 2),
    (("random", 60000, 300000), 4),
]


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("kind,d", CASES)
def test_partitioned_cg_matches_oracle(gsls, orc, kind, d, mixed):
    torch = pytest.importorskip("torch")
    rp, cp = _graph(kind)
    n, nnz = rp.size - 1, cp.size
    V0, R0 = _system(rp, cp, d, 7)
    tol = 1e-5 if mixed else 1e-10
    rp32, cp32 = rp.astype(np.int32), cp.astype(np.int32)
    lhs = fsils.FSILS_LHS_CREATE(n, n, nnz, np.arange(1, n + 1, dtype=np.int32), rp32 + 1,
                                 cp32 + 1, 1)
    s = orc.OracleSolver(n, rp32, cp32, 1)
    ols = orc.ls_create(orc.LS_TYPE_CG, relTol=1e-10, mItr=500)
    Ro, Vo = R0.copy(), V0.copy()
    s.solve(ols, d, Ro, Vo, orc.PRECOND_FSILS)
    out = []
    for _ in range(2):
        ls = fsils.FSILS_LS_CREATE(fsils.LS_TYPE_CG, relTol=tol, maxItr=500)
        dR = torch.tensor(R0, dtype=torch.float64, device="cuda")
        dV = torch.tensor(V0, dtype=torch.float32 if mixed else torch.float64, device="cuda")
        torch.cuda.synchronize()
        _lib.check(gsls.gsls_solve_dev(lhs.h, C.byref(ls), d, C.c_void_p(dR.data_ptr()),
                                       C.c_void_p(dV.data_ptr()),
                                       _lib.PREC_MIXED if mixed else _lib.PREC_FP64,
                                       fsils.PRECOND_FSILS, None, None), "gsls_solve_dev")
        assert ls.RI.suc == 1
        out.append(dR.cpu().numpy())
    err = np.linalg.norm(out[0] - Ro) / np.linalg.norm(Ro)
    assert err <= 10 * tol
    if not mixed:
        assert abs(ls.RI.itr - ols.RI.itr) <= 1
    assert np.array_equal(out[0], out[1])  # the same sums in every run
    lhs.free()
