"""FP32 row sums of the SpMV entry point keep one order, whatever number of
lanes shares a row: the blocks at even and at odd places of a row are two
chains of fused multiply-adds, added at the end.

The emulation takes each product in FP64, where it is exact (24 + 24 bits),
adds there and rounds to FP32: an FMA but for the sums that FP64 rounds onto a
tie of FP32, about one in 2^29.  So all values are equal, to the bit (the
largest case has 2.7 M sums).
"""
import ctypes as C

import numpy as np
import pytest

from svfsi_gb300 import _lib, fsils, meshgen

pytestmark = pytest.mark.gpu


def _fma32(a, x, s):
    return (a.astype(np.float64) * x + s).astype(np.float32)


def _row_sums(rp, cp, V, x):
    """y of two FP32 chains per row (V (nnz, d, d), x (n, d), both float32)."""
    n, d = x.shape
    acc = np.zeros((2, n, d), np.float32)
    for k in range(int(np.diff(rp).max())):
        i = np.flatnonzero(np.diff(rp) > k)
        j = rp[i] + k
        s = acc[k & 1][i]
        for c in range(d):
            s = _fma32(V[j, :, c], x[cp[j], c][:, None], s)
        acc[k & 1][i] = s
    return acc[0] + acc[1]


@pytest.mark.parametrize("d,n", [(1, (1, 1, 1)), (1, (20, 20, 20)), (1, (55, 41, 37)),
                                 (2, (5, 4, 3)), (2, (21, 20, 19)), (2, (45, 41, 30)),
                                 (3, (4, 3, 3)), (3, (33, 32, 31)), (4, (3, 3, 2)),
                                 (4, (24, 23, 22)), (4, (36, 33, 30))])
def test_fp32_row_sums_keep_their_order(gsls, d, n):
    torch = pytest.importorskip("torch")
    x, ien = meshgen.kuhn_box(*n)
    rp, cp = (np.asarray(a) for a in meshgen.csr_from_ien(x.shape[0], ien))
    nn = x.shape[0]
    lhs = fsils.FSILS_LHS_CREATE(nn, nn, cp.size, np.arange(1, nn + 1, dtype=np.int32),
                                 (rp + 1).astype(np.int32), (cp + 1).astype(np.int32), 1)
    rng = np.random.default_rng(d)
    V = rng.standard_normal((cp.size, d, d)).astype(np.float32)
    v = rng.standard_normal((nn, d))
    dV = torch.tensor(np.concatenate([V.ravel(), np.zeros(8, np.float32)]), device="cuda")
    dx = torch.tensor(v, dtype=torch.float64, device="cuda")
    dy = torch.full_like(dx, 7.0)
    torch.cuda.synchronize()
    _lib.check(gsls.gsls_spmv_dev(lhs.h, d, C.c_void_p(dV.data_ptr()), fsils.PREC_MIXED,
                                  C.c_void_p(dx.data_ptr()), C.c_void_p(dy.data_ptr())))
    want = _row_sums(rp, cp, V, v.astype(np.float32))
    assert np.array_equal(dy.cpu().numpy(), want.astype(np.float64))
    lhs.free()
