"""Plain fp64 (DMMA) tiles at their edges: rows, columns and k around the 64 x 64 tile and the 16-deep
slab, aligned copies, 16-byte copies with a lone last row, and 8-byte copies (odd leading dimensions
or bases), against the FP64-exact oracle within 4 k u."""
import ctypes as ct

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", [(64, 64, 16), (63, 65, 15), (65, 1, 17), (1, 63, 48), (66, 130, 33), (127, 62, 50)])
@pytest.mark.parametrize("pad,shift", [(0, 0), (1, 0), (2, 1)])
def test_dmma_edges(ta, tb, m, n, k, pad, shift):
    import torch
    import ssblasex_b200 as S
    from ssblasex_b200 import workloads as W
    S.set_math_mode(S.SSBLAS_MATH_PLAIN)
    S.set_sync_mode(True)
    ar, br = (m if ta == 0 else k), (k if tb == 0 else n)
    p = W.make_problem("f64", ta, tb, m, n, k, 2, 0.75, -0.5, lda=ar + pad, ldb=br + pad, ldc=m + pad,
                       seed=m + 3 * n + 5 * k + pad)
    bufs, ptrs = [], []
    for X in (p.A, p.B, p.C):
        per = X[0].size + shift
        flat = torch.full((shift + per * 2,), float("nan"), dtype=torch.float64, device="cuda")
        for b in range(2):
            flat[shift + b * per: shift + b * per + X[b].size] = torch.from_numpy(X[b].reshape(-1)).cuda()
        bufs.append(flat)
        ptrs.append((ct.c_void_p * 2)(*[flat.data_ptr() + 8 * (shift + b * per) for b in range(2)]))
    al, be = np.array([p.alpha]), np.array([p.beta])
    st = S.lib().ssblasGemmBatchedEx(ta, tb, m, n, k, al.ctypes.data, ptrs[0], S.SSBLAS_R_64F, p.lda, ptrs[1],
                                     S.SSBLAS_R_64F, p.ldb, be.ctypes.data, ptrs[2], S.SSBLAS_R_64F, p.ldc, 2, 0, 0)
    assert st == 0 and S.last_run_info()["path"] == "dmma"
    flat, per = bufs[2].cpu().numpy(), p.C[0].size + shift
    C = np.stack([flat[shift + b * per: shift + b * per + p.C[0].size] for b in range(2)]).reshape(p.C.shape)
    assert O.normalized_error(p, C) <= 4 * k * 2.0 ** -53
    np.testing.assert_array_equal(C.reshape(2, n, -1)[:, :, m:], p.C.reshape(2, n, -1)[:, :, m:])
