"""int8 operands off the 16-byte grid: one or both copied onto it (align_i8), at every byte offset of the
base, odd leading dimensions, lines shorter than a vector and one byte past one, unevenly spaced
instances; bit for bit against the restated reference."""
import ctypes as ct

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (15, 17, 33), (16, 130, 129), (129, 31, 16), (257, 300, 100)])
@pytest.mark.parametrize("pads,shifts", [((0, 0, 0), (1, 0)), ((1, 16, 3), (0, 0)), ((3, 5, 1), (7, 13)),
                                         ((16, 2, 0), (0, 15))])
def test_align_copies(ta, tb, m, n, k, pads, shifts):
    import torch
    import ssblasex_b200 as S
    from ssblasex_b200 import workloads as W
    S.set_sync_mode(True)
    r16 = lambda x: (x + 15) // 16 * 16
    ar, br = (m if ta == 0 else k), (k if tb == 0 else n)
    lda = r16(ar) if pads[0] in (0, 16) else ar + pads[0]
    ldb = r16(br) if pads[1] in (0, 16) else br + pads[1]
    p = W.make_problem("i8", ta, tb, m, n, k, 3, 3, -2, lda=lda, ldb=ldb, ldc=m + pads[2], seed=m + n + k + pads[0])
    bufs, ptrs = [], []
    for i, X in enumerate((p.A, p.B, p.C)):
        size, shift = X[0].size, shifts[i] if i < 2 else 0
        per = r16(size) + 16
        at = [shift, shift + per, shift + 2 * per + (16 if shifts[0] == 7 else 0)]   # the last one off the spacing
        flat = torch.full((at[2] + size + 64,), 77, dtype=torch.from_numpy(X).dtype, device="cuda")
        for b in range(3):
            flat[at[b]: at[b] + size] = torch.from_numpy(X[b].reshape(-1)).cuda()
        bufs.append((flat, at, size))
        ptrs.append((ct.c_void_p * 3)(*[flat.data_ptr() + flat.element_size() * a for a in at]))
    al, be = np.array([p.alpha], np.int32), np.array([p.beta], np.int32)
    st = S.lib().ssblasGemmBatchedEx(ta, tb, m, n, k, al.ctypes.data, ptrs[0], S.SSBLAS_R_8I, lda, ptrs[1], S.SSBLAS_R_8I,
                                     ldb, be.ctypes.data, ptrs[2], S.SSBLAS_R_32I, p.ldc, 3, 0, 0)
    info = S.last_run_info()
    copied = lda % 16 or ldb % 16 or shifts[0] or shifts[1]
    assert st == 0 and info["path"] == "i8_tcgen05" and info["kernel_launches"] == (2 if copied else 1)
    flat, at, size = bufs[2]
    C = np.stack([flat[a: a + size].cpu().numpy() for a in at]).reshape(p.C.shape)
    np.testing.assert_array_equal(C, O.restated_gemm(p)[1])
    # the operands and everything around them are as they were
    for (f, at, size), X in zip(bufs[:2], (p.A, p.B)):
        host = f.cpu().numpy()
        keep = np.ones(host.size, bool)
        for b, a in enumerate(at):
            np.testing.assert_array_equal(host[a: a + size], X[b].reshape(-1))
            keep[a: a + size] = False
        assert np.all(host[keep] == 77)
