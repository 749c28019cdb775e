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


@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 1)])
def test_thin_operand_beyond_the_memory_left(ta, tb):
    """Lines of 3 bytes grow to 16 in the copy: where that does not fit the memory left, the call still runs."""
    import torch
    import ssblasex_b200 as S
    S.set_sync_mode(True)
    S.set_math_mode(S.SSBLAS_MATH_PLAIN)
    S.release_workspace()
    torch.cuda.empty_cache()
    thin, other, k, batch = 3, 16, 16384, 4200      # 206 MB of operand, 1.1 GB of copy
    g = torch.Generator(device="cuda").manual_seed(3)
    X = torch.randint(-128, 128, (batch, k, thin), generator=g, device="cuda", dtype=torch.int8)
    Y = torch.randint(-128, 128, (batch, other, k), generator=g, device="cuda", dtype=torch.int8)   # read in place
    C = torch.zeros((batch, other, thin) if ta == 0 else (batch, thin, other), dtype=torch.int32, device="cuda")
    px = torch.arange(batch, device="cuda") * X.stride(0) + X.data_ptr()
    py = torch.arange(batch, device="cuda") * Y.stride(0) + Y.data_ptr()
    pc = torch.arange(batch, device="cuda") * (C.stride(0) * 4) + C.data_ptr()
    one, zero = np.array([1], np.int32), np.array([0], np.int32)
    # op(A) op(B) with the thin operand, 3 x 16384 with its rows contiguous, as op(A) = A or as op(B) = B^T
    a, b, lda, ldb, m, n = (px, py, thin, k, thin, other) if ta == 0 else (py, px, k, thin, other, thin)
    left = torch.cuda.mem_get_info()[0]
    hold = torch.empty(left - (600 << 20), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    st = S.lib().ssblasGemmBatchedEx(ta, tb, m, n, k, one.ctypes.data, a.data_ptr(), S.SSBLAS_R_8I, lda, b.data_ptr(),
                                     S.SSBLAS_R_8I, ldb, zero.ctypes.data, pc.data_ptr(), S.SSBLAS_R_32I, m, batch, 0, 0)
    path = S.last_run_info()["path"]
    del hold
    torch.cuda.empty_cache()
    assert st == 0 and path == "simt"
    for i in (0, 1, batch // 2, batch - 1):
        want = Y[i].double() @ X[i].double()             # other x thin, whole numbers below 2^28
        got = C[i].double()
        assert torch.equal(got, want if ta == 0 else want.T)
