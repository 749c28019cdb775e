"""Plain fp32 and 3xBF16 on the BF16 tensor cores with the operands split inside the kernel
(f32_split.cu), against the FP64-exact oracle.

Tolerance of the plain form, derived from its arithmetic, in units of u = 2^-24 times
|alpha| |op(A)||op(B)| + |beta||C|: per chunk of 32 k two truncations at full magnitude (2 u each) and
the rounding of the small products (below 2^-7 of it) make at most 5 u, left-out products at most
1 u, every chunk sum is rounded once when it is added (k / 32 u), alpha and beta 2 u: k / 32 + 8."""
import ctypes as ct
import dataclasses

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
U = 2.0 ** -24


@pytest.fixture(scope="module")
def S():
    import torch
    assert torch.cuda.is_available()
    import ssblasex_b200 as S
    S.set_math_mode(S.SSBLAS_MATH_PLAIN)
    S.set_sync_mode(True)
    yield S
    S.set_math_mode(S.SSBLAS_MATH_PLAIN)


def problem(ta, tb, m, n, k, batch, beta, pads, seed, dist="uniform"):
    from ssblasex_b200 import workloads as W
    ar, br = (m if ta == 0 else k), (k if tb == 0 else n)
    return W.make_problem("f32", ta, tb, m, n, k, batch, 0.75, beta, lda=ar + pads[0], ldb=br + pads[1],
                          ldc=m + pads[2], seed=seed, dist=dist)


def run(S, p, pad=0, C=None):
    """One call with host arrays of device pointers; each instance starts `pad` floats further on, so odd
    pads break the 16-byte alignment and the spacing."""
    import torch
    bufs, ptrs = [], []
    for X in (p.A, p.B, p.C if C is None else C):
        per = X[0].size + pad
        flat = torch.full((pad + per * p.batch,), float("nan"), dtype=torch.float32, device="cuda")
        for b in range(p.batch):
            flat[pad + b * per: pad + b * per + X[b].size] = torch.from_numpy(X[b].reshape(-1)).cuda()
        bufs.append(flat)
        ptrs.append((ct.c_void_p * p.batch)(*[flat.data_ptr() + 4 * (pad + b * per) for b in range(p.batch)]))
    al, be = np.array([p.alpha], np.float32), np.array([p.beta], np.float32)
    st = S.lib().ssblasGemmBatchedEx(p.transa, p.transb, p.m, p.n, p.k, al.ctypes.data, ptrs[0], S.SSBLAS_R_32F, p.lda,
                                     ptrs[1], S.SSBLAS_R_32F, p.ldb, be.ctypes.data, ptrs[2], S.SSBLAS_R_32F, p.ldc,
                                     p.batch, 0, 0)
    assert st == 0
    flat, per = bufs[2].cpu().numpy(), p.C[0].size + pad
    return np.stack([flat[pad + b * per: pad + b * per + p.C[0].size] for b in range(p.batch)]).reshape(p.C.shape)


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("shape", [(64, 64, 128, 5), (65, 63, 129, 3), (128, 128, 160, 2), (129, 65, 191, 2),
                                   (1, 1, 128, 3), (127, 257, 255, 2), (300, 200, 161, 40), (40, 30, 300, 700)])
@pytest.mark.parametrize("pads,pad,beta", [((0, 0, 0), 0, 0.0), ((4, 8, 4), 0, 0.25), ((3, 1, 2), 1, -1.5)])
def test_plain_against_exact(S, ta, tb, shape, pads, pad, beta):
    m, n, k, batch = shape
    p = problem(ta, tb, m, n, k, batch, beta, pads, 31 + m + 2 * ta + tb, "outliers" if m == 300 else "uniform")
    C0 = p.C.copy()
    if beta == 0.0:                       # beta == 0 never reads C
        C0.reshape(batch, n, -1)[:, :, :m] = np.nan
    C = run(S, p, pad, C0)
    assert S.last_run_info()["path"] == "f32_tcgen05"
    for b in range(0, batch, max(1, batch // 3)):
        ex, nrm = O.exact_f64(p, b)
        err = np.abs(p.c_view(C, b).astype(np.float64) - ex)
        assert np.all(err <= (k / 32 + 8) * U * nrm)
    np.testing.assert_array_equal(C.reshape(batch, n, -1)[:, :, m:], C0.reshape(batch, n, -1)[:, :, m:])


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("ta,tb,pad", [(0, 0, 0), (0, 1, 3), (1, 0, 4), (1, 1, 1)])
def test_pair_tiles(S, mode, ta, tb, pad):
    """Ragged 256 x 256 tiles of CTA pairs (one per instance, 70 for 74 pairs), beside the same instances
    one by one, whose tiles are a single CTA's: equal bit for bit, and within the bound."""
    m, n, k, batch = 250, 255, 1000, 70
    p = problem(ta, tb, m, n, k, batch, 0.25, (pad, pad, pad), 91 + ta, "outliers")
    S.set_math_mode(mode)
    try:
        C = run(S, p)
        for b in (0, 37, 69):
            one = dataclasses.replace(p, batch=1, A=p.A[b:b + 1], B=p.B[b:b + 1], C=p.C[b:b + 1])
            np.testing.assert_array_equal(run(S, one).view(np.uint32), C[b:b + 1].view(np.uint32))
            ex, nrm = O.exact_f64(one, 0)
            bound = (k / 32 + 8) * U if mode == 0 else 2.0 ** -14
            assert np.all(np.abs(p.c_view(C, b).astype(np.float64) - ex) <= bound * nrm)
    finally:
        S.set_math_mode(0)
    np.testing.assert_array_equal(C.reshape(batch, n, -1)[:, :, m:], p.C.reshape(batch, n, -1)[:, :, m:])


@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 1)])
@pytest.mark.parametrize("kind", ["inf", "nan", "huge", "tiny", "zero"])
def test_plain_ends_of_the_range(S, ta, tb, kind):
    """Inf, NaN, values that round to Inf in BF16 or overflow when scaled, subnormals and elements
    whose low bits are below BF16's range: what an FFMA chain gives. Inf and NaN exactly; the others within
    the FP32 bound of the exact product, with FP32's own underflow (2^-149 per term)."""
    m, n, k = 70, 90, 140
    p = problem(ta, tb, m, n, k, 2, 0.0, (0, 0, 0), 5)
    rng = np.random.default_rng(3)
    opa, opb = p.op_a(0), p.op_b(0)
    if kind == "inf":
        opa[3, 7], opb[9, 11], opb[:, 20] = np.inf, -np.inf, 0.0
    elif kind == "nan":
        opa[69, 139], opb[0, 0] = np.nan, np.nan
    elif kind == "huge":
        opa[5, :], opb[:, 6] = 3.395e38 * np.sign(opa[5, :]), opb[:, 6] * np.float32(2.0 ** -100)
        opa[6, :] = opa[6, :] * np.float32(2.0 ** 110)
    elif kind == "tiny":
        opa[2, :] = (rng.integers(-2 ** 20, 2 ** 20, k) * 2.0 ** -149).astype(np.float32)
        opb[:, 4] = (rng.standard_normal(k) * 2.0 ** -115).astype(np.float32)
        opa[8, :] = 0.0
        opa[8, 1], opb[1, 5] = np.float32(1.2345678e-35), 1.0
    else:
        opa[:], opb[:, ::2] = 0.0, 0.0
    C = run(S, p)
    S.set_kernel_config("simt", 3)
    try:
        R = run(S, p)
    finally:
        S.set_kernel_config("simt", -1)
    got, ref = p.c_view(C, 0), p.c_view(R, 0)
    if kind in ("inf", "nan"):
        np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
        np.testing.assert_array_equal(got[np.isinf(ref)], ref[np.isinf(ref)])
        np.testing.assert_array_equal(np.isinf(got), np.isinf(ref))
    ok = np.isfinite(ref)
    A, B = opa.astype(np.float64), opb.astype(np.float64)
    A, B = np.where(np.isfinite(A), A, 0.0), np.where(np.isfinite(B), B, 0.0)
    ex, nrm = 0.75 * (A @ B), 0.75 * (np.abs(A) @ np.abs(B))
    with np.errstate(over="ignore", invalid="ignore"):
        fine = ok & (nrm < 2.0 ** 127)
        assert np.all(np.abs(got.astype(np.float64) - ex)[fine] <= (4 * k * U * nrm + k * 2.0 ** -149)[fine])
    np.testing.assert_array_equal(np.isfinite(got), ok)


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("shape", [(200, 130, 31, 3), (129, 64, 33, 2), (50, 300, 100, 4), (64, 64, 1, 3)])
@pytest.mark.parametrize("pad", [0, 1])
def test_bf16x3_split_in_kernel(S, ta, tb, shape, pad):
    """Configuration 3 of the 3xBF16 mode: the products of the emulation oracle, accumulated in FP32."""
    m, n, k, batch = shape
    p = problem(ta, tb, m, n, k, batch, 0.25, (pad, pad, 3), 77 + m + 2 * ta + tb, "outliers")
    S.set_math_mode(S.SSBLAS_MATH_FP32_BF16X3)
    S.set_kernel_config("bf16x3_tcgen05", 3)
    try:
        C = run(S, p, pad)
        info = S.last_run_info()
    finally:
        S.set_kernel_config("bf16x3_tcgen05", -1)
        S.set_math_mode(S.SSBLAS_MATH_PLAIN)
    assert info["path"] == "bf16x3_tcgen05" and info["kernel_launches"] == 1
    for b in range(batch):
        emu = O.bf16x3_f32(p, b)
        _, nrm = O.exact_f64(p, b)
        assert np.max(np.abs(p.c_view(C, b).astype(np.float64) - emu) / nrm) <= 4 * k * U
    np.testing.assert_array_equal(C.reshape(batch, n, -1)[:, :, m:], p.C.reshape(batch, n, -1)[:, :, m:])


def test_skipped_chunk_is_reported(S):
    """A converter signal that never comes: the waits run out, the call reports it, the next is right."""
    p = problem(0, 0, 200, 200, 200, 3, 0.0, (0, 0, 0), 9)
    assert S.set_fault_injection(S.SSBLAS_FAULT_SKIP_COPY) == 0
    from ssblasex_b200 import runner
    dp = runner.DeviceProblem(p)
    st, _ = runner.call(p, mode="host_array", dp=dp)
    assert st == S.SSBLAS_STATUS_INTERNAL_ERROR and S.last_run_info()["device_error"] != 0
    C = run(S, p)
    ex, nrm = O.exact_f64(p, 0)
    assert np.all(np.abs(p.c_view(C, 0).astype(np.float64) - ex) <= (200 / 32 + 8) * U * nrm)


# one shape for each form of the kernel: 64 x 64, 128 x 64, 128 x 128 tiles, and 256 x 256 by a pair of CTAs
FORMS = {"64x64": (60, 50, 140, 3), "128x64": (120, 150, 140, 2), "128x128": (125, 127, 256, 140), "pair": (250, 255, 1000, 70)}


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("ta,tb,pad", [(0, 0, 1), (0, 1, 0), (1, 0, 4), (1, 1, 3)])
@pytest.mark.parametrize("beta", [0.0, 0.25])
def test_out_of_range_in_every_form(S, form, ta, tb, pad, beta):
    """Inf, NaN, huge operands and sums that overflow on the scaled accumulators, in the first and the last rows and
    columns of a tile and in between: what an FFMA kernel gives, and the rest within the FP32 bound. C is read once,
    and nothing past the matrices is written."""
    m, n, k, batch = FORMS[form]
    p = problem(ta, tb, m, n, k, batch, beta, (pad, pad, pad), 7 + m)
    last = batch - 1
    for b in (0, last):
        opa, opb = p.op_a(b), p.op_b(b)
        opa[1, 3] = np.inf
        opa[m - 1, k - 1] = -np.inf
        opa[m // 2, :] *= np.float32(2.0 ** 90)          # sums beyond 2^80, finite
        opb[k // 2, n - 1] = np.nan
        if b == last:
            opa[40, :] *= np.float32(2.0 ** 105)         # operands beyond 2^104
            opb[5, n // 2] = np.inf
            opa[17, 5] = 0.0                             # Inf * 0
    C = run(S, p)
    S.set_kernel_config("simt", 3)
    try:
        R = run(S, p)
    finally:
        S.set_kernel_config("simt", -1)
    for b in sorted({0, 1, last}):
        got, ref = p.c_view(C, b).astype(np.float64), p.c_view(R, b).astype(np.float64)
        np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
        ok = np.isfinite(ref)
        np.testing.assert_array_equal(got[~ok & ~np.isnan(ref)], ref[~ok & ~np.isnan(ref)])
        A, B = (np.where(np.isfinite(x), x, 0.0).astype(np.float64) for x in (p.op_a(b), p.op_b(b)))
        C0 = beta * p.c_view(p.C, b).astype(np.float64)
        ex, nrm = 0.75 * (A @ B) + C0, 0.75 * (np.abs(A) @ np.abs(B)) + np.abs(C0)
        assert np.all(np.abs(got - ex)[ok] <= (4 * k * U * nrm)[ok])
    np.testing.assert_array_equal(C.reshape(batch, n, -1)[:, :, m:], p.C.reshape(batch, n, -1)[:, :, m:])


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("ea,eb", [(-50, -52), (-60, -64), (-66, -70), (-72, -76), (30, -135), (100, -140)])
def test_small_results(S, form, ea, eb):
    """Results down to FP32's smallest subnormal, and subnormal operands, on the tensor cores: the plain bound, and
    two roundings to FP32's subnormals (half of 2^-149 each) for the sum and for alpha."""
    m, n, k, batch = FORMS[form]
    p = problem(0, 0, m, n, k, batch, 0.0, (0, 0, 0), 3 + m)
    p.A *= np.float32(2.0) ** np.float32(ea)
    p.B[:] = np.ldexp(p.B.astype(np.float64), eb).astype(np.float32)
    C = run(S, p)
    assert S.last_run_info()["path"] == "f32_tcgen05"
    for b in (0, batch - 1):
        ex, nrm = O.exact_f64(p, b)
        err = np.abs(p.c_view(C, b).astype(np.float64) - ex)
        assert np.all(err <= (k / 32 + 8) * U * nrm + 2.0 ** -149)


@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 1)])
def test_more_tiles_than_one_launch_holds(S, ta, tb):
    """A launch holds 4096 tiles per worker; the tiles of the next launch go on where it ended, also those that
    are computed again."""
    m, n, k, batch = 1, 1, 128, 4096 * 148 + 300
    import torch
    g = torch.Generator(device="cuda").manual_seed(5)
    A, B = (torch.rand((batch, k), generator=g, device="cuda") * 2 - 1 for _ in range(2))
    bad = [0, 147, 148, 4096 * 148 - 1, 4096 * 148, batch - 1]
    A[bad, 5] = 1e30
    C = torch.full((batch,), float("nan"), device="cuda")
    ptrs = [t.data_ptr() + torch.arange(batch, device="cuda") * (4 * s) for t, s in ((A, k), (B, k), (C, 1))]
    al, be = np.array([1.0], np.float32), np.array([0.0], np.float32)
    st = S.lib().ssblasGemmBatchedEx(ta, tb, m, n, k, al.ctypes.data, ptrs[0].data_ptr(), S.SSBLAS_R_32F, k if ta else 1,
                                     ptrs[1].data_ptr(), S.SSBLAS_R_32F, 1 if tb else k, be.ctypes.data,
                                     ptrs[2].data_ptr(), S.SSBLAS_R_32F, 1, batch, 0, 0)
    info = S.last_run_info()
    assert st == 0 and info["path"] == "f32_tcgen05" and info["kernel_launches"] == 2
    ex, nrm = (A.double() * B.double()).sum(1), (A.double() * B.double()).abs().sum(1)
    err = (C.double() - ex).abs()
    plain = torch.ones(batch, dtype=torch.bool, device="cuda")
    plain[bad] = False
    assert bool((err <= (k / 32 + 8) * U * nrm)[plain].all())
    assert bool((err <= 4 * k * U * nrm)[~plain].all())


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 1)])
def test_results_of_one_product(S, form, ta, tb):
    """One nonzero per row of op(A): each result is one product. Its error, in u of the product: the sum of hi hi and
    the smaller products is rounded once (1 u), mid lo and lo mid are left out (|mid| <= 2^-8 and |lo| <= 2^-17 of an
    operand: 1 u), and the smaller products, at most 2^-7 (1 + 2^-8) of the product, are truncated five times (2 u
    each at their magnitude: 0.08 u); alpha = 1 and beta = 0 round nothing: 2.1 u."""
    m, n, k, batch = FORMS[form]
    p = problem(ta, tb, m, n, k, batch, 0.0, (0, 0, 0), 21 + m)
    p = dataclasses.replace(p, alpha=np.float32(1.0))
    rng = np.random.default_rng(m)
    for b in range(batch):
        opa = p.op_a(b)
        keep = rng.integers(0, k, m)
        row = opa[np.arange(m), keep].copy()
        opa[:] = 0.0
        opa[np.arange(m), keep] = row
    C = run(S, p)
    assert S.last_run_info()["path"] == "f32_tcgen05"
    for b in range(0, batch, max(1, batch // 8)):
        ex, nrm = O.exact_f64(p, b)
        err = np.abs(p.c_view(C, b).astype(np.float64) - ex)
        assert np.all(err <= 2.1 * U * nrm)


def test_compute_type_keeps_ffma(S):
    """SSBLAS_COMPUTE_32F, honoured under its extension, keeps plain fp32 off the tensor cores at any k."""
    import torch
    m, n, k = 70, 50, 300
    g = torch.Generator(device="cuda").manual_seed(2)
    A, B = (torch.rand(s, generator=g, device="cuda") * 2 - 1 for s in ((k, m), (n, k)))
    C = torch.zeros((n, m), device="cuda")
    ptrs = [(ct.c_void_p * 1)(t.data_ptr()) for t in (A, B, C)]
    one, zero = np.array([1.0], np.float32), np.array([0.0], np.float32)
    assert S.set_extensions(S.SSBLAS_EXT_COMPUTE_TYPE) == 0
    try:
        st = S.lib().ssblasGemmBatchedEx(0, 0, m, n, k, one.ctypes.data, ptrs[0], S.SSBLAS_R_32F, m, ptrs[1], S.SSBLAS_R_32F,
                                         k, zero.ctypes.data, ptrs[2], S.SSBLAS_R_32F, m, 1, S.SSBLAS_COMPUTE_32F, 0)
        assert st == 0 and S.last_run_info()["path"] == "simt"
    finally:
        S.set_extensions(S.SSBLAS_EXT_NONE)
    ex = B.double() @ A.double()
    nrm = B.double().abs() @ A.double().abs()
    assert bool(((C.double() - ex).abs() <= k * U * nrm).all())


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("shape", [(64, 64, 700, 1), (70, 33, 513, 3), (300, 200, 544, 2), (129, 257, 1000, 1)])
@pytest.mark.parametrize("pad,beta", [(0, 0.25), (4, 0.0), (3, -1.5)])
def test_bf16x3_planes_and_split_kernel_agree(S, ta, tb, shape, pad, beta):
    """The split pass with the tiled GEMM (either tile width) and the split kernel: the same bits, so the choice between
    them may follow the number of tiles."""
    m, n, k, batch = shape
    p = problem(ta, tb, m, n, k, batch, beta, (pad, pad, pad), 13 + m, "outliers")
    S.set_math_mode(S.SSBLAS_MATH_FP32_BF16X3)
    out = []
    try:
        # (by default instances of at most 128 x 128 may take a kernel of their own, with another order of sums)
        for cfg in (3, 0, 1) if max(m, n) <= 128 else (3, 0, 1, -1):
            S.set_kernel_config("bf16x3_tcgen05", cfg)
            out.append(run(S, p, pad % 2).view(np.uint32))
    finally:
        S.set_kernel_config("bf16x3_tcgen05", -1)
        S.set_math_mode(S.SSBLAS_MATH_PLAIN)
    for o in out[1:]:
        np.testing.assert_array_equal(o, out[0])


def test_bf16x3_without_memory_for_planes(S):
    """A call that would take the planes runs on the split kernel where their scratch cannot be had; an injected failure
    of the allocation is reported."""
    import torch
    from ssblasex_b200 import runner
    p = problem(0, 1, 1536, 1024, 4096, 1, 0.0, (3, 3, 3), 4)      # 31 MB for each plane pair and more
    dp = runner.DeviceProblem(p)
    S.set_math_mode(S.SSBLAS_MATH_FP32_BF16X3)
    S.release_workspace()
    torch.cuda.empty_cache()
    try:
        st, want = runner.call(p, "host_array", dp)
        assert st == 0 and S.last_run_info()["kernel_launches"] == 2
        S.release_workspace()
        dp.reset_c()
        hold = torch.empty(torch.cuda.mem_get_info()[0] - (24 << 20), dtype=torch.uint8, device="cuda")
        st, got = runner.call(p, "host_array", dp)
        launches = S.last_run_info()["kernel_launches"]
        del hold
        torch.cuda.empty_cache()
        assert st == 0 and launches == 1
        np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
        S.release_workspace()
        assert S.set_fault_injection(S.SSBLAS_FAULT_ALLOC) == 0
        assert runner.call(p, "host_array", dp)[0] == S.SSBLAS_STATUS_ALLOC_FAILED
    finally:
        S.set_math_mode(S.SSBLAS_MATH_PLAIN)
        S.release_workspace()
