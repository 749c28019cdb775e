"""Performance cases of ssblasGemmBatchedEx and ssblasGemmGroupedBatchedEx.

Each case is one call as a program makes it: inputs and pointer arrays are in hand (prepare), one
pass is one call of the entry point (run). Matrices are column-major with any leading dimension;
an operand of a batch is one tensor (batch, stored columns, ld), instance b at a fixed stride.
"""
import ctypes as ct
import math

import numpy as np
import torch

import ssblasex_b200 as S

# row -> (type code of A and B, of C, operand dtype, C dtype, numpy scalar type of alpha / beta)
ROWS = {
    "f32": (S.SSBLAS_R_32F, S.SSBLAS_R_32F, torch.float32, torch.float32, np.float32),
    "f64": (S.SSBLAS_R_64F, S.SSBLAS_R_64F, torch.float64, torch.float64, np.float64),
    "i8": (S.SSBLAS_R_8I, S.SSBLAS_R_32I, torch.int8, torch.int32, np.int32),
}
MODES = {"plain": S.SSBLAS_MATH_PLAIN, "ozaki": S.SSBLAS_MATH_FP64_OZAKI, "bf16x3": S.SSBLAS_MATH_FP32_BF16X3,
         "emulated": S.SSBLAS_MATH_FP64_OZAKI | S.SSBLAS_MATH_FP32_BF16X3}


def batched(name, row, ta, tb, m, n, k, batch, alpha, beta, mode="plain", pad=0, dist="uniform", sync=False,
            where="device"):
    """pad: elements by which each leading dimension exceeds the stored rows; sync: the library's
    default synchronous mode (otherwise asynchronous on the current stream); where: "device" = host
    arrays of device pointers, "host" = host arrays of host pointers, one allocation per matrix."""
    return dict(name=name, entry="batched", row=row, ta=ta, tb=tb, m=m, n=n, k=k, batch=batch, alpha=alpha, beta=beta,
                mode=mode, pad=pad, dist=dist, sync=sync, where=where)


def listed():
    return [
        # the smallest call: a few small matrices, synchronous as a relinked program calls it
        batched("f32_8x32_sync", "f32", 0, 0, 32, 32, 32, 8, 1.0, 0.0, sync=True),
        # per-head / per-element transforms: tens of 128^3 products in fp32
        batched("f32_64x128_nn", "f32", 0, 0, 128, 128, 128, 64, 1.0, 0.5),
        # thousands of small fp32 matrices, both transposed, entries with outliers
        batched("f32_4096x64_tt", "f32", 1, 1, 64, 64, 64, 4096, 0.75, 0.25, dist="outliers"),
        # fp32 matrices of ordinary size
        batched("f32_16x1024_nn", "f32", 0, 0, 1024, 1024, 1024, 16, 1.0, 0.0),
        # the fp32 emulation mode on mid-sized matrices
        batched("f32_bf16x3_256x256_nt", "f32", 0, 1, 256, 256, 256, 256, 1.0, 0.0, mode="bf16x3"),
        # quantised inference: int8 products accumulated into int32
        batched("i8_512x512_tn", "i8", 1, 0, 512, 512, 512, 512, 1, 1),
        # int8 matrices whose sizes and leading dimensions come from the data, not from the hardware
        batched("i8_64x501_nn_odd", "i8", 0, 0, 501, 517, 509, 64, 1, 0, pad=2),
        # fp64 of uneven shape (the library's plain double precision)
        batched("f64_64x500_tn", "f64", 1, 0, 500, 300, 700, 64, 1.0, 1.0, pad=4),
        # the headline workload: fp64 emulation on large matrices with spread exponents
        batched("f64_ozaki_32x1024_nt", "f64", 0, 1, 1024, 1024, 1024, 32, 1.0, 0.0, mode="ozaki", pad=8,
                dist="expspread"),
        # a program written for the reference library: host matrices, each its own allocation
        batched("f64_host_16x512_nn", "f64", 0, 0, 512, 512, 512, 16, 1.0, 0.0, sync=True, where="host"),
        # thousands of uneven products in one grouped call, emulation on
        dict(name="grouped_10000_emulated", entry="grouped", mode="emulated", count=10000, lo=8, hi=512, sizes=5),
        # the same kind of call, smaller, in the default math mode
        dict(name="grouped_2000_plain", entry="grouped", mode="plain", count=2000, lo=8, hi=512, sizes=7),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["f32", "f32", "f32", "bf16x3", "i8", "i8", "f64", "f64", "ozaki", "ozaki", "host", "grouped"])
    if kind == "grouped":
        return dict(entry="grouped", mode=rng.choice(["plain", "emulated"]), count=_log_int(rng, 100, 6000), lo=8,
                    hi=rng.choice([128, 256, 512]), sizes=rng.randrange(1 << 20))
    row = {"f32": "f32", "bf16x3": "f32", "i8": "i8"}.get(kind, "f64")
    lo, hi = {"f32": (16, 1024), "bf16x3": (32, 1024), "i8": (32, 1024), "f64": (16, 1024), "ozaki": (64, 1024),
              "host": (64, 512)}[kind]
    m, n, k = (_log_int(rng, lo, hi) for _ in range(3))
    if rng.random() < 0.5:   # half of the shapes are multiples of 16
        m, n, k = ((x + 15) // 16 * 16 for x in (m, n, k))
    # operations of the call, and at most 4096 matrices (48 on the host)
    most = {"f32": 3e10, "bf16x3": 3e10, "i8": 1e11, "f64": 1e10, "ozaki": 5e10, "host": 4e9}[kind]
    ops = math.exp(rng.uniform(math.log(1e6), math.log(most)))
    batch = max(1, min(48 if kind == "host" else 4096, int(ops / (2.0 * m * n * k))))
    size = {"f32": 4, "i8": 1, "f64": 8}[row]
    batch = min(batch, max(1, int((6e7 if kind == "host" else 8e8) / (size * (m * k + k * n) + max(4, size) * m * n))))
    return dict(entry="batched", row=row, ta=rng.randrange(2), tb=rng.randrange(2), m=m, n=n, k=k, batch=batch,
                alpha=1 if row == "i8" else rng.choice([1.0, 0.75]),
                beta=rng.choice([0, 1]) if row == "i8" else rng.choice([0.0, 0.0, 0.25, 1.0]),
                mode={"bf16x3": "bf16x3", "ozaki": "ozaki"}.get(kind, "plain"), pad=rng.choice([0, 0, 3, 8]),
                dist={"ozaki": "expspread", "bf16x3": "uniform"}.get(kind, "uniform" if row != "f32" else
                                                                     rng.choice(["uniform", "outliers"])),
                sync=kind == "host" or rng.random() < 0.25, where="host" if kind == "host" else "device")


# ------------------------------------------------------------------------------- batched ------
def _stored(trans, rows, cols):
    return (cols, rows) if trans else (rows, cols)


def _fill(gen, shape, row, dist, is_c):
    """Random entries of a (batch, stored columns, stored rows) block on the generator's device."""
    dev = gen.device
    if row == "i8":
        lim = (1 << 20) if is_c else 128
        return torch.randint(-lim, lim, shape, generator=gen, device=dev, dtype=torch.int32 if is_c else torch.int8)
    dt = ROWS[row][2]
    x = torch.rand(shape, generator=gen, device=dev, dtype=dt) * 2 - 1
    if dist == "expspread":   # sign * U[1, 2) * 2^U{-8..8}
        x = x + torch.where(x < 0, -1.0, 1.0).to(dt)
        return torch.ldexp(x, torch.randint(-8, 9, shape, generator=gen, device=dev)).to(dt)
    if dist == "outliers":    # one entry in a hundred is 1e4 times larger
        return torch.where(torch.rand(shape, generator=gen, device=dev) < 0.01, x * 1e4, x)
    return x


def _operands(case, seed, device):
    """A, B, C as (batch, stored columns, ld) tensors; the padding rows are zero."""
    gen = torch.Generator(device=device).manual_seed(int(seed))
    m, n, k = case["m"], case["n"], case["k"]
    out = []
    for i, (r, c) in enumerate((_stored(case["ta"], m, k), _stored(case["tb"], k, n), (m, n))):
        x = torch.zeros((case["batch"], c, r + case["pad"]), dtype=ROWS[case["row"]][2 if i < 2 else 3], device=device)
        x[:, :, :r] = _fill(gen, (case["batch"], c, r), case["row"], case["dist"], i == 2)
        out.append(x)
    return out


def _prepare_batched(case, seed):
    host = case["where"] == "host"
    tensors = _operands(case, seed, "cpu" if host else "cuda")
    if host:
        # one allocation per matrix, in pageable memory
        keep = [[x[b].numpy().copy() for b in range(case["batch"])] for x in tensors]
        ptrs = [[a.ctypes.data for a in arrs] for arrs in keep]
        out = keep[2]
    else:
        keep = tensors
        ptrs = [[x.data_ptr() + b * x.stride(0) * x.element_size() for b in range(case["batch"])] for x in tensors]
        out = tensors[2]
    arrays = [(ct.c_void_p * case["batch"])(*p) for p in ptrs]
    ab, c, _, _, scale = ROWS[case["row"]]
    al, be = np.array([case["alpha"]], scale), np.array([case["beta"]], scale)
    lda, ldb, ldc = (x.shape[2] for x in tensors)
    args = (case["ta"], case["tb"], case["m"], case["n"], case["k"], al.ctypes.data, ct.addressof(arrays[0]), ab, lda,
            ct.addressof(arrays[1]), ab, ldb, be.ctypes.data, ct.addressof(arrays[2]), c, ldc, case["batch"])
    return dict(fn=S.ssblasGemmBatchedEx, args=args, out=out, host=host, m=case["m"], keep=(keep, arrays, al, be))


def _exact_batched(case, seed):
    if case["row"] == "i8":
        return None   # whole numbers are compared as they are
    A, B, C = _operands(case, seed, "cpu" if case["where"] == "host" else "cuda")
    m, k = case["m"], case["k"]
    r = []
    for b in range(case["batch"]):   # the stored columns x rows of op(A) op(B) are (op(A) op(B))^T
        At = A[b, :, :_stored(case["ta"], m, k)[0]].double()
        Bt = B[b, :, :_stored(case["tb"], k, case["n"])[0]].double()
        P = torch.matmul(Bt.T if case["tb"] else Bt, At.T if case["ta"] else At)
        r.append(case["alpha"] * P + case["beta"] * C[b, :, :m].double())
    return [x.numpy() for x in r] if case["where"] == "host" else torch.stack(r)


# ------------------------------------------------------------------------------- grouped ------
def _group_sizes(case):
    """(m, n, k) log-uniform in [lo, hi], transposes, leading dimensions rounded up to 8; the first
    half of the instances is fp64, the others fp32."""
    rng = np.random.default_rng(case["sizes"])
    cnt = case["count"]
    dims = np.floor(np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"] + 1), size=(cnt, 3)))).astype(np.int64)
    dims = np.clip(dims, case["lo"], case["hi"])
    tr = rng.integers(0, 2, size=(cnt, 2)).astype(np.int32)
    m, n, k = dims.T
    up = lambda v: (v + 7) // 8 * 8
    lda, ca = up(np.where(tr[:, 0] == 1, k, m)), np.where(tr[:, 0] == 1, m, k)
    ldb, cb = up(np.where(tr[:, 1] == 1, n, k)), np.where(tr[:, 1] == 1, k, n)
    return dims, tr, [(lda, ca), (ldb, cb), (up(m), n)], cnt // 2


def _group_operands(case, seed):
    """For each of A, B, C: the two flat buffers (fp64 instances, fp32 instances) and each
    instance's offset in its buffer."""
    dims, tr, shapes, half = _group_sizes(case)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    out = []
    for i, (ld, cols) in enumerate(shapes):
        size = ld * cols
        bufs, offs = [], np.zeros_like(size)
        for part, dt in ((slice(0, half), torch.float64), (slice(half, None), torch.float32)):
            offs[part] = np.cumsum(size[part]) - size[part]
            n = int(size[part].sum())
            bufs.append(torch.zeros(n, dtype=dt, device="cuda") if i == 2 else
                        torch.rand(n, generator=gen, dtype=dt, device="cuda") * 2 - 1)
        out.append((bufs, offs))
    return dims, tr, shapes, half, out


def _prepare_grouped(case, seed):
    dims, tr, shapes, half, ops = _group_operands(case, seed)
    cnt = case["count"]
    ptrs = []
    for bufs, offs in ops:
        p = np.empty(cnt, np.int64)
        p[:half] = bufs[0].data_ptr() + 8 * offs[:half]
        p[half:] = bufs[1].data_ptr() + 4 * offs[half:]
        ptrs.append(torch.from_numpy(p).cuda())
    types = np.where(np.arange(cnt) < half, S.SSBLAS_R_64F, S.SSBLAS_R_32F).astype(np.int32)
    m, n, k = (np.ascontiguousarray(dims[:, i]) for i in range(3))
    ta, tb = (np.ascontiguousarray(tr[:, i]) for i in range(2))
    lds = [np.ascontiguousarray(s[0]) for s in shapes]
    one = [np.array([1.0], t) for t in (np.float64, np.float32)]
    zero = [np.array([0.0], t) for t in (np.float64, np.float32)]
    al = np.array([one[0].ctypes.data if i < half else one[1].ctypes.data for i in range(cnt)], np.int64)
    be = np.array([zero[0].ctypes.data if i < half else zero[1].ctypes.data for i in range(cnt)], np.int64)
    gs = np.ones(cnt, np.int64)
    d = lambda a: a.ctypes.data
    args = (d(ta), d(tb), d(m), d(n), d(k), d(al), ptrs[0].data_ptr(), d(types), d(lds[0]), ptrs[1].data_ptr(),
            d(types), d(lds[1]), d(be), ptrs[2].data_ptr(), d(types), d(lds[2]), cnt, d(gs), 0, 0)
    return dict(fn=S.ssblasGemmGroupedBatchedEx, args=args, out=ops[2][0], host=False, m=None,
                keep=(ops, ptrs, types, m, n, k, ta, tb, lds, one, zero, al, be, gs))


def _exact_grouped(case, seed):
    dims, tr, shapes, half, ops = _group_operands(case, seed)
    out = [torch.zeros(b.numel(), dtype=torch.float64, device="cuda") for b in ops[2][0]]
    A64, B64 = ([b.double() for b in ops[i][0]] for i in range(2))

    def mat(bufs, offs, i, part, which, rows):   # stored columns x stored rows of instance i
        ld, cols = int(shapes[which][0][i]), int(shapes[which][1][i])
        return bufs[part][int(offs[i]):int(offs[i]) + ld * cols].view(cols, ld)[:, :rows]

    for i in range(case["count"]):
        part = 0 if i < half else 1
        m, n, k = (int(v) for v in dims[i])
        At = mat(A64, ops[0][1], i, part, 0, _stored(tr[i, 0], m, k)[0])
        Bt = mat(B64, ops[1][1], i, part, 1, _stored(tr[i, 1], k, n)[0])
        mat(out, ops[2][1], i, part, 2, m)[:] = torch.matmul(Bt.T if tr[i, 1] else Bt, At.T if tr[i, 0] else At)
    return out


# ------------------------------------------------------------------------------- interface ----
def prepare(case, seed):
    S.set_math_mode(MODES[case["mode"]])
    S.set_sync_mode(bool(case.get("sync", False)))
    S.set_stream(torch.cuda.current_stream().cuda_stream)
    return _prepare_grouped(case, seed) if case["entry"] == "grouped" else _prepare_batched(case, seed)


def run(state):
    status = state["fn"](*state["args"])
    if status != S.SSBLAS_STATUS_SUCCESS:
        raise RuntimeError(S.STATUS_NAMES.get(status, str(status)))
    out = state["out"]
    if state["host"]:
        return [c[:, :state["m"]] for c in out]
    return out if state["m"] is None else out[:, :, :state["m"]]


def exact(case, seed):
    return _exact_grouped(case, seed) if case["entry"] == "grouped" else _exact_batched(case, seed)


def work(case):
    if case["entry"] == "grouped":
        dims, _, _, half = _group_sizes(case)
        m, n, k = dims.T.astype(float)
        size = np.where(np.arange(case["count"]) < half, 8.0, 4.0)
        return {"bytes": float((size * (m * k + k * n + m * n)).sum()), "flops": float((2 * m * n * k).sum())}
    m, n, k = case["m"], case["n"], case["k"]
    ab, c = {"f32": (4, 4), "f64": (8, 8), "i8": (1, 4)}[case["row"]]
    per = ab * (m * k + k * n) + c * m * n * (2 if case["beta"] else 1)
    return {"bytes": float(per * case["batch"]), "flops": 2.0 * m * n * k * case["batch"]}
