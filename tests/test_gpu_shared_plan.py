"""Grouped calls that share a plan's scratch, or a kept pointer array, where the streams' handles do not tell
the streams apart."""
import threading

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
PER_THREAD = 2   # cudaStreamPerThread: one handle, a stream per host thread


@pytest.fixture
def S():
    import torch
    assert torch.cuda.is_available()
    import ssblasex_b200 as S
    yield S
    torch.cuda.synchronize()
    S.set_stream(None)
    S.set_sync_mode(True)
    S.set_math_mode(S.SSBLAS_MATH_PLAIN)


def problems(seed, count=40, row="f64"):
    from ssblasex_b200 import workloads as W
    rng = np.random.default_rng(5)
    return [W.make_problem(row, i % 2, i // 2 % 2, *(int(x) for x in rng.integers(1, 200, 3)), 1, 1.0, 0.0,
                           seed=1000 * seed + i) for i in range(count)]


@pytest.mark.parametrize("device_arrays", [True, False])
def test_two_threads_on_the_per_thread_stream(S, device_arrays):
    import torch
    from ssblasex_b200 import runner
    S.set_math_mode(S.SSBLAS_MATH_FP64_OZAKI)
    sets = [problems(1), problems(2)]
    dev = [runner.GroupedDevice(p) for p in sets]
    for d in dev:
        d.reset_c()
    torch.cuda.synchronize()
    S.set_sync_mode(False)
    S.set_stream(PER_THREAD)
    status = [[], []]

    def work(i):
        for _ in range(20):
            status[i].append(dev[i].call(device_arrays=device_arrays))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert status == [[0] * 20, [0] * 20]
    for p, d in zip(sets, dev):
        for q, C in zip(p, d.results()):
            np.testing.assert_array_equal(C.view(np.uint64), O.ozaki_f64(q, 7)[1].view(np.uint64))


@pytest.mark.parametrize("same_shapes", [True, False])
def test_host_arrays_on_two_streams(S, same_shapes):
    """Asynchronous calls with host arrays of device pointers: each call's kernels read its own pointers, also
    while another stream's call uploads others."""
    import torch
    from ssblasex_b200 import runner
    sets = [problems(3, 60, "f32"), problems(4, 60 if same_shapes else 50, "f32")]
    dev = [runner.GroupedDevice(p) for p in sets]
    for d in dev:
        d.reset_c()
    streams = [torch.cuda.Stream() for _ in dev]
    torch.cuda.synchronize()
    S.set_sync_mode(False)
    for _ in range(20):
        for d, s in zip(dev, streams):
            S.set_stream(s.cuda_stream)
            assert d.call(device_arrays=False) == 0
    torch.cuda.synchronize()
    for p, d in zip(sets, dev):
        for q, C in zip(p, d.results()):
            assert O.normalized_error(q, C) <= 4 * q.k * 2.0 ** -24


@pytest.mark.parametrize("row", ["f64", "i8"])
def test_batched_scratch_on_two_streams(S, row):
    """Asynchronous batched calls on two streams share the slices (fp64, Ozaki) or the aligned copies (int8)."""
    import torch
    from ssblasex_b200 import runner, workloads as W
    S.set_math_mode(S.SSBLAS_MATH_FP64_OZAKI)
    probs = [W.make_problem(row, 0, 1, 203, 190 - 50 * i, 301 + 70 * i, 6, 1, 0, lda=206, seed=i) for i in range(2)]
    dev = [runner.DeviceProblem(p) for p in probs]
    args = []
    for p, d in zip(probs, dev):
        a, t = d.host_arrays(), p.types
        al, be = np.array([p.alpha], p.scale_dtype), np.array([p.beta], p.scale_dtype)
        args.append((a, al, be, (p.transa, p.transb, p.m, p.n, p.k, al.ctypes.data, a[0], t[0], p.lda, a[1], t[1], p.ldb,
                                 be.ctypes.data, a[2], t[2], p.ldc, p.batch, 0, 0)))
    streams = [torch.cuda.Stream() for _ in dev]
    torch.cuda.synchronize()
    S.set_sync_mode(False)
    for _ in range(20):
        for a, s in zip(args, streams):
            S.set_stream(s.cuda_stream)
            assert S.lib().ssblasGemmBatchedEx(*a[3]) == 0
    torch.cuda.synchronize()
    for p, d in zip(probs, dev):
        want = O.restated_gemm(p)[1] if row == "i8" else O.ozaki_f64(p, 7)[1]
        np.testing.assert_array_equal(d.C.cpu().numpy().reshape(-1), want.reshape(-1))
