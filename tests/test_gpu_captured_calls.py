"""Calls in a CUDA graph: what the graph reads stays in place whatever calls come between capture and replay."""
import ctypes as ct

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture
def S():
    import torch
    assert torch.cuda.is_available()
    import ssblasex_b200 as S
    S.release_workspace()
    yield S
    torch.cuda.synchronize()
    S.set_stream(None)
    S.set_sync_mode(True)
    S.set_math_mode(S.SSBLAS_MATH_PLAIN)
    S.release_workspace()


def problems(shapes, seed, count=12):
    from ssblasex_b200 import workloads as W
    rng = np.random.default_rng(shapes)
    return [W.make_problem(("f64", "f32", "i8")[i % 3], i % 2, i // 2 % 2, *(int(x) for x in rng.integers(1, 150, 3)), 1,
                           1, 0, seed=100 * seed + i) for i in range(count)]


def check(probs, results):
    for p, C in zip(probs, results):
        if p.row == "i8":
            np.testing.assert_array_equal(C, O.restated_gemm(p)[1])
        elif p.row == "f64":
            np.testing.assert_array_equal(C.view(np.uint64), O.ozaki_f64(p, 7)[1].view(np.uint64))
        else:
            assert O.normalized_error(p, C) <= 2.0 ** -14


@pytest.mark.parametrize("device_arrays", [True, False])
@pytest.mark.parametrize("mode", ["emulated", "plain"])
def test_grouped_replay_after_other_shapes(S, device_arrays, mode):
    import torch
    from ssblasex_b200 import runner
    emulated = mode == "emulated"
    S.set_math_mode(3 if emulated else 0)
    d = runner.GroupedDevice(problems(1, 1))
    others = [(p, runner.GroupedDevice(p)) for p in [problems(1, 50)] + [problems(2 + i, 60 + i) for i in range(7)]]
    assert d.call(device_arrays=device_arrays) == 0
    s = torch.cuda.Stream()
    S.set_sync_mode(False)
    S.set_stream(s.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        with torch.cuda.graph(graph, stream=s):
            assert d.call(device_arrays=device_arrays) == 0
            assert d.call(device_arrays=device_arrays) == 0
    S.set_sync_mode(True)
    # more shapes than plans are kept, the graph's among them
    for _ in range(2):
        for p, o in others:
            o.reset_c()
            assert o.call(device_arrays=device_arrays) == 0
            if emulated:
                check(p, o.results())
    # other matrices in the graph's buffers
    fresh = problems(1, 2)
    for q, (a, b, c) in zip(fresh, d.tensors):
        a.copy_(torch.from_numpy(q.A[0]))
        b.copy_(torch.from_numpy(q.B[0]))
        c.zero_()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        graph.replay()
    s.synchronize()
    got = d.results()
    if emulated:
        check(fresh, got)
    else:
        for q, C in zip(fresh, got):
            if q.row == "i8":
                np.testing.assert_array_equal(C, O.restated_gemm(q)[1])
            else:
                assert O.normalized_error(q, C) <= 4 * q.k * (2.0 ** -53 if q.row == "f64" else 2.0 ** -24)


@pytest.mark.parametrize("warm", [True, False])
def test_batched_host_arrays_replay_after_other_calls(S, warm):
    """Host arrays of device pointers: uploaded before the capture goes on, and not rewritten."""
    import torch
    from ssblasex_b200 import runner, workloads as W
    mk = lambda i: W.make_problem("f64", 0, 1, 40 + i, 50, 60, 3 + i, 1.0, 0.0, seed=i)
    p = mk(0)
    dp = runner.DeviceProblem(p)
    keep = []

    def call(q, dq):
        arr = dq.host_arrays()
        al, be = np.array([q.alpha], np.float64), np.array([q.beta], np.float64)
        keep.append((arr, al, be))
        t = q.types
        return S.lib().ssblasGemmBatchedEx(q.transa, q.transb, q.m, q.n, q.k, al.ctypes.data, arr[0], t[0], q.lda, arr[1],
                                           t[1], q.ldb, be.ctypes.data, arr[2], t[2], q.ldc, q.batch, 0, 0)

    if warm:
        assert call(p, dp) == 0
    s = torch.cuda.Stream()
    S.set_sync_mode(False)
    S.set_stream(s.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        with torch.cuda.graph(graph, stream=s):
            assert call(p, dp) == 0
    for i in range(1, 14):      # more layouts than are kept, and than upload slots
        q = mk(i)
        dq = runner.DeviceProblem(q)
        assert call(q, dq) == 0
        s.synchronize()
        assert O.normalized_error(q, dq.C.cpu().numpy().reshape(q.C.shape)) <= 4 * q.k * 2.0 ** -53
    dp.C.zero_()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        graph.replay()
    s.synchronize()
    assert O.normalized_error(p, dp.C.cpu().numpy().reshape(p.C.shape)) <= 4 * p.k * 2.0 ** -53


@pytest.mark.parametrize("row,mode", [("f64", "ozaki"), ("i8", "plain")])
def test_batched_replay_after_larger_calls(S, row, mode):
    """The scratch that a captured call reads is not freed when a larger call needs more."""
    import torch
    from ssblasex_b200 import runner, workloads as W
    if mode == "ozaki":
        S.set_math_mode(S.SSBLAS_MATH_FP64_OZAKI)
    mk = lambda m, batch, seed: W.make_problem(row, 0, 1, m, 50, 61, batch, 1, 0, lda=m + 3, seed=seed)
    want = lambda q: O.ozaki_f64(q, 7)[1] if row == "f64" else O.restated_gemm(q)[1]
    p, fresh = mk(40, 3, 1), mk(40, 3, 2)
    dp = runner.DeviceProblem(p)
    assert runner.call(p, "device_array", dp)[0] == 0      # (synchronous: equal spacing is found)
    s = torch.cuda.Stream()
    S.set_sync_mode(False)
    S.set_stream(s.cuda_stream)
    arrays = dp.host_arrays()
    al, be = np.array([p.alpha], p.scale_dtype), np.array([p.beta], p.scale_dtype)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        with torch.cuda.graph(graph, stream=s):
            assert S.lib().ssblasGemmBatchedEx(p.transa, p.transb, p.m, p.n, p.k, al.ctypes.data, arrays[0], p.types[0],
                                               p.lda, arrays[1], p.types[1], p.ldb, be.ctypes.data, arrays[2],
                                               p.types[2], p.ldc, p.batch, 0, 0) == 0
    S.set_sync_mode(True)
    for i in range(4):
        q = mk(200 + 100 * i, 8, 10 + i)
        st, C = runner.call(q, "host_array")
        assert st == 0
        np.testing.assert_array_equal(C.reshape(-1), want(q).reshape(-1))
    dp.A.copy_(torch.from_numpy(fresh.A))
    dp.B.copy_(torch.from_numpy(fresh.B))
    dp.C.copy_(torch.from_numpy(fresh.C))
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        graph.replay()
    s.synchronize()
    np.testing.assert_array_equal(dp.C.cpu().numpy().reshape(-1), want(fresh).reshape(-1))
