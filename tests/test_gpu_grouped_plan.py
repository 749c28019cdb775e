"""Grouped calls that share a plan: the same shapes on other matrices, other scalars or shapes between
them, other streams, and more shapes than plans are kept."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S():
    import torch
    assert torch.cuda.is_available()
    import ssblasex_b200 as S
    S.set_sync_mode(True)
    yield S
    S.set_math_mode(S.SSBLAS_MATH_PLAIN)
    S.set_sync_mode(True)
    S.set_stream(None)


def problems(seed, count=12, alpha=1.0, beta=0.0, shift=0):
    from ssblasex_b200 import workloads as W
    rng = np.random.default_rng(3 + shift)   # shapes from `shift` alone
    out = []
    for i in range(count):
        m, n, k = (int(x) for x in rng.integers(1, 200, 3))
        out.append(W.make_problem(("f64", "f32", "i8")[i % 3], i % 2, (i // 2) % 2, m, n, k, 1,
                                  2 if i % 3 == 2 else alpha, 1 if i % 3 == 2 else beta, seed=seed * 1000 + i))
    return out


def check(probs, results, mode):
    for p, C in zip(probs, results):
        if p.row == "i8":
            np.testing.assert_array_equal(C, O.restated_gemm(p)[1])
        elif p.row == "f64" and mode:
            np.testing.assert_array_equal(C.view(np.uint64), O.ozaki_f64(p, 7)[1].view(np.uint64))
        else:
            u = 2.0 ** -53 if p.row == "f64" else 2.0 ** -24
            # the 3xBF16 mode states 2^-14
            assert O.normalized_error(p, C) <= (2.0 ** -14 if mode and p.row == "f32" else 4 * p.k * u), p.name


@pytest.mark.parametrize("mode", [0, 3])
@pytest.mark.parametrize("device_arrays", [True, False])
def test_same_shapes_on_other_matrices(S, mode, device_arrays):
    from ssblasex_b200 import runner
    S.release_workspace()
    S.set_math_mode(mode)
    sets = [problems(1), problems(2), problems(3, alpha=0.5, beta=-1.0), problems(4, shift=1)]
    dev = [runner.GroupedDevice(p) for p in sets]
    for i in (0, 1, 2, 3, 1, 0, 3, 2):
        dev[i].reset_c()
        assert dev[i].call(device_arrays=device_arrays) == 0
        check(sets[i], dev[i].results(), mode)


def test_more_shapes_than_plans(S):
    from ssblasex_b200 import runner
    S.set_math_mode(3)
    sets = [problems(10 + i, count=3, shift=10 + i) for i in range(7)]
    dev = [runner.GroupedDevice(p) for p in sets]
    for _ in range(2):
        for p, d in zip(sets, dev):
            d.reset_c()
            assert d.call() == 0
            check(p, d.results(), 3)


def test_one_plan_on_two_streams(S):
    """Asynchronous calls of one plan on alternating streams share its packed buffers: ordered by the
    library."""
    import torch
    from ssblasex_b200 import runner
    S.set_math_mode(3)
    sets = [problems(20, count=60), problems(21, count=60)]
    dev = [runner.GroupedDevice(p) for p in sets]
    for d in dev:
        d.reset_c()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    S.set_sync_mode(False)
    try:
        for _ in range(20):
            for d, s in zip(dev, streams):
                S.set_stream(s.cuda_stream)
                assert d.call() == 0
        torch.cuda.synchronize()
    finally:
        S.set_sync_mode(True)
        S.set_stream(None)
    # int8 instances accumulate (beta = 1); the others are recomputed by every call
    for p, d in zip(sets, dev):
        keep = [i for i, q in enumerate(p) if q.row != "i8"]
        res = d.results()
        check([p[i] for i in keep], [res[i] for i in keep], 3)


def test_arguments_are_checked_beside_a_plan(S):
    from ssblasex_b200 import runner
    S.set_math_mode(0)
    d = runner.GroupedDevice(problems(30))
    assert d.call() == 0
    ld = d.lda[0]
    d.lda[0] = 0
    assert d.call() == S.SSBLAS_STATUS_INVALID_VALUE
    d.lda[0] = ld
    d.m[1], m = 0, d.m[1]
    assert d.call() == S.SSBLAS_STATUS_INTERNAL_ERROR
    d.m[1] = m
    d.alpha[2], al = None, d.alpha[2]
    assert d.call() == S.SSBLAS_STATUS_INVALID_VALUE
    d.alpha[2] = al
    assert d.call() == 0
