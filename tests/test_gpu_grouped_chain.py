"""A plain grouped call's launches run into each other: work that follows on the stream sees all of their
results, also when the call is captured into a CUDA graph, with tiles of very different lengths in each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problems():
    from ssblasex_b200 import workloads as W
    rng = np.random.default_rng(17)
    out = []
    for i in range(400):
        m, n = (int(x) for x in rng.integers(1, 130, 2))
        # the first layout of each kind has the longest tiles
        lay = i % 4
        k = 2000 if lay == 0 and i < 8 else int(rng.integers(1, 90))
        out.append(W.make_problem("f64" if i // 4 % 2 else "f32", lay % 2, lay // 2, m, n, k, 1, 1.0, 0.0, seed=i))
    return out


@pytest.mark.parametrize("captured", [False, True])
def test_following_work_sees_every_launch(captured):
    import torch
    import ssblasex_b200 as S
    from ssblasex_b200 import runner
    S.set_math_mode(S.SSBLAS_MATH_PLAIN)
    S.set_sync_mode(True)
    d = runner.GroupedDevice(_problems())
    assert d.call() == 0
    want = [c.clone() for _, _, c in d.tensors]
    s = torch.cuda.Stream()
    S.set_sync_mode(False)
    S.set_stream(s.cuda_stream)
    try:
        with torch.cuda.stream(s):
            got = [torch.empty_like(c) for c in want]

            def step():
                for _, _, c in d.tensors:
                    c.fill_(float("nan"))
                assert d.call() == 0
                for g, (_, _, c) in zip(got, d.tensors):
                    g.copy_(c)

            step()
            s.synchronize()
            if captured:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=s):
                    step()
                step = graph.replay
            for _ in range(5):
                for g in got:
                    g.zero_()
                step()
                assert all(torch.equal(a, b) for a, b in zip(got, want))
            s.synchronize()
    finally:
        torch.cuda.synchronize()
        S.set_stream(None)
        S.set_sync_mode(True)
