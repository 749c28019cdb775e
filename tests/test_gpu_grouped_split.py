"""fp32 instances of a grouped call in the 3xBF16 mode: the edges of 128 x 128 tiles and 32-wide K chunks,
all operand orders, leading dimensions on and off the 16-byte grid, and more tiles than a CTA's records
hold at a time."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
BOUND = 2.0 ** -14   # what the 3xBF16 mode states, relative to |alpha| |A| |B| + |beta| |C|


def _run(probs):
    import ssblasex_b200 as S
    from ssblasex_b200 import runner
    S.set_sync_mode(True)
    S.set_math_mode(S.SSBLAS_MATH_FP32_BF16X3)
    try:
        d = runner.GroupedDevice(probs)
        assert d.call() == 0
        out = d.results()
    finally:
        S.set_math_mode(S.SSBLAS_MATH_PLAIN)
    for p, C in zip(probs, out):
        assert O.normalized_error(p, C) <= BOUND, p.name
        pad = np.ones(p.C[0].size, bool)
        for j in range(p.n):
            pad[j * p.ldc:j * p.ldc + p.m] = False
        np.testing.assert_array_equal(C[0].ravel()[pad], p.C[0].ravel()[pad])


@pytest.mark.parametrize("transa", [0, 1])
@pytest.mark.parametrize("transb", [0, 1])
@pytest.mark.parametrize("pad", [0, 1, 4])
def test_tile_edges(transa, transb, pad):
    from ssblasex_b200 import workloads as W
    sizes = [(1, 1, 1), (1, 128, 31), (127, 1, 32), (128, 128, 33), (129, 127, 64), (63, 65, 95), (257, 129, 97),
             (64, 300, 161), (5, 7, 300)]
    probs = []
    for i, (m, n, k) in enumerate(sizes):
        ar, br = (k if transa else m), (n if transb else k)
        probs.append(W.make_problem("f32", transa, transb, m, n, k, 1, (1.0, -0.5)[i % 2], (0.0, 0.75, 1.0)[i % 3],
                                    lda=ar + pad, ldb=br + pad, ldc=m + i % 4, seed=100 + i, name=f"{m}x{n}x{k}"))
    _run(probs)


@pytest.mark.parametrize("k", [3, 70])
def test_many_tiles_per_cta(k):
    """2560 + 8 tiles: more than sixteen per CTA, of very different lengths."""
    from ssblasex_b200 import workloads as W
    probs = [W.make_problem("f32", i % 2, (i // 2) % 2, 2048, 2048, k, 1, 1.0, 0.5, seed=i, name=f"big{i}") for i in range(10)]
    probs += [W.make_problem("f32", 0, 0, 20 + i, 30, 900, 1, 1.0, 0.0, seed=50 + i, name=f"long{i}") for i in range(8)]
    _run(probs)
