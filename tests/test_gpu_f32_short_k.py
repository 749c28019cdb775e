"""Plain fp32 with k <= 64 by the library's own choice of kernel: 64 x 64 tiles, or 32 x 32 where they cover
at most half the area. Both sides of that line, sizes around the tiles' edges, orders and alignments: the
same bits as configuration 3, which sums in the same order, and within 4 k u of the exact product."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(64, 64, 64), (65, 64, 1), (32, 32, 64), (33, 32, 63), (32, 64, 17), (1, 1, 1),
                                   (96, 96, 40), (97, 31, 33), (130, 140, 16), (4, 200, 50)])
@pytest.mark.parametrize("trans", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("pad,beta", [(0, 0.0), (1, 0.5)])
def test_short_k(m, n, k, trans, pad, beta):
    import ssblasex_b200 as S
    from ssblasex_b200 import runner, workloads as W
    ta, tb = trans
    S.set_math_mode(S.SSBLAS_MATH_PLAIN)
    S.set_sync_mode(True)
    p = W.make_problem("f32", ta, tb, m, n, k, 3, 0.75, beta, lda=(k if ta else m) + pad, ldb=(n if tb else k) + pad,
                       ldc=m + 2 * pad, seed=m + 7 * n + 13 * k)
    C0 = p.C.copy()
    if beta == 0.0:
        C0.reshape(3, n, -1)[:, :, :m] = np.nan   # not read
    st, C = runner.call(p, dp=runner.DeviceProblem(p, C=C0))
    assert st == 0 and S.last_run_info()["path"] == "simt"
    S.set_kernel_config("simt", 3)
    try:
        st, C3 = runner.call(p, dp=runner.DeviceProblem(p, C=C0))
    finally:
        S.set_kernel_config("simt", -1)
    assert st == 0
    np.testing.assert_array_equal(np.asarray(C).view(np.uint32), np.asarray(C3).view(np.uint32))
    assert O.normalized_error(p, C) <= 4 * k * 2.0 ** -24
