"""Batched dense LU at the sizes where its launch rules change (one thread per
system, then 32 to 512 threads per system, then the global work slice):
the same bits as the reference's LU at every one of them."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(16, 65), (17, 65), (22, 33), (23, 33), (32, 33), (33, 33), (40, 17), (41, 17),
                                     (64, 9), (65, 9), (88, 9), (89, 9), (166, 5)])
def test_bits_at_the_launch_rule_edges(ctx, n, batch):
    rng = np.random.default_rng(1000 + n)
    A = rng.standard_normal((batch, n, n))
    A[rng.random((batch, n, n)) < 0.3] = 0.0  # zero entries: multipliers and pivot candidates that are 0
    A[0] = np.round(A[0])                     # equal magnitudes
    A[1, :, n // 2] = A[1, :, n // 2 - 1]     # dependent columns: singular or nearly so
    b = rng.standard_normal((batch, n))
    b[2] = 0.0
    mats = np.ascontiguousarray(A.transpose(0, 2, 1)).ravel()
    res = ctx.solve_batch(mats, b.ravel(), n, batch)
    sol, sing = oracle.solve_batch(mats, b.ravel(), n, batch)
    assert res.singular_indices == [int(i) for i in np.nonzero(sing)[0]]
    g, w = np.asarray(res.solutions), np.asarray(sol).ravel()
    nan = np.isnan(w)
    assert np.array_equal(np.isnan(g), nan)
    assert np.array_equal(g[~nan].view(np.uint64), w[~nan].view(np.uint64))
