"""Pow-claim combination around the sizes where its kernels change hands.

Few outputs run with lanes over the points, in groups of 8 outputs shared by
8, 2 or 1 warps; larger arrays use power tables.  Points 0, 1 and p - 1 and
extreme scales bound the 64-bit sums.  Exact against the oracle.
"""
import numpy as np
import pytest

import whir_gb300 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n", [
    (0, 1), (1, 33), (2, 32), (3, 513), (9, 31), (10, 240), (10, 1025), (11, 1), (11, 257),
    (12, 100), (13, 1), (13, 97), (14, 31), (14, 32), (15, 31), (15, 129), (16, 5), (16, 40),
])
def test_combine_pows_edges(ctx, oracle, k, n):
    w = oracle.rand_fe(7 + k, 4 << k)
    vars_, scales = oracle.rand_fe(70 + n, n), oracle.rand_fe(71 + n, 4 * n)
    vars_[0], scales[:4] = 0, W.P - 1
    vars_[n // 2] = W.P - 1
    scales[4 * (n // 2):4 * (n // 2) + 4] = W.P - 1
    dev = ctx.to_device(w)
    W.combine_pows_scaled(ctx, dev, k, vars_, n, scales)
    assert np.array_equal(dev.download(4 << k), oracle.combine_pows_scaled(w, k, vars_, n, scales))


def test_lockstep_counts(ctx, oracle):
    # instances' query counts differ (deduplication); 2^8 and 2^4 outputs each
    params = (12, 4, 1, 1, 1, 100)
    polys = [oracle.rand_fe(300 + i, 1 << 12) for i in range(7)]
    got = W.prove_batch(ctx, params, polys, claims=1)
    for i, p in enumerate(polys):
        assert got[i] == W.prove_harness(ctx, params, [p], [12], [[0]])
