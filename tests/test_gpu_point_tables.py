"""Claims, evaluations and eq combinations whose kernels form their own eq
tables: the block shapes (2^12 words a block from 12 variables on), fewer
variables than a block, and both sides of the line to the table kernels.
Exact against the oracle; coordinates 0, 1 and p - 1 are among the points.
"""
import numpy as np
import pytest

import whir_gb300 as W

pytestmark = pytest.mark.gpu

ONE = 0x01FFFFFE  # Montgomery form of 1


def _point(oracle, seed, k):
    p = oracle.rand_fe(seed, 4 * k)
    if k > 2:
        p[0:4] = 0
        p[4:8] = (ONE, 0, 0, 0)
        p[8:12] = W.P - 1
    return p


@pytest.mark.parametrize("kept", range(0, 9))
@pytest.mark.parametrize("k", [8, 11, 12, 13, 17])
def test_compress_hi(ctx, oracle, k, kept):
    poly, point = oracle.rand_fe(k, 1 << k), _point(oracle, 20 + k + kept, k - kept)
    poly[:16] = W.P - 1
    got = W.compress_hi(ctx, ctx.to_device(poly), k, point, k - kept)
    assert np.array_equal(got, oracle.compress_hi(poly, k, point, k - kept))


@pytest.mark.parametrize("k", [0, 1, 2, 7, 8, 9, 12, 18, 19])
def test_eval_ext(ctx, oracle, k):
    poly, point = oracle.rand_fe(60 + k, 4 << k), _point(oracle, 61 + k, k)
    got = W.eval_ext(ctx, ctx.to_device(poly), k, point)
    assert np.array_equal(got, oracle.eval_ext(poly, k, point))


@pytest.mark.parametrize("k,n", [(0, 1), (1, 9), (3, 8), (4, 2), (7, 8), (8, 17), (9, 1), (11, 3),
                                 (15, 8), (15, 9), (16, 4), (16, 5), (18, 1), (18, 2)])
def test_combine_eqs(ctx, oracle, k, n):
    w, alpha = oracle.rand_fe(80 + k, 4 << k), oracle.rand_fe(81, 4)
    points = np.concatenate([_point(oracle, 90 + t, k) for t in range(n)]) if k else \
        np.zeros(0, np.uint32)
    dev = ctx.to_device(w)
    W.combine_eqs(ctx, dev, k, points, n, alpha)
    assert np.array_equal(dev.download(4 << k), oracle.combine_eqs(w, k, points, n, alpha))


def test_combine_eqs_refuses_before_writing(ctx, oracle):
    w = oracle.rand_fe(5, 4 << 5)
    points = oracle.rand_fe(6, 4 * 5 * 12)
    points[-1] = W.P
    dev = ctx.to_device(w)
    with pytest.raises(W.WhirError):
        W.combine_eqs(ctx, dev, 5, points, 12, oracle.rand_fe(7, 4))
    assert np.array_equal(dev.download(4 << 5), w)
