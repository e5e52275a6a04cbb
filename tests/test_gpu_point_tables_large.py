"""Claims and evaluations over large polynomials whose kernels form their own eq tables: the
longest blocks of few kept variables, and more blocks per CTA than its prologue
forms high entries at once.  Exact against the oracle.
"""
import numpy as np
import pytest

import whir_gb300 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,kept", [(19, 0), (19, 1), (20, 0), (20, 1), (21, 0), (25, 0), (27, 4)])
def test_compress_hi(ctx, oracle, k, kept):
    poly, point = oracle.rand_fe(k, 1 << k), oracle.rand_fe(20 + k, 4 * (k - kept))
    poly[:4096] = W.P - 1
    got = W.compress_hi(ctx, ctx.to_device(poly), k, point, k - kept)
    assert np.array_equal(got, oracle.compress_hi(poly, k, point, k - kept))


def test_eval_ext(ctx, oracle):
    k = 24
    poly, point = oracle.rand_fe(60 + k, 4 << k), oracle.rand_fe(61 + k, 4 * k)
    got = W.eval_ext(ctx, ctx.to_device(poly), k, point)
    assert np.array_equal(got, oracle.eval_ext(poly, k, point))
