"""The column DFT at every sub-transform size of its vectorised tiles: radix 8
first and last with one to four stages between (2^6 and up), two steps (2^4,
2^5), packed and whole tiles of 4 and 8 columns, in the one-pass form, the
coset form with its pre-twiddles and the two passes with their post-twiddles.
Exact against the oracle; ragged heights, widths off the powers of two.
"""
import numpy as np
import pytest

import whir_gb300 as W

pytestmark = pytest.mark.gpu


def _check(ctx, oracle, log_h, width, h_in):
    x = oracle.rand_fe(log_h + width, h_in * width)
    x[:width] = W.P - 1
    got = W.dft_batch(ctx, ctx.to_device(x), h_in, width, log_h).download(width << log_h)
    assert np.array_equal(got, oracle.dft_batch(x, h_in, width, log_h))


@pytest.mark.parametrize("width", [4, 8, 20])
@pytest.mark.parametrize("log_h", range(3, 12))
def test_one_pass(ctx, oracle, log_h, width):
    _check(ctx, oracle, log_h, width, (1 << log_h) - 3)


@pytest.mark.parametrize("log_in", range(3, 13))
@pytest.mark.parametrize("width,extra", [(4, 1), (8, 3), (12, 2)])
def test_cosets(ctx, oracle, log_in, width, extra):
    _check(ctx, oracle, max(12, log_in + extra), width, (1 << log_in) - 1)


@pytest.mark.parametrize("log_h,width,h_in", [
    (13, 8, 8000), (14, 20, 5000), (15, 4, 1 << 15), (16, 8, 8192), (17, 12, 9001),
    (18, 8, 1 << 14), (19, 4, 1 << 16), (20, 16, 1 << 17), (21, 8, 1 << 20), (22, 4, 1 << 22),
    (23, 4, 1 << 22), (23, 8, 3 << 20), (24, 4, 1 << 21),
])
def test_two_passes(ctx, oracle, log_h, width, h_in):
    _check(ctx, oracle, log_h, width, h_in)
