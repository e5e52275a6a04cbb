"""The column DFT on each side of its lines for few tiles: 4-column slices up to
76 tiles of 8 columns, and two passes up to 64 tiles of 2^12 rows.  Exact
against the oracle, whole and ragged heights.
"""
import numpy as np
import pytest

import whir_gb300 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_h,width,log_in", [
    (14, 72, 11), (14, 80, 11), (11, 608, 11), (11, 616, 11), (13, 152, 10), (13, 160, 10),
    (9, 16, 8), (12, 8, 7),
    (12, 16, 12), (13, 4, 12), (14, 64, 12), (14, 68, 12), (15, 32, 12), (15, 36, 12),
])
@pytest.mark.parametrize("short", [0, 5])
def test_lines(ctx, oracle, log_h, width, log_in, short):
    h_in = (1 << log_in) - short
    x = oracle.rand_fe(log_h + width, h_in * width)
    x[-width:] = W.P - 1
    got = W.dft_batch(ctx, ctx.to_device(x), h_in, width, log_h).download(width << log_h)
    assert np.array_equal(got, oracle.dft_batch(x, h_in, width, log_h))
