"""DFT tiles on both sides of the line between the kernels of three and of four
CTAs per SM, for every number of stages; exact against the oracle."""
import numpy as np
import pytest

import whir_gb300 as W

pytestmark = pytest.mark.gpu


# coset tiles of 2^S rows: 32, 16 (S = 11) or 8 (S = 12, 4 columns) per column
# slice, so 448 CTAs and the next width
@pytest.mark.parametrize("stages,widths", [(s, (112, 120)) for s in range(4, 11)]
                         + [(11, (224, 232)), (12, (224, 228))])
def test_both_sides(ctx, oracle, stages, widths):
    for width in widths:
        h_in = (1 << stages) - 1
        x = oracle.rand_fe(stages, h_in * width)
        x[:width] = W.P - 1
        got = W.dft_batch(ctx, ctx.to_device(x), h_in, width, 15).download(width << 15)
        assert np.array_equal(got, oracle.dft_batch(x, h_in, width, 15)), width


@pytest.mark.parametrize("log_h", range(4, 12))
@pytest.mark.parametrize("width", [4, 8, 640])
def test_single_tiles(ctx, oracle, log_h, width):
    x = oracle.rand_fe(50 + log_h, width << log_h)
    got = W.dft_batch(ctx, ctx.to_device(x), 1 << log_h, width, log_h).download(width << log_h)
    assert np.array_equal(got, oracle.dft_batch(x, 1 << log_h, width, log_h))
