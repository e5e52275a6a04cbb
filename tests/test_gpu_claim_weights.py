"""Weights written by the first claims instead of added to a cleared array:
claims by value and through tables (2^18 entries times points is the line),
none at all, stacked layouts whose claims cover parts only or parts and the
whole (out-of-domain points), and one query's worth of fold_with_code
arguments.  Proofs equal the oracle's.
"""
import numpy as np
import pytest

import whir_gb300 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("params,ks,groups", [
    ((12, 4, 1, 1, 1, 100), [12], [[0]]),
    ((18, 2, 1, 1, 1, 64), [18], [[0]] * 5),          # 2^16 entries, tables
    ((18, 2, 1, 1, 1, 64), [18], [[0]]),
    ((10, 3, 1, 1, 0, 32), [8, 6, 6, 8, 5], [[0, 3], [1, 2], [4]]),  # unique decoding: parts only
    ((10, 3, 1, 1, 2, 32), [8, 6, 6, 8, 5], [[0, 3], [1, 2], [4]]),  # and the whole
    ((10, 3, 2, 1, 1, 32), [10], []),                   # no claims
    ((8, 4, 3, 1, 2, 3), [8], [[0]]),                   # a query or none
])
def test_proofs(ctx, oracle, params, ks, groups):
    polys = [oracle.rand_fe(5 + i, 1 << k) for i, k in enumerate(ks)]
    want = oracle.prove(params, polys, ks, groups)
    for _ in range(2):  # the second over the first one's arrays
        assert W.prove_harness(ctx, params, polys, ks, groups) == want
    if len(ks) == 1:
        got = W.prove_batch(ctx, params, [polys[0]] * 3, claims=len(groups))
        assert got == [want] * 3
