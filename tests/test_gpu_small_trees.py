"""Merkle trees of few rows: leaves hashed one row per warp up to 2^10 rows, on
four lanes up to 2^13,
and the narrow levels in one to three launches (one warp or a quad of lanes
per node).  Every height has its own split, so every level of every height up
to 13 equals the oracle's; row lengths cover empty, full and short last
chunks.
"""
import numpy as np
import pytest

import whir_gb300 as W

pytestmark = pytest.mark.gpu


def _check(ctx, oracle, log_h, row_len):
    rows = oracle.rand_fe(500 + 17 * log_h + row_len, row_len << log_h)
    rows[:row_len] = W.P - 1
    rows[row_len:2 * row_len] = 0
    t = W.MerkleTree(ctx, ctx.to_device(rows), log_h, row_len)
    assert np.array_equal(t.levels(), oracle.merkle_tree(rows, log_h, row_len))
    t.close()


@pytest.mark.parametrize("log_h", range(0, 15))
def test_heights(ctx, oracle, log_h):
    _check(ctx, oracle, log_h, 16)


@pytest.mark.parametrize("row_len", [1, 7, 15, 17, 31, 32, 33, 64, 129])
@pytest.mark.parametrize("log_h", [3, 10, 11, 13])
def test_row_lengths(ctx, oracle, log_h, row_len):
    _check(ctx, oracle, log_h, row_len)


@pytest.mark.parametrize("k,n", [(8, 1), (8, 6), (10, 33), (12, 9), (13, 20)])
def test_lockstep_trees(ctx, oracle, k, n):
    params = (k, 4, 2, 1, 1, 100)
    polys = [oracle.rand_fe(600 + i, 1 << k) for i in range(n)]
    got = W.prove_batch(ctx, params, polys, claims=1)
    for i in (0, n // 2, n - 1):
        assert got[i] == W.prove_harness(ctx, params, [polys[i]], [k], [[0]])
    assert got[0] == oracle.prove(params, [polys[0]], [k], [[0]])
