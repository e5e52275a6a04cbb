"""Merkle trees and path checks on both sides of the lines between the hash
kernels: leaves at 2^15 and 2^16 rows, nodes at 2^17 and 2^18, opened paths at
three CTAs of quads per SM.  Exact against the oracle."""
import numpy as np
import pytest

import whir_gb300 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_h,row_len", [(15, 16), (16, 16), (16, 5), (18, 8), (19, 4), (19, 16)])
def test_levels(ctx, oracle, log_h, row_len):
    rows = oracle.rand_fe(700 + log_h, row_len << log_h)
    rows[:row_len] = W.P - 1
    rows[row_len:2 * row_len] = 0
    t = W.MerkleTree(ctx, ctx.to_device(rows), log_h, row_len)
    assert np.array_equal(t.levels(), oracle.merkle_tree(rows, log_h, row_len))
    t.close()


def test_paths(ctx, oracle):
    # one proof's openings at every count near the line, one of them corrupted
    params = (12, 4, 1, 1, 1, 100)
    poly = oracle.rand_fe(71, 1 << 12)
    proof, cp = W.prove_harness(ctx, params, [poly], [12], [[0]])
    bad = bytearray(proof)
    bad[-5] ^= 1  # a word of the last opening's path
    bad = bytes(bad)
    want = [W.verify(params, [12], [[0]], p) for p in (proof, bad)]
    assert want[0] == (0, cp) and want[1][0] != 0
    for n in (20, 40, 80, 160):
        proofs = [proof] * n
        proofs[n // 2] = bad
        got = W.verify_batch(ctx, params, [12], [[0]], proofs)
        assert got == [want[1] if i == n // 2 else want[0] for i in range(n)]
