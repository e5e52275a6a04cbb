"""Batched path checks on warps, quads of lanes and threads: batches whose path
counts lie on each side of the two lines (1024 and 10240), with proofs of
mixed row lengths and heights in one warp, and corrupted openings among them.
Each result is whir_verify's for the proof alone.
"""
import numpy as np
import pytest

import whir_gb300 as W

pytestmark = pytest.mark.gpu


# rows of 8 and 32 words at folding 3, of 16 and 64 at 4, of 4 at 2 (a short
# chunk); about 120 paths a proof
@pytest.mark.parametrize("params", [(12, 4, 1, 1, 1, 100), (13, 3, 1, 1, 1, 100),
                                    (10, 2, 1, 1, 1, 64)])
@pytest.mark.parametrize("n", [1, 7, 9, 40, 130])
def test_batches(ctx, oracle, params, n):
    k = params[0]
    poly = oracle.rand_fe(k, 1 << k)
    proof, cp = W.prove_batch(ctx, params, [poly], claims=1)[0]
    rng = np.random.default_rng(n)
    batch, want = [], []
    alone = {}
    for i in range(n):
        b = proof
        if i % 5 == 4:  # one flipped bit of a word's low byte, anywhere in the proof
            bad = bytearray(proof)
            bad[4 * int(rng.integers(0, len(bad) // 4))] ^= 1
            b = bytes(bad)
        if b not in alone:
            alone[b] = W.verify(params, [k], [[0]], b)
        batch.append(b)
        want.append(alone[b])
    assert alone[proof] == (0, cp)
    assert W.verify_batch(ctx, params, [k], [[0]], batch) == want
    assert n < 7 or any(r != 0 for r, _ in want)
