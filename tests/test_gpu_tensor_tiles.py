"""Node compression on the tensor cores over several passes of its five tiles
per CTA, the last one partly filled (97280 nodes a pass): single trees and an
interleaved batch of three.  Exact against the oracle and single commitments.
"""
import numpy as np
import pytest

import whir_gb300 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_h", [18, 19, 20])
def test_levels(ctx, oracle, log_h):
    rows = oracle.rand_fe(log_h, 4 << log_h)
    rows[:64] = W.P - 1
    t = W.MerkleTree(ctx, ctx.to_device(rows), log_h, 4)
    assert np.array_equal(t.levels(), oracle.merkle_tree(rows, log_h, 4))
    t.close()


def test_interleaved_batch(ctx, oracle):
    params, n = (19, 2, 1, 1, 1, 100), 3  # 3 x 2^18 leaves, 3 x 2^17 nodes
    polys = [oracle.rand_fe(70 + i, 1 << 19) for i in range(n)]
    got = W.prove_batch(ctx, params, polys, claims=0, commit_only=True)
    for i in range(n):
        w, t = W.Whir(ctx, *params), W.PoseidonWriter()
        w.commit(t, [polys[i]], [19])
        cp = t.draw_base()
        assert got[i] == (t.finalize(), cp)
