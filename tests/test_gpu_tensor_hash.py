"""Merkle trees at the sizes where the tensor-core hash kernels take over.

The leaf and node kernels are chosen by row and node count; every level of
each tree equals the oracle's (exact: zero tolerance).  Row lengths cover one
and several sponge chunks, a shorter last chunk, and rows off the 16-byte
grid; the first rows hold the extreme words 0 and p - 1, which bound the
kernels' sums.
"""
import ctypes

import numpy as np
import pytest

import whir_gb300 as W

pytestmark = pytest.mark.gpu


def _rows(oracle, log_h, row_len):
    rows = oracle.rand_fe(900 + log_h + row_len, row_len << log_h)
    rows[:row_len] = 0
    rows[row_len:3 * row_len] = W.P - 1
    rows[3 * row_len:5 * row_len:2] = W.P - 1
    rows[3 * row_len + 1:5 * row_len:3] = 0
    return rows


@pytest.mark.parametrize("log_h,row_len", [
    (15, 64), (16, 16), (16, 17), (16, 31), (16, 64), (16, 100), (17, 4), (17, 8), (17, 12), (17, 16),
    (17, 2), (17, 33), (18, 48),
])
def test_levels(ctx, oracle, log_h, row_len):
    rows = _rows(oracle, log_h, row_len)
    t = W.MerkleTree(ctx, ctx.to_device(rows), log_h, row_len)
    assert np.array_equal(t.levels(), oracle.merkle_tree(rows, log_h, row_len))
    t.close()


def test_rows_off_the_vector_grid(ctx, oracle):
    log_h, row_len = 17, 16
    rows = _rows(oracle, log_h, row_len)
    dev = ctx.to_device(np.concatenate([np.zeros(1, np.uint32), rows]))
    h, root = ctypes.c_void_p(), np.zeros(8, np.uint32)
    W._check(W.lib().whir_merkle_commit(ctx.h, dev.ptr + 4, log_h, row_len, ctypes.byref(h),
                                        root.ctypes.data_as(W.u32p)))
    W._check(W.lib().whir_merkle_free(h))
    assert np.array_equal(root, oracle.merkle_tree(rows, log_h, row_len)[-8:])


def test_interleaved_batch(ctx, oracle):
    # 5 x 2^15 leaves in one launch
    params, n = (18, 4, 1, 1, 1, 100), 5
    polys = [oracle.rand_fe(40 + i, 1 << 18) for i in range(n)]
    got = W.prove_batch(ctx, params, polys, claims=0, commit_only=True)
    for i in range(n):
        w, t = W.Whir(ctx, *params), W.PoseidonWriter()
        w.commit(t, [polys[i]], [18])
        cp = t.draw_base()
        assert got[i] == (t.finalize(), cp)
