"""A hash kernel whose wait for the matrix unit runs out reports an error.

Expired waits let a healthy launch give up: the kernel goes on without
waiting, waits for its products once at its end, and the call returns an error.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

import whir_gb300 as W

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GIVE_UP = """
import sys
import numpy as np
import whir_gb300 as W
log_h, row_len = int(sys.argv[1]), int(sys.argv[2])
ctx = W.Context(0)
dev = ctx.to_device(np.ones(row_len << log_h, np.uint32))
W.debug_expire_waits(ctx)
try:
    W.MerkleTree(ctx, dev, log_h, row_len)
except W.WhirError as e:
    assert "wait ran out" in str(e), e
    print("gave up")
"""


# leaves and nodes on the tensor kernels, one tile and several in turn
@pytest.mark.parametrize("log_h,row_len", [(17, 16), (16, 40), (20, 16)])
def test_a_wait_that_runs_out_is_reported(log_h, row_len):
    r = subprocess.run([sys.executable, "-c", GIVE_UP, str(log_h), str(row_len)], cwd=ROOT,
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "gave up" in r.stdout, r.stderr


# ---- the error belongs to the context whose kernel gave up, and is reported once ----
@pytest.fixture
def own():
    c = W.Context(0)
    yield c
    W.debug_expire_waits(c, False)
    c.close()


def _fails(ctx, fn):
    W.debug_expire_waits(ctx)
    with pytest.raises(W.WhirError, match="wait ran out"):
        fn()
    W.debug_expire_waits(ctx, False)


def test_the_next_call_and_other_contexts_are_not_failed(own, ctx, oracle):
    log_h, row_len = 17, 16
    rows = oracle.rand_fe(31, row_len << log_h)
    root = oracle.merkle_tree(rows, log_h, row_len)[-8:]
    mine, other = own.to_device(rows), ctx.to_device(rows)
    _fails(own, lambda: W.MerkleTree(own, mine, log_h, row_len))
    for c, dev in ((ctx, other), (own, mine), (W.Context(0), mine)):
        assert np.array_equal(W.MerkleTree(c, dev, log_h, row_len).root, root)


def test_an_earlier_tree_is_released(own, oracle):
    rows = own.to_device(oracle.rand_fe(32, 16 << 17))
    t = W.MerkleTree(own, rows, 17, 16)
    _fails(own, lambda: W.MerkleTree(own, rows, 17, 16))
    assert W.lib().whir_merkle_free(t.h) == 0
    t.h = None


def test_provers_go_on_after_it(own, oracle):
    params, k = (19, 4, 2, 1, 1, 100), 19  # 2^17 rows
    poly = oracle.rand_fe(33, 1 << k)
    whir = W.Whir(own, *params)
    want = W.prove_harness(own, params, [poly], [k], [[0]], whir)
    _fails(own, lambda: W.prove_harness(own, params, [poly], [k], [[0]], whir))
    assert W.prove_harness(own, params, [poly], [k], [[0]], whir) == want
    _fails(own, lambda: W.prove_batch(own, params, [poly] * 2))
    assert W.prove_batch(own, params, [poly] * 2) == [want] * 2


def test_autotune_reports_its_own(own):
    try:
        _fails(own, lambda: W.autotune(own, 19, 19))
        W.autotune(own, 19, 19)
    finally:
        W.tune_reset()
