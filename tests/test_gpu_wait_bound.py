"""A hash kernel whose wait for the matrix unit runs out reports an error.

Expired waits let a healthy launch give up: the kernel goes on without
waiting, waits for its products once at its end, and the call returns an error.
"""
import os
import subprocess
import sys

import pytest

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
