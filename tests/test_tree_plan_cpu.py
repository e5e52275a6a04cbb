"""How a tree's narrow part is cut into launches (tree_plan.h), compiled for the
host, and the tunings that the library takes."""
import ctypes
import os
import subprocess

import pytest

import whir_gb300 as W

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "whir_gb300", "csrc")
SOURCE = """
#include "tree_plan.h"
extern "C" int split(int S, int t) { return whir::gpu::tree_first_split(S, t); }
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SOURCE)
    so = str(d / "plan.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", so,
                    str(d / "plan.cpp")], check=True)
    return ctypes.CDLL(so)


def test_a_split_moves_the_default_where_subtrees_fit(plan):
    # at most 2^9 nodes per CTA in the first launch, and 2^9 CTAs
    for levels in range(1, 19):
        base = plan.split(levels, 0)
        for t in (-1, 0, 1):
            g = plan.split(levels, t)
            assert max(0, levels - 9) <= g <= min(9, levels)
            assert g == min(max(base + t, levels - 9, 0), levels, 9), (levels, t)


def test_default_splits(plan):
    # the sizes of the default threshold: up to 2^16 nodes at the first narrow level
    want = {1: 0, 5: 0, 6: 3, 9: 4, 10: 6, 11: 7, 14: 7, 15: 7, 16: 7, 17: 8, 18: 9}
    assert {s: plan.split(s, 0) for s in want} == want


def test_tunings_taken():
    try:
        for log_h in (0, 9, 16, 17, 18, 24, 40):
            for wide in range(9, 20):
                for split in (-2, -1, 0, 1, 2):
                    ok = 10 <= wide <= 18 and abs(split) <= 1 and \
                        not (min(log_h, wide) == 18 and split == -1)
                    assert (W.lib().whir_tune_tree(log_h, wide, split) == 0) == ok
    finally:
        W.tune_reset()
