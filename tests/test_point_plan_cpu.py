"""Launch shapes of the kernels that form their own eq tables (point_plan.h),
compiled for the host and checked over every size the entry points take."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "whir_gb300", "csrc")
SOURCE = """
#include "point_plan.h"
extern "C" int low(int k, int ks) { return whir::gpu::compress_hi_point_low(k, ks); }
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SOURCE)
    so = str(d / "plan.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", so,
                    str(d / "plan.cpp")], check=True)
    return ctypes.CDLL(so)


def test_blocks_of_large_polynomials_amortise_their_product(plan):
    # a thread (of 256) multiplies its words of a block into one extension
    # product: at least four of them, sixteen where a low table of 2^10 reaches
    for k in range(20, 31):
        for ks in range(0, 9):
            s = plan.low(k, ks)
            assert 0 <= s <= min(10, k - ks)
            assert s + ks >= min(12, 10 + ks), (k, ks, s)


def test_low_tables_fit_every_size(plan):
    for k in range(0, 31):
        for ks in range(0, min(k, 8) + 1):
            assert 0 <= plan.low(k, ks) <= min(10, k - ks)
