"""Launch shapes of the kernels that form their own eq tables (point_plan.h),
compiled for the host and checked over every size the entry points take."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "whir_gb300", "csrc")
SOURCE = """
#include <stdint.h>
#include "point_plan.h"
using namespace whir::gpu;
extern "C" int low(int k, int ks) { return compress_hi_point_low(k, ks); }
static void put(const PointLaunch &l, uint64_t *out) { out[0] = l.ctas; out[1] = l.smem; }
extern "C" void compress(int k, int ks, uint64_t *out) { put(compress_hi_point_launch(k, ks), out); }
extern "C" void eval_ext(int k, uint64_t *out) { put(eval_ext_point_launch(k), out); }
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


def _launch(fn, *args):
    out = (ctypes.c_uint64 * 2)()
    fn(*args, out)
    return out[0], out[1]


def test_every_size_fits_shared_memory(plan):
    # no size the entry points take (at most 32 fixed variables, 30 for an
    # evaluation) needs another kernel: 48 KB hold a CTA's tables, its columns'
    # sums, the high entries of all its blocks and the kernel's static words
    for k in range(0, 41):
        for ks in range(max(0, k - 32), min(k, 8) + 1):
            s = plan.low(k, ks)
            ctas, smem = _launch(plan.compress, k, ks)
            blocks = 1 << (k - ks - s)
            assert 1 <= ctas <= blocks and ctas < 1 << 31
            need = 16 * ((1 << s) + 64 - (-blocks // ctas)) + (32 << ks)
            assert need <= smem <= 47 * 1024, (k, ks)
    for k in range(0, 31):
        ctas, smem = _launch(plan.eval_ext, k)
        blocks = 1 << max(0, k - 8)
        assert 1 <= ctas <= blocks
        assert 16 * (64 - (-blocks // ctas)) <= smem <= 47 * 1024, k


def test_usual_sizes_keep_the_usual_ctas(plan):
    assert _launch(plan.compress, 24, 4)[0] == 152 * 3
    assert _launch(plan.compress, 24, 0)[0] == 152 * 4
    assert _launch(plan.compress, 30, 0)[0] == 152 * 4
    assert _launch(plan.eval_ext, 24)[0] == 152 * 8
    assert _launch(plan.eval_ext, 29)[0] == 152 * 8
