"""The rules that choose a pair's form (csrc/sw_plan.h), compiled for the
host: every query length has a bin whose lanes and rows hold it, and no pair
that may pass 16 bits is laid beside another one."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = """
#include "sw_plan.h"
using namespace tpz::sw;
extern "C" {
int t_row_bin(int ql, int sl, int64_t pairs, int steps) { return row_bin(ql, sl, forms_of(pairs), steps); }
int t_group_lanes(int ql) { return group_lanes(ql); }
int64_t t_boundary_blocks(int64_t want, int classes, int64_t cols, int sms) {
    return boundary_blocks(want, classes, cols, sms);
}
unsigned t_grid_blocks(int64_t sms, int64_t per_sm, int64_t pairs, int64_t fit) {
    return grid_blocks(sms, per_sm, pairs, fit);
}
int64_t t_boundary_bytes() { return kBoundaryBytes; }
int t_shared_steps(int floor, int entry) { return shared_steps(floor, entry); }
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "plan.so")
    subprocess.check_call(["g++", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "topaz_b200", "csrc"),
                           str(d / "shim.cpp"), "-o", so])
    lib = ctypes.CDLL(so)
    lib.t_boundary_blocks.restype = lib.t_boundary_bytes.restype = ctypes.c_int64
    lib.t_boundary_blocks.argtypes = [ctypes.c_int64, ctypes.c_int, ctypes.c_int64, ctypes.c_int]
    lib.t_row_bin.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int64, ctypes.c_int]
    lib.t_grid_blocks.argtypes = [ctypes.c_int64] * 4
    return lib


def _rows_lanes(b):
    if b < 24:
        return b + 9, 32
    if b < 48:
        return (b - 24) % 8 + 9, (16, 8, 4)[(b - 24) // 8]
    return {48: (4, 4), 49: (8, 4), 55: (4, 8), 56: (8, 8), 57: (8, 16), 58: (8, 32)}[b]


@pytest.mark.parametrize("pairs,stripe,wide,long_slen", [
    (1, 0, 0, None), (64, 0, 0, None), (65, 64, 64, None), (1536, 64, 64, None), (1537, 64, 64, 3072),
    (4096, 64, 64, 3072), (4097, 1024, 64, None), (8192, 1024, 64, None), (8193, 1024, 0, None), (1 << 30, 1024, 0, None)])
def test_every_length_has_a_bin_that_holds_it(plan, pairs, stripe, wide, long_slen):
    for sl in (0, 100, 3071, 3072, 1 << 23):
        for ql in range(1, 8193):
            b = plan.t_row_bin(ql, sl, pairs, 1 << 30)
            is_wide = 16 < ql <= wide or (64 < ql <= 256 and long_slen is not None and sl >= long_slen)
            if ql > 1024:
                assert 50 <= b <= 52 and ql <= (2048, 4096, 8192)[b - 50]
            elif ql > stripe and not is_wide:
                assert b == (53 if ql <= 512 else 54)
            else:
                R, G = _rows_lanes(b)
                assert R * G >= ql and (R <= 16 or G == 32) and (b >= 55) == is_wide


@pytest.mark.parametrize("floor,entry", [(76, 11), (97, 15), (238, 17), (373, 64), (637, 127), (513, 127), (65, 1)])
def test_pairs_past_16_bits_have_their_words_to_themselves(plan, floor, entry):
    steps = plan.t_shared_steps(floor, entry)
    assert floor + steps * entry <= 65535 < floor + (steps + 1) * entry
    for n in (1, 30, 100, 400, 505, 512, 513, 516, 517, 1000, 1024):
        for m in (0, 100, 505, 513, 517, 1024, 5000):
            b = plan.t_row_bin(n, m, 1 << 20, steps)
            assert (b in (53, 54)) == (min(n, m) * entry + floor > 65535)
    assert plan.t_shared_steps(floor, 0) == plan.t_shared_steps(floor, -3) == 2 ** 31 - 1


def test_boundary_rows_stay_within_their_bytes(plan):
    total = plan.t_boundary_bytes()
    for cols in (0, 1, 300, 5000, 36_000, 110_000, 1_000_000, (1 << 24) - 1):
        for classes in (1, 2, 4):
            for want in (1, 7, 74, 148, 296):
                got = plan.t_boundary_blocks(want, classes, cols, 148)
                assert 0 <= got <= want
                assert classes * got * 8 * 8 * max(cols, 1) <= total
                assert got == 0 or 2 * got >= min(want, 148)
    assert plan.t_boundary_blocks(296, 4, 5000, 148) == 296
    assert plan.t_boundary_blocks(148, 1, 36_000, 148) == 148
    assert plan.t_boundary_blocks(1, 1, (1 << 24) - 1, 148) == 0


def test_admission_counts_what_a_batch_takes_once(plan):
    from topaz_b200 import native, serve
    short, long_ = native.batch_device_bytes(1024), native.batch_device_bytes(1025)
    assert long_ - short == plan.t_boundary_bytes()
    assert native.batch_device_bytes(1025, report_hits=0) > long_
    assert native.batch_device_bytes(9000) == short            # not searched

    taken = []

    class Index:
        def search(self, queries, mat, report=None, **kw):
            taken.append([len(q) for q in queries])
            raise RuntimeError("not searched here")

    # room for the short queries, none for the long one's boundary rows
    q = [b"A" * 900] * 3 + [b"A" * 1500] + [b"A" * 900] * 2
    share = [serve.query_device_bytes(len(x)) for x in q]
    srv = serve.SearchServer(Index(), np.zeros((25, 25), np.int8), workers=1,
                             mem_budget=short + sum(share[:4]))
    f = srv.submit(q)
    assert isinstance(f.exception(timeout=30), RuntimeError)
    srv.close()
    assert taken == [[900] * 3, [1500], [900] * 2]


def test_blocks_of_a_launch(plan):
    # more SMs than fixed scratch is for: as many blocks as it holds
    assert plan.t_grid_blocks(148, 4, 1 << 20, 148 * 4) == 148 * 4
    assert plan.t_grid_blocks(160, 4, 1 << 20, 148 * 4) == 148 * 4
    assert plan.t_grid_blocks(148, 4, 100, 148 * 4) == 100
    assert plan.t_grid_blocks(148, 4, 0, 148 * 4) == 1
