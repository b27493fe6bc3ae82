"""The rules that choose a pair's form (csrc/sw_plan.h), compiled for the
host: every query length has a bin whose lanes and rows hold it, and no pair
that may pass 16 bits is laid beside another one."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = """
#include "sw_plan.h"
using namespace tpz::sw;
extern "C" {
int t_row_bin(int ql, int sl, int small, int steps) { return row_bin(ql, sl, small, steps); }
int t_group_lanes(int ql) { return group_lanes(ql); }
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
    return ctypes.CDLL(so)


def _rows_lanes(b):
    if b < 24:
        return b + 9, 32
    if b < 48:
        return (b - 24) % 8 + 9, (16, 8, 4)[(b - 24) // 8]
    return (4, 8)[b - 48], 4


def test_every_length_has_a_bin_that_holds_it(plan):
    for ql in range(1, 8193):
        b = plan.t_row_bin(ql, 100, 0, 1 << 30)
        if ql <= 1024:
            R, G = _rows_lanes(b)
            assert b < 50 and R * G >= ql and (R <= 16 or G == 32)
            small = plan.t_row_bin(ql, 100, 1, 1 << 30)
            assert small in (53, 54) and (small == 54) == (ql > 512)
        else:
            assert 50 <= b <= 52 and ql <= (2048, 4096, 8192)[b - 50]
            assert plan.t_row_bin(ql, 100, 1, 1 << 30) == b


@pytest.mark.parametrize("floor,entry", [(76, 11), (97, 15), (238, 17), (373, 64), (637, 127), (513, 127), (65, 1)])
def test_pairs_past_16_bits_have_their_words_to_themselves(plan, floor, entry):
    steps = plan.t_shared_steps(floor, entry)
    assert floor + steps * entry <= 65535 < floor + (steps + 1) * entry
    for n in (1, 30, 100, 400, 505, 512, 513, 516, 517, 1000, 1024):
        for m in (0, 100, 505, 513, 517, 1024, 5000):
            b = plan.t_row_bin(n, m, 0, steps)
            assert (b >= 50) == (min(n, m) * entry + floor > 65535)
    assert plan.t_shared_steps(floor, 0) == plan.t_shared_steps(floor, -3) == 2 ** 31 - 1
