"""How many CTAs share an attention tile: only as many as run at once beside the call's other tiles, so that a call that fills
the GPU by itself walks its tiles whole, and never so many that the grid outgrows what a launch takes."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "x-deeplearning_b200", "csrc")


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src, so = str(d / "plan.cc"), str(d / "plan.so")
    with open(src, "w") as f:
        f.write('#include "xb_att_plan.h"\nextern "C" int plan(long long tiles, int T, const int* slots) {\n'
                "  return xb::att_split(tiles, T, [slots](int lg) { return slots[lg]; });\n}\n")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I" + CSRC, src, "-o", so])
    lib = ctypes.CDLL(so)
    lib.plan.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_void_p]
    return lambda tiles, T, slots: lib.plan(tiles, T, (ctypes.c_int * 4)(*slots))


@pytest.mark.parametrize("slots", [(148, 148, 144, 136), (74, 72, 64, 64), (148, 0, -1, 0)])
def test_split(split, slots):
    for T in (1, 2, 3, 8, 17, 50, 100, 256):
        for tiles in list(range(1, 200)) + [592, 10_000, 1 << 28, (1 << 31) - 1]:
            s = split(tiles, T, slots)
            assert s in (1, 2, 4, 8) and s <= T
            assert s == 1 or tiles * s <= slots[s.bit_length() - 1]
            assert tiles * s < 1 << 31
            if s > 1:
                assert -(-T // s) + 11 < T + 8
    full = (148, 148, 144, 136)
    assert [split(t, 100, full) for t in (1, 16, 17, 32, 36, 37, 72, 74, 75, 96, 148, 192, 448)] == [8, 8, 8, 4, 4, 2, 2, 2, 1, 1, 1, 1, 1]
