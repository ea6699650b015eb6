"""How a pooling group's segments are split over warps, for any number of SMs (a slice of the GPU has few of them): every
segment is some warp's, and a group whose counts its warps add up themselves is walked in single rounds, because such a warp
knows the start of one round only."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "x-deeplearning_b200", "csrc")
GENERAL, FAST, SHORT, QUEUE = range(4)


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src, so = str(d / "plan.cc"), str(d / "plan.so")
    with open(src, "w") as f:
        f.write('#include "xb_pool_plan.h"\n'
                'extern "C" long long plan(int path, long long batch, int tl, double avg, int counts, int q, int sms, int* segs) {\n'
                "  const xb::PoolSplit s = xb::pool_split((xb::PoolPath)path, batch, tl, avg, counts != 0, q, sms);\n"
                "  *segs = s.segs;\n  return s.warps;\n}\n")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I" + CSRC, src, "-o", so])
    lib = ctypes.CDLL(so)
    lib.plan.restype = ctypes.c_longlong
    lib.plan.argtypes = [ctypes.c_int, ctypes.c_longlong, ctypes.c_int, ctypes.c_double, ctypes.c_int, ctypes.c_int, ctypes.c_int,
                         ctypes.POINTER(ctypes.c_int)]

    def call(path, batch, tl, avg, counts, q, sms):
        segs = ctypes.c_int()
        warps = lib.plan(path, batch, tl, avg, counts, q, sms, ctypes.byref(segs))
        return segs.value, warps

    return call


@pytest.mark.parametrize("sms", [1, 8, 16, 36, 42, 43, 74, 132, 148])
@pytest.mark.parametrize("tl", [2, 4, 8, 16, 32])
def test_split(split, sms, tl):
    spw = 32 // tl
    for batch in (1, 2, spw, spw + 1, 31, 512, 1000, 1023, 1024):
        for avg in (0.0, 2.0, 2.99, 3.0, 50.0):
            segs, warps = split(FAST, batch, tl, avg, 1, 32, sms)
            assert segs == 1 and warps == (batch + spw - 1) // spw
    for batch in (1, 1025, 8192, 74000, 1 << 22, (1 << 31) - 1):
        for avg in (1.0, 15.0):
            for path in (GENERAL, FAST, SHORT, QUEUE):
                for q in (8, 32):
                    segs, warps = split(path, batch, tl, avg, 0, q, sms)
                    per_warp = segs if path == QUEUE else segs * spw
                    assert 1 <= segs <= max(32, spw) and (warps - 1) * per_warp < batch <= warps * per_warp
