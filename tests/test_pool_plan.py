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


QUEUE_SRC = '''#include "xb_pool_plan.h"
extern "C" void shares(const long long* batch, const double* avg, int n, int lanes, long long warps, int* segs) {
  xb::PoolQueueGroup g[32];
  for (int i = 0; i < n; ++i) g[i] = {batch[i], xb::pool_queue_cost(avg[i], lanes)};
  const xb::PoolQueueShare q = xb::pool_queue_share(g, n, 32 / lanes, warps);
  for (int i = 0; i < n; ++i) segs[i] = xb::pool_queue_segs(q, g[i].cost, 32 / lanes);
}
extern "C" long long segment(int m, long long w, long long warps, int segs) { return xb::pool_queue_segment(m, w, warps, segs); }
'''


@pytest.fixture(scope="module")
def queue(tmp_path_factory):
    d = tmp_path_factory.mktemp("queue")
    src, so = str(d / "queue.cc"), str(d / "queue.so")
    with open(src, "w") as f:
        f.write(QUEUE_SRC)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I" + CSRC, src, "-o", so])
    lib = ctypes.CDLL(so)
    lib.segment.restype = ctypes.c_longlong
    lib.segment.argtypes = [ctypes.c_int, ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int]
    lib.shares.argtypes = [ctypes.POINTER(ctypes.c_longlong), ctypes.POINTER(ctypes.c_double), ctypes.c_int, ctypes.c_int, ctypes.c_longlong,
                           ctypes.POINTER(ctypes.c_int)]
    return lib


@pytest.mark.parametrize("lanes", [2, 4, 8, 16])
@pytest.mark.parametrize("warps", [4736, 1184])
@pytest.mark.parametrize("groups", [[(8192, 15.5)] * 32, [(8192, 45)] + [(8192, 4)] * 31, [(65536, a) for a in (3, 15, 30, 45, 5, 4.5, 45, 15)],
                                    [(16384, 40), (16384, 3)] * 16, [(1_000_000, 4), (3000, 47)], [(300_000, 9), (33, 9)]])
def test_the_queue_kernels_shares_take_the_same_time(queue, groups, lanes, warps):
    """One wave, and no warp has more than a third above what every warp would have, but for the rounding up to a list a sub-team."""
    n, spw = len(groups), 32 // lanes
    batch, avg, segs = (ctypes.c_longlong * n)(*[b for b, _ in groups]), (ctypes.c_double * n)(*[a for _, a in groups]), (ctypes.c_int * n)()
    queue.shares(batch, avg, n, lanes, warps, segs)
    cost = [max(1.0, a / lanes + 0.5) for _, a in groups]
    assert sum(-(-b // s) for (b, _), s in zip(groups, segs)) <= warps
    fair = sum(b * c for (b, _), c in zip(groups, cost)) / warps
    mean = sum(b * c for (b, _), c in zip(groups, cost)) / sum(b for b, _ in groups)
    for s, c in zip(segs, cost):
        assert s >= spw and (s >= 8 or c > mean) and (s * c <= 1.34 * fair + c or s <= max(8, spw))


@pytest.mark.parametrize("batch,segs", [(1, 8), (9, 8), (100, 17), (101, 33), (8192, 69), (5000, 16), (70001, 55), (300, 299), (37900, 8)])
def test_every_segment_is_one_warps(queue, batch, segs):
    warps = -(-batch // segs)
    got = [queue.segment(m, w, warps, segs) for w in range(warps) for m in range(segs)]
    assert sorted(x for x in got if x < batch) == list(range(batch)) and len(set(got)) == len(got)
    for w in range(warps):                                     # past the end only after a warp's last one
        mine = got[w * segs:(w + 1) * segs]
        assert mine == sorted(mine)
