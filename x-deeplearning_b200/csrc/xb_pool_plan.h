// How a pooling group's segments are split over warps: host arithmetic alone, so that it can be checked for any number of SMs.
#pragma once

#include <algorithm>
#include <cstdint>

#ifdef __CUDACC__
#define XB_PLAN_HD __host__ __device__ __forceinline__
#else
#define XB_PLAN_HD inline
#endif

namespace xb {

enum class PoolPath { GENERAL, FAST, SHORT, QUEUE };      // pool_kernel, pool_fast_kernel, pool_short_kernel, pool_queue_kernel

struct PoolSplit {
  int segs;             // rounds of 32 / tl segments a warp walks; queue kernel: segments a warp owns
  int64_t warps;
};

// `tl` lanes work on a segment; `avg` ids a segment; `counts`: the group's segments are counts that the warps add up themselves
inline PoolSplit pool_split(PoolPath path, int64_t batch, int tl, double avg, bool counts, int queue_segs, int sms) {
  const int spw = 32 / tl;
  const int64_t rounds = (batch + spw - 1) / spw;
  auto clamp8 = [](int64_t v) { return (int)std::max<int64_t>(1, std::min<int64_t>(8, v)); };
  PoolSplit s;
  s.segs = 1;
  switch (path) {
    case PoolPath::QUEUE:
      s.segs = std::max(queue_segs, spw);
      s.warps = (batch + s.segs - 1) / s.segs;
      return s;
    case PoolPath::SHORT:
      // the short-segment kernel walks 8 rounds per warp (its prefetch needs a few), fewer only for small groups
      s.segs = clamp8(rounds / ((int64_t)sms * 16));
      break;
    case PoolPath::FAST:
      // The specialised kernel gives a warp several rounds, as long as every SM still gets dozens of warps (fewer with a
      // list of one or two ids, whose warp is a chain of latencies: its rounds overlap, while a second wave of warps would
      // begin the chain again: 2 x 74 000 single ids and their requests' lists 17.7 -> 13.1 us). A warp that adds up the
      // counts before its first segment knows the start of one round only, whatever the number of SMs.
      if (!counts) s.segs = clamp8(rounds / ((int64_t)sms * (avg < 3.0 ? 12 : 48)));
      break;
    case PoolPath::GENERAL: break;
  }
  s.warps = (rounds + s.segs - 1) / s.segs;
  return s;
}

// Queue kernel. A launch is one wave of warps, so a warp's share is all that it will do, and shares are made equal in time: in batches
// of ids, not in segments. A list of `avg` ids is this many batches of `lanes` ids on average.
inline double pool_queue_cost(double avg, int lanes) { return std::max(1.0, avg / lanes + 0.5); }

struct PoolQueueGroup { int64_t batch; double cost; };
struct PoolQueueShare { double share, mean; };          // cost of a warp's share, mean cost of a list

// Segments a warp owns in a group whose lists cost `cost`, no less than 8 mean lists' worth. Lists much longer than the launch's
// other ones go to whole rounds of the `spw` sub-teams: with one list more than those a warp takes twice the time.
inline int pool_queue_segs(const PoolQueueShare& q, double cost, int spw) {
  int64_t segs = (int64_t)(q.share / cost);
  if (cost >= 2 * q.mean && segs < 4 * spw) segs = segs / spw * spw;
  else if ((double)segs * cost < q.share) ++segs;
  const int least = std::max(spw, (int)std::min(8.0, 8 * q.mean / cost + 0.999));
  return (int)std::max<int64_t>(least, std::min<int64_t>(segs, 1 << 30));
}

// The share with which the groups of a launch fit `warps` warps.
inline PoolQueueShare pool_queue_share(const PoolQueueGroup* g, int n, int spw, int64_t warps) {
  PoolQueueShare q = {0, 0};
  double segments = 0;
  for (int i = 0; i < n; ++i) { q.share += (double)g[i].batch * g[i].cost; segments += (double)g[i].batch; }
  q.mean = q.share / segments;
  q.share /= (double)std::max<int64_t>(warps - n, 1);
  for (int tries = 0; tries < 32; ++tries, q.share *= 1.03) {
    int64_t need = 0;
    for (int i = 0; i < n; ++i) {
      const int segs = pool_queue_segs(q, g[i].cost, spw);
      need += (g[i].batch + segs - 1) / segs;
    }
    if (need <= warps) break;
  }
  return q;
}

// Segment number m of warp w of a group's `warps`, `segs` segments each: pieces side by side, and what is left of the shares at the
// end, in turn from either side, so that lists sorted by length, or lengths that drift over the group, spread over the warps. May lie
// past the group's end.
constexpr int POOL_QUEUE_PIECE_LOG = 4;
XB_PLAN_HD int64_t pool_queue_segment(int m, int64_t w, int64_t warps, int segs) {
  const int piece = m >> POOL_QUEUE_PIECE_LOG, pieces = (segs - 1) >> POOL_QUEUE_PIECE_LOG, first = piece << POOL_QUEUE_PIECE_LOG;
  const int64_t at = piece & 1 ? warps - 1 - w : w;
  return (int64_t)first * warps + at * (piece < pieces ? 1 << POOL_QUEUE_PIECE_LOG : segs - first) + (m - first);
}

}  // namespace xb
