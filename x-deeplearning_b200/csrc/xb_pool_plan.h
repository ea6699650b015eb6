// How a pooling group's segments are split over warps: host arithmetic alone, so that it can be checked for any number of SMs.
#pragma once

#include <algorithm>
#include <cstdint>

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

}  // namespace xb
