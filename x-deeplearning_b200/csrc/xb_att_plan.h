// How many CTAs share an attention tile: host arithmetic alone, so that it can be checked for any call.
#pragma once

#include <cstdint>

namespace xb {

// As many as there is room for beside the call's other tiles, where that shortens the walk of `T` steps (a CTA spends about 8
// steps' worth around its steps, a cluster's barriers about 3). slots[lg]: CTAs that can be resident at once as clusters of
// 1 << lg; asked for only as far as needed.
// Clusters that do not all run at once only trim the last wave, and what a CTA spends around its steps is paid again for each:
// on two streams 192 tiles took 141 us a call as clusters of 2 and 119 whole (161 and 180 alone), 96 tiles as clusters of 4
// 94 and 74 (104 and 100 alone). 72 tiles as clusters of 2 take 74 either way, and 69 instead of 99 alone.
template <typename Slots>
inline int att_split(int64_t tiles, int T, Slots slots) {
  int best = 1, cost = T + 8;
  for (int lg = 1; lg <= 3; ++lg) {
    const int s = 1 << lg, c = (T + s - 1) / s + 8 + 3;
    if (s <= T && c < cost && tiles * s <= slots(lg)) { cost = c; best = s; }
  }
  return best;
}

}  // namespace xb
