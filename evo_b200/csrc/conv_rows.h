// Host rule of evo_conv_act: rows per CTA of the kernel with four channels per thread.
#pragma once
#include <algorithm>
#include <cstdint>

namespace evo {

// CTAs of `rows` consecutive rows of one sequence and one block of channels (`per` of these pairs), `slots` of them on the chip at once.  A wave takes the time of its rows and of a CTA's start,
// about 16 rows' (taps, the inputs in front): one wave of CTAs that end together instead of many short ones (4 x 4096 x 6144 with six CTAs per SM: 88 us by 32 rows, 83 so).  Where that leaves
// many places empty, more waves of shorter CTAs may fill them better.  Candidates are k waves with the most CTAs per pair, m, that they have room for: by k where a wave holds all pairs, by m
// where it does not.  k waves take no less than all rows spread evenly and k starts; the search ends where that is no gain any more.  Host time: below 1 us at every length whose
// rows fit a GPU, 0.3 at most for 8192 rows (a search through 1024 splits took 3, and 11 from 32768 rows on).
inline int64_t conv_rows(int64_t L, int64_t per, int64_t slots, int64_t least) {
  constexpr int64_t START = 16, MOST = 1 << 30;
  const int64_t even = L * per / slots, longest = std::max<int64_t>(1, L / least);
  int64_t best = least, cost = INT64_MAX;
  for (int64_t step = 1; step <= 100; ++step) {
    const int64_t k = per <= slots ? step : (step * per + slots - 1) / slots, m = std::min(per <= slots ? step * slots / per : step, longest);
    if (even + k * START >= cost) break;
    const int64_t rows = std::min(MOST, std::max(least, ((L + m - 1) / m + 3) / 4 * 4));
    if (k * (rows + START) < cost) { cost = k * (rows + START); best = rows; }
    if (m == longest) break;
  }
  return best;
}

}  // namespace evo
