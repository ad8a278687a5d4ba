// How the rows of a 2-D grid are divided among the blocks of the marching steps
// (mlw2d_march.cuh).
#pragma once

namespace cans {

// Rows per block of the marching kernel, two of whose blocks fit an SM: a launch
// takes as long as its busiest SM.  A block alone leaves the pipes to its own
// latencies, a second one beside it fills them: the cost is that of pairs and of the
// odd block, in units of a fifth of a microsecond, fitted to the FP64 step at 64^2 ..
// 512^2 (a block of 3, 4, 7, 14, 32 rows alone on its SM 26, 27, 36, 56, 113 us; two
// of 7, 27 rows 49, 146 us).  A segment need not be a whole number of chunks (its
// last chunk may be short, as at the end of the grid).  Against the blocks an SM gets
// times their rows: 192^2 48.9 -> 35.0, 256^2 56 -> 49, 384^2 113 -> 98 us a step.
//
// The cost grows with the rows at an equal number of segments, so only the shortest
// segment of each number is tried: some 2 sqrt(rows) instead of `rows` (every launch
// outside a captured loop searches: 2048 rows 13.4 -> 1.1 us of the host).
inline int balance_seg(int strips, int rows, int ch, int sms) {
  int best = rows;
  long long best_cost = -1;
  for (int seg = 1, n; seg <= rows; seg = n > 1 ? (rows - 1) / (n - 1) + 1 : rows + 1) {
    n = (rows + seg - 1) / seg;
    const long long blocks = (long long)strips * n;
    const long long per_sm = (blocks + sms - 1) / sms, chunks = (seg + ch - 1) / ch;
    const long long cost =
        per_sm / 2 * (80 + 40 * chunks + 18 * seg) + per_sm % 2 * (75 + 25 * chunks + 11 * seg);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = seg;
    }
  }
  return best;
}
// The same with whole chunks per block, balanced by waves of resident
// blocks (slots = SMs x resident blocks per SM): for a step that is bound by
// latency more than by one pipe, fewer and longer blocks can win.
inline int balance_seg_waves(int strips, int rows, int ch, int slots) {
  int best = ch, best_cost = -1;
  for (int seg = ch; seg <= rows + ch - 1; seg += ch) {
    const int blocks = strips * ((rows + seg - 1) / seg);
    const int waves = (blocks + slots - 1) / slots;
    const int cost = waves * (seg + 2);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = seg;
    }
  }
  return best;
}

}  // namespace cans
