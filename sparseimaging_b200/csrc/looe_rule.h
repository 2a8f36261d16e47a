// On how many streams the leave-one-out errors of a call run.  Host arithmetic
// only.
#pragma once

namespace mf {

// Streams for B solutions of `panels` panels of active pixels and `rows`
// visibilities: each costs a call 0.09 ms (its creation and destruction, its
// scratch), and a solution takes 0.04 ms, 0.04 a panel and 0.05 per thousand
// rows at least.  With a stream for every solution up to four, two to five
// solutions of one panel took 5-20 % longer than on one stream (3 of 3 pixels,
// 40 rows: 0.99 ms, 1.15 on three).
inline int looe_lanes(int B, int panels, int rows, int most) {
  constexpr long kLane = 90, kSolution = 40, kOfPanel = 40, kRowsOfOne = 20;  // us
  int best = 1;
  long cost = 0;
  for (int n = 1; n <= most && n <= B; ++n) {
    const long t = n * kLane + (long)((B + n - 1) / n) * (kSolution + kOfPanel * panels + rows / kRowsOfOne);
    if (n == 1 || t < cost) {
      best = n;
      cost = t;
    }
  }
  return best;
}

}  // namespace mf
