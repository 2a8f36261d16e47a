// How long an FGP launch takes by the kernel and cluster that run it: the rule
// that picks them (Solver::pick_fgp_shape).  Host arithmetic only.
#pragma once
#include <algorithm>

namespace mf {

// A candidate: k_fgp_reg with `nr` rows a thread (1 or 2), or k_fgp (nr = 0),
// `cs` CTAs a problem, of which `resident` problems fit the GPU at once.
struct FgpCandidate {
  int nr, cs, resident;
};

// Microseconds of 50 iterations for B problems of NX x NY on `sms` SMs.
// Problems run in rounds of those resident at once; a round takes
//   (base + per * work) (1 + share * max(0, CTAs per SM - alone)),
// work: the CTA's threads by 1024 (k_fgp_reg: one pass over its pixels, bound
// by the barrier and the FP64 or FP32 pipe), or the passes of its 256 threads
// over its rows (k_fgp: each a chain of shared-memory accesses); share: what
// the CTAs of an SM cost each other.  Fitted to 3000 launches on B200 (both
// precisions, 32 to 160 pixels a side, 1 to 128 problems, every candidate):
// mean error 4 %; the candidate it picks takes 0.6 % more than the fastest on
// average and 13 % at most, and 6 % less than a rule with one time per
// candidate, which took up to 1.5 times as long as k_fgp (FP32, 128 problems of
// 72 x 72: 580 us, now 381).
inline double fgp_cost(const FgpCandidate& c, bool fp64, int NX, int NY, int B, int sms) {
  struct Fit {
    double base, per, share, alone;
  };
  static const Fit fit[2][3] = {{{57, 34, 0.10, 0.6}, {61, 11, 0.05, 0.6}, {92, 30, 0.05, 0.0}},    // FP32: nr 0, 1, 2
                                {{54, 34, 0.10, 0.6}, {54, 16, 0.10, 0.6}, {105, 45, 0.07, 0.2}}};  // FP64
  if (c.resident < 1) return 1e300;
  const int rows = (NY + c.cs - 1) / c.cs;
  double work;
  if (c.nr) {
    work = (double)((rows + c.nr - 1) / c.nr) * NX / 1024;
  } else {
    const int per_pass = std::max(1, 256 / NX);
    work = (double)((rows + per_pass - 1) / per_pass) * ((NX + 255) / 256);
  }
  const Fit& f = fit[fp64 ? 1 : 0][c.nr];
  auto round = [&](int n) {
    return n ? (f.base + f.per * work) * (1 + f.share * std::max(0.0, (double)n * c.cs / sms - f.alone)) : 0.0;
  };
  return (B / c.resident) * round(c.resident) + round(B % c.resident);
}

}  // namespace mf
