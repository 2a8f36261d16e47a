// How long an FGP launch, and the launches of a solve, take by the kernel and
// cluster that run them: the rule that picks them (Solver::pick_fgp_shape).
// Host arithmetic only.
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
// mean error 4 %; the fastest candidate by it takes 0.6 % more than the fastest
// on average and 13 % at most.
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

// What the candidates are compared by: a launch with every problem active and
// one with a single problem left.  Solves of a batch end one by one, so many of
// their launches run few problems, and the kernel that is fastest with all of
// them can be the slowest then (FP32, 16 of 128 x 128: k_fgp 220 us, 195 with one
// left; k_fgp_reg 246 and 107; 100 iterations of the solve 74 and 53 ms).  The
// weight fits 48 batches of 8 to 64 problems, 64 to 160 pixels a side, both
// precisions, for 100 iterations and to convergence: the pick's solve takes 1.2
// % more than the fastest on average and 10 % at most; by the full launch alone
// 12 % and 72 %, by one fixed time per candidate 30 % and 168 %.
inline double fgp_solve_cost(const FgpCandidate& c, bool fp64, int NX, int NY, int B, int sms) {
  return fgp_cost(c, fp64, NX, NY, B, sms) + 1.25 * fgp_cost(c, fp64, NX, NY, 1, sms);
}

}  // namespace mf
