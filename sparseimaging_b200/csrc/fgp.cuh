// FGP total-variation proximal operator (c/mfista_TV_lib.c:124-384) as one
// persistent launch per problem: a thread-block cluster owns a problem, each
// CTA a slab of image rows (the NY x NX view of the flat image), and all FGP
// iterations run inside the kernel.  Dual variables live in shared memory
// when the slab fits (halo rows are read from the neighbouring CTA's shared
// memory through DSMEM), otherwise in a per-problem global scratch that the
// same code addresses directly; cluster barriers separate the two stencil
// phases of every iteration.  No TMA and no multicast are used.
//
// Per iteration (c/mfista_TV_lib.c:208-244):
//   A: xv = prox(b - lambda_tv * Lpq(r, s))
//   B: r' = r + Lx(xv)_p / (8 lambda_tv), s' likewise; (np, nq) = P_pqiso(r', s');
//      r = np (1 + (t-1)/t') - p (t-1)/t'; p = np  (same for s, q)
// and finally x = prox(b - lambda_tv * Lpq(p, q)).
#pragma once
#include <cooperative_groups.h>
#include "common.cuh"

namespace mf {

namespace cg = cooperative_groups;

struct FgpArgs {
  const double* z;      // per problem, stride xstride
  const double* dfdx;
  double* xnew;
  long xstride;
  const ProbParams* prm;
  const ProbState* st;
  const float* box;     // shared clean box or null
  int NX, NY;
  int iters;
  int rows_per_cta;
  void* scratch;        // global slabs when not in shared memory
  long scratch_stride;  // bytes per problem
};

// projection of a pixel's duals (P_pqiso, c/mfista_TV_lib.c:160-187): divided by
// their norm where it exceeds 1 (hp, hq: the pixel has a right / lower
// neighbour; a single dual is clamped).  A warp whose duals all lie in the unit
// ball skips the root: most do in a solve (k_fgp, FP32, 100 iterations of one
// 192 x 192 problem 125 ms, 137 without the test), none on the random image of
// mfista_fgp_profile, where the test costs k_fgp 2 %.
template <typename T>
__device__ __forceinline__ void fgp_project(bool hp, bool hq, T rp, T sq, T& np, T& nq) {
  np = rp;
  nq = sq;
  if (hp && hq) {
    const T n2 = fma(rp, rp, sq * sq);
    if (!(n2 <= 1)) {
      if constexpr (sizeof(T) == 8) {  // a third of the instructions of a root and two divisions
        const T inv = rsqrt(n2);
        np = rp * inv;
        nq = sq * inv;
      } else {
        const T tmp = sqrt(n2);
        np = rp / tmp;
        nq = sq / tmp;
      }
    }
  } else if (hp) {
    if (!(fabs(rp) <= 1)) np = rp / fabs(rp);
  } else if (hq) {
    if (!(fabs(sq) <= 1)) nq = sq / fabs(sq);
  }
}

// betas[2 k], [2 k + 1]: (1 + (t_k - 1) / t_{k+1}) and -(t_k - 1) / t_{k+1},
// t_0 = 1
static __global__ void k_fgp_betas(double* __restrict__ betas, int iters) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double tt = 1.0;
  for (int it = 0; it < iters; ++it) {
    double tnew = (1 + sqrt(1 + 4 * tt * tt)) / 2;
    betas[2 * it] = 1 + (tt - 1) / tnew;
    betas[2 * it + 1] = -(tt - 1) / tnew;
    tt = tnew;
  }
}

// slab arrays: xv, p, q, r, s, b — each rows_per_cta x NX values of T
template <typename T, bool SMEM>
__global__ void k_fgp(FgpArgs a, const double* __restrict__ betas) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int csize = (int)cluster.num_blocks();
  const int b = blockIdx.y;
  const ProbState& S = a.st[b];
  // uniform over the cluster (same problem): safe to return before barriers
  if (!gate_ok(S, kGateTrial)) return;
  const ProbParams P = a.prm[b];
  const int NX = a.NX, NY = a.NY, rpc = a.rows_per_cta;
  const int j0 = rank * rpc;
  const int j1 = min(NY, j0 + rpc);
  const int nrow = max(0, j1 - j0);
  const size_t slab = (size_t)rpc * NX;
  T* base;
  if (SMEM) base = reinterpret_cast<T*>(smem_raw);
  else base = reinterpret_cast<T*>(reinterpret_cast<char*>(a.scratch) + (size_t)b * a.scratch_stride) + (size_t)rank * 6 * slab;
  T* XV = base;
  T* PP = base + slab;
  T* QQ = base + 2 * slab;
  T* RR = base + 3 * slab;
  T* SS = base + 4 * slab;
  T* BB = base + 5 * slab;
  // neighbour slabs (rank-1 for the row above, rank+1 for the row below)
  auto peer = [&](T* local, int r) -> T* {
    if (SMEM) return cluster.map_shared_rank(local, r);
    return local + (ptrdiff_t)(r - rank) * 6 * (ptrdiff_t)slab;
  };
  const double c = S.c;
  const double lam_tv = P.lambda_tv / c;
  const double lam_l1 = P.lambda_l1 / c;
  const bool nonneg = P.nonneg == 1;
  const float* box = P.box_flag == 1 ? a.box : nullptr;
  const double* z = a.z + (size_t)b * a.xstride;
  const double* d = a.dfdx + (size_t)b * a.xstride;
  // b = xtmp (c/mfista_nufft_lib.c:424-441) ; duals start at zero
  // thread -> (row, column) walk without integer division: rows_per_pass
  // rows of NX columns per pass when NX <= blockDim.x, else one row with
  // the columns strided by blockDim.x
  const int nt = (int)blockDim.x;
  const int rpp = NX <= nt ? nt / NX : 1;
  const int c_step = NX <= nt ? NX : nt;
  const int jl0 = NX <= nt ? (int)threadIdx.x / NX : 0;
  const int ic0 = NX <= nt ? (int)threadIdx.x - jl0 * NX : (int)threadIdx.x;
  const bool walker = jl0 < rpp;
#define FGP_FOR_LOCAL(JL, I) \
  if (walker)                \
    for (int JL = jl0; JL < nrow; JL += rpp) \
      for (int I = ic0; I < NX; I += c_step)
  FGP_FOR_LOCAL(jl_, i_) {
    const int t = jl_ * NX + i_;
    int f = j0 * NX + t;
    double bv;
    if (nonneg) bv = ((1.0 * (-P.lambda_l1 / c)) + d[f] * (1.0 / c)) + z[f];
    else bv = d[f] * (1.0 / c) + z[f];
    BB[t] = (T)bv;
    PP[t] = 0;
    QQ[t] = 0;
    RR[t] = 0;
    SS[t] = 0;
  }
  const T alpha1 = (T)(-lam_tv);
  const T alpha3 = (T)(1.0 / (8 * lam_tv));
  const T eta = (T)lam_l1;
  auto prox = [&](T v, int f) -> T {
    if (nonneg) {
      if (box && box[f] == 0.0f) return 0;
      return v < 0 ? T(0) : v;
    }
    if (box) {
      if (box[f] == 0.0f || (v < eta && v > -eta)) return 0;
      return v >= eta ? v - eta : v + eta;
    }
    if (v >= eta) return v - eta;
    if (v <= -eta) return v + eta;
    return 0;
  };
  // Lpq of (p, q) at local element t (global row j, column i)
  auto lpq = [&](const T* p, const T* q, const T* q_above, int t, int i, int j) -> T {
    T v = 0;
    if (i >= 1) v -= p[t - 1];
    if (i < NX - 1) v += p[t];
    if (j >= 1) v -= (t >= NX ? q[t - NX] : q_above[i]);
    if (j < NY - 1) v += q[t];
    return v;
  };
  cluster.sync();
  for (int it = 0; it <= a.iters; ++it) {
    const bool last = it == a.iters;
    // read before the barriers, which leave nothing of them in the cache
    const T beta1 = last ? T(0) : (T)betas[2 * it], beta2 = last ? T(0) : (T)betas[2 * it + 1];
    const T* pr = last ? PP : RR;
    const T* qs = last ? QQ : SS;
    // phase A
    {
      const T* qa = (j0 >= 1 && nrow > 0) ? peer(const_cast<T*>(qs), rank - 1) + (size_t)(rpc - 1) * NX : nullptr;
      FGP_FOR_LOCAL(jl, i) {
        const int t = jl * NX + i;
        int j = j0 + jl;
        T l = lpq(pr, qs, qa, t, i, j);
        T v = l * alpha1 + BB[t];
        v = prox(v, j * NX + i);
        if (last) a.xnew[(size_t)b * a.xstride + (size_t)j * NX + i] = (double)v;
        else XV[t] = v;
      }
    }
    if (last) {
      cluster.sync();  // peers may still be reading this CTA's q slab
      break;
    }
    cluster.sync();
    // phase B
    {
      const T* xb = (j1 < NY && nrow > 0 && rank + 1 < csize) ? peer(XV, rank + 1) : nullptr;
      FGP_FOR_LOCAL(jl, i) {
        const int t = jl * NX + i;
        int j = j0 + jl;
        T xv = XV[t];
        bool hp = i < NX - 1, hq = j < NY - 1;
        T rp = 0, sq = 0;
        if (hp) rp = RR[t] + alpha3 * (xv - XV[t + 1]);
        if (hq) {
          T below = (jl + 1 < nrow) ? XV[t + NX] : xb[i];
          sq = SS[t] + alpha3 * (xv - below);
        }
        T np, nq;
        fgp_project<T>(hp, hq, rp, sq, np, nq);
        if (hp) {
          RR[t] = fma(np, beta1, beta2 * PP[t]);
          PP[t] = np;
        }
        if (hq) {
          SS[t] = fma(nq, beta1, beta2 * QQ[t]);
          QQ[t] = nq;
        }
      }
    }
    cluster.sync();
  }
}
#undef FGP_FOR_LOCAL

// ---------------------------------------------------------------------------
// The same iteration with the dual variables in registers, for images whose
// slab rows fit a CTA's threads.  A thread owns NR consecutive rows of one
// column; shared memory carries only what neighbours need (the fast duals r, s
// and the image x: 7 accesses a pixel, 18 with all six arrays there), and one
// cluster barrier an iteration suffices: a CTA forms the image row below its
// slab itself, from that row's r and s, and every CTA pushes its first r, s row
// and its last s row into its neighbours' halo buffers (two sets, by parity)
// when it updates them.  Arithmetic and its order per pixel are k_fgp's, so
// both give the same bits.
//
// Bound by the chain of an iteration (barrier, shared-memory hops, the FP64
// root) with few problems and by the FP64 / FP32 pipes with many.  Measured on
// B200, 50 iterations, us (k_fgp before -> here, NR = 1, 16 CTAs a problem):
// one problem of 64 x 64 FP64 101 -> 55, 128 x 128 219 -> 73 (FP32 189 -> 74);
// 13 of 96 x 96 FP32 166 -> 105 (NR = 2).
// ---------------------------------------------------------------------------
constexpr int kFgpThreads = 1024;

template <typename T> size_t fgp_reg_smem(int rows, int NX) { return sizeof(T) * (size_t)(3 * rows + 7) * NX; }

template <typename T, int NR>
__global__ void __launch_bounds__(kFgpThreads, 1) k_fgp_reg(FgpArgs a, const double* __restrict__ betas) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int b = blockIdx.y;
  const ProbState& S = a.st[b];
  // uniform over the cluster (same problem): safe to return before barriers
  if (!gate_ok(S, kGateTrial)) return;
  const ProbParams P = a.prm[b];
  const int NX = a.NX, NY = a.NY, rpc = a.rows_per_cta;
  const int j0 = rank * rpc;
  const int j1 = min(NY, j0 + rpc);
  const int nrow = max(0, j1 - j0);
  T* RR = reinterpret_cast<T*>(smem_raw);   // [rpc][NX]
  T* SS = RR + (size_t)rpc * NX;            // [rpc][NX]
  T* XX = SS + (size_t)rpc * NX;            // [rpc + 1][NX]
  T* HS = XX + (size_t)(rpc + 1) * NX;      // s of the row above, [2][NX]
  T* HR = HS + 2 * NX;                      // r of the row below, [2][NX]
  T* HB = HR + 2 * NX;                      // s of the row below, [2][NX]
  const double c = S.c;
  const double lam_tv = P.lambda_tv / c;
  const double lam_l1 = P.lambda_l1 / c;
  const bool nonneg = P.nonneg == 1;
  const float* box = P.box_flag == 1 ? a.box : nullptr;
  const double* z = a.z + (size_t)b * a.xstride;
  const double* d = a.dfdx + (size_t)b * a.xstride;
  auto rhs = [&](int f) -> T {
    double bv;
    if (nonneg) bv = ((1.0 * (-P.lambda_l1 / c)) + d[f] * (1.0 / c)) + z[f];
    else bv = d[f] * (1.0 / c) + z[f];
    return (T)bv;
  };
  const T alpha1 = (T)(-lam_tv);
  const T alpha3 = (T)(1.0 / (8 * lam_tv));
  const T eta = (T)lam_l1;
  auto prox = [&](T v, int f) -> T {
    if (nonneg) {
      if (box && box[f] == 0.0f) return 0;
      return v < 0 ? T(0) : v;
    }
    if (box) {
      if (box[f] == 0.0f || (v < eta && v > -eta)) return 0;
      return v >= eta ? v - eta : v + eta;
    }
    if (v >= eta) return v - eta;
    if (v <= -eta) return v + eta;
    return 0;
  };
  // thread -> column i, rows jl0 .. jl0 + NR - 1 of the slab
  const int grp = (int)threadIdx.x / NX, i = (int)threadIdx.x - grp * NX;
  const int jl0 = grp * NR;
  const int mine = max(0, min(NR, nrow - jl0));
  // the thread of the slab's last row also forms the row below it
  const bool below = j1 < NY && mine > 0 && jl0 + mine == nrow;
  T p[NR], q[NR], r[NR], s[NR], bb[NR], x[NR];
#pragma unroll
  for (int k = 0; k < NR; ++k) {
    p[k] = q[k] = r[k] = s[k] = x[k] = 0;
    bb[k] = k < mine ? rhs((j0 + jl0 + k) * NX + i) : T(0);
    if (k < mine) RR[(jl0 + k) * NX + i] = SS[(jl0 + k) * NX + i] = 0;
  }
  const T bbelow = below ? rhs(j1 * NX + i) : T(0);
  if (grp == 0)
    for (int h = 0; h < 2; ++h) HS[h * NX + i] = HR[h * NX + i] = HB[h * NX + i] = 0;
  // one pixel of b - lambda_tv Lpq(r, s), as k_fgp forms it
  auto image = [&](T left, T here, T above, T self, T bv, int j) -> T {
    T v = 0;
    if (i >= 1) v -= left;
    if (i < NX - 1) v += here;
    if (j >= 1) v -= above;
    if (j < NY - 1) v += self;
    T w = v * alpha1 + bv;
    return prox(w, j * NX + i);
  };
  cluster.sync();
  for (int it = 0; it <= a.iters; ++it) {
    const bool last = it == a.iters;
    const int par = it & 1;
    // phase A (with p, q in r, s after the last update)
#pragma unroll
    for (int k = 0; k < NR; ++k)
      if (k < mine) {
        const int jl = jl0 + k, t = jl * NX + i, j = j0 + jl;
        const T left = i >= 1 ? RR[t - 1] : T(0);
        const T above = k > 0 ? s[k > 0 ? k - 1 : 0] : jl > 0 ? SS[t - NX] : HS[par * NX + i];
        x[k] = image(left, r[k], above, s[k], bb[k], j);
        if (last) a.xnew[(size_t)b * a.xstride + (size_t)j * NX + i] = (double)x[k];
        else XX[t] = x[k];
      }
    if (last) break;
    T xb = 0;  // image row below the slab
    if (below) {
      const T left = i >= 1 ? HR[par * NX + i - 1] : T(0);
      T above = 0;
#pragma unroll
      for (int k = 0; k < NR; ++k)
        if (k == mine - 1) above = s[k];
      xb = image(left, HR[par * NX + i], above, HB[par * NX + i], bbelow, j1);
    }
    __syncthreads();
    const T beta1 = (T)betas[2 * it];
    const T beta2 = (T)betas[2 * it + 1];
    const bool lead = it + 1 == a.iters;  // the next phase A is the last one: hand on p, q
    T* up = rank > 0 ? cluster.map_shared_rank(HR, rank - 1) : nullptr;        // its row below is my first
    T* down = j1 < NY ? cluster.map_shared_rank(HS, rank + 1) : nullptr;       // its row above is my last
    // phase B
#pragma unroll
    for (int k = 0; k < NR; ++k)
      if (k < mine) {
        const int jl = jl0 + k, t = jl * NX + i, j = j0 + jl;
        const bool hp = i < NX - 1, hq = j < NY - 1;
        T rp = 0, sq = 0;
        if (hp) rp = r[k] + alpha3 * (x[k] - XX[t + 1]);
        if (hq) {
          const T xd = jl + 1 == nrow ? xb : k + 1 < NR ? x[k + 1 < NR ? k + 1 : k] : XX[t + NX];
          sq = s[k] + alpha3 * (x[k] - xd);
        }
        T np, nq;
        fgp_project<T>(hp, hq, rp, sq, np, nq);
        if (hp) {
          r[k] = fma(np, beta1, beta2 * p[k]);
          p[k] = np;
        }
        if (hq) {
          s[k] = fma(nq, beta1, beta2 * q[k]);
          q[k] = nq;
        }
        if (lead) {
          r[k] = p[k];
          s[k] = q[k];
        }
        RR[t] = r[k];
        SS[t] = s[k];
        if (jl == 0 && up) {
          up[(par ^ 1) * NX + i] = r[k];
          up[2 * NX + (par ^ 1) * NX + i] = s[k];
        }
        if (jl + 1 == nrow && down) down[(par ^ 1) * NX + i] = s[k];
      }
    cluster.sync();
  }
}


}  // namespace mf
