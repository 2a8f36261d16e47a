// Operator of the DFT variant (c/mfista_dft_lib.c:30-66, :253-278): a dense
// real M x N column-major matrix A.
//   residual  r = y - A z            (calc_yAz, dgemv "N")
//   gradient  A^T r - lambda_tsv d_TSV(z)   (dF_dx, dgemv "T" with beta)
// FP64 GEMV kernels for the plain method: A z is split over column chunks
// (one CTA per 256 rows x chunk, deterministic second pass), A^T r is one
// warp per column with coalesced reads down the column.
#pragma once
#include "common.cuh"
#include "dgemm_mma.cuh"
#include "nufft_ops.cuh"  // dtsv_at / tsv_terms_at

namespace mf {

struct DftGeom {
  const double* A;   // column-major M x N (lda = M), shared by the batch
  const double* y;   // [M]
  int M, N;
  int nchunk, chunk; // column split of A z
  double* az_part;   // [B][nchunk][M]
  double* resid;     // [B][M]
};

__global__ void k_dft_az(DftGeom g, const double* __restrict__ zall, long xstride, const ProbState* __restrict__ st,
                         int gate) {
  int b = blockIdx.z;
  if (!gate_ok(st[b], gate)) return;
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  int c = blockIdx.y;
  int n0 = c * g.chunk, n1 = min(g.N, n0 + g.chunk);
  const double* z = zall + (size_t)b * xstride;
  extern __shared__ double zs[];
  for (int n = n0 + threadIdx.x; n < n1; n += blockDim.x) zs[n - n0] = z[n];
  __syncthreads();
  if (m >= g.M) return;
  double s = 0.0;
  const double* a = g.A + (size_t)n0 * g.M + m;
  for (int n = n0; n < n1; ++n, a += g.M) s += *a * zs[n - n0];
  g.az_part[((size_t)b * g.nchunk + c) * g.M + m] = s;
}

__global__ void k_dft_resid(DftGeom g, const ProbState* __restrict__ st, int gate, Partials part, int qchi,
                            int store) {
  __shared__ double sh[32];
  int b = blockIdx.y;
  if (!gate_ok(st[b], gate)) return;
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  double acc[1] = {0.0};
  if (m < g.M) {
    double s = 0.0;
    for (int c = 0; c < g.nchunk; ++c) s += g.az_part[((size_t)b * g.nchunk + c) * g.M + m];
    double r = g.y[m] - s;
    acc[0] = r * r;
    if (store) g.resid[(size_t)b * g.M + m] = r;
  }
  block_sum<1>(acc, sh);
  if (threadIdx.x == 0) part.at(qchi, b)[blockIdx.x] = acc[0];
}

// dfdx[n] = beta * dTSV(z)[n] + sum_m A[m + n M] r[m]  (beta = -lambda_tsv or 0)
__global__ void k_dft_atr(DftGeom g, double* __restrict__ dall, long xstride, const double* __restrict__ zall,
                          const ProbParams* __restrict__ prm, int tsvNX, int tsvNY, const ProbState* __restrict__ st,
                          int gate, Partials part, int qtsv) {
  __shared__ double sh[32];
  int b = blockIdx.y;
  if (!gate_ok(st[b], gate)) return;
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int n = blockIdx.x * nw + warp;
  const double* r = g.resid + (size_t)b * g.M;
  const ProbParams& pp = prm[b];
  bool fuse = zall != nullptr && pp.lambda_tsv > 0.0;
  double acc[1] = {0.0};
  if (n < g.N) {
    const double* col = g.A + (size_t)n * g.M;
    double s = 0.0;
    for (int m = lane; m < g.M; m += 32) s += col[m] * r[m];
    s = warp_sum(s);
    if (lane == 0) {
      double* d = dall + (size_t)b * xstride;
      if (fuse) {
        const double* z = zall + (size_t)b * xstride;
        d[n] = dtsv_at(z, n, tsvNX, tsvNY) * (-pp.lambda_tsv) + s;
        acc[0] = tsv_terms_at(z, n, tsvNX, tsvNY);
      } else {
        d[n] = s;
      }
    }
  }
  if (qtsv >= 0) {
    block_sum<1>(acc, sh);
    if (threadIdx.x == 0) part.at(qtsv, b)[blockIdx.x] = acc[0];
  }
}

}  // namespace mf

// ===========================================================================
// Batched DFT (B problems share A): A Z and A^T R as FP64 matrix products
// (dgemm_mma.cuh) with split K; a CTA forms a 64 x 64 (rows x problems) tile.
// A tile's problems are the batch's active ones in index order, so a batch
// with few left forms only their columns.  Results are per-K-chunk partials
// summed in a fixed order afterwards: deterministic, and a problem's sums do
// not depend on its place in a tile or on the size of its batch (of two or
// more; one problem has kernels of its own).
//
// A 8000 x 4096, 64 problems on B200: A Z 440 -> 147 us, A^T R 375 -> 169 us;
// with 8 of them left 61 and 77 us
// (4.2 GFLOP: 113 us at the FP64 rate; 40 us for A at the HBM rate).
// ===========================================================================
namespace mf {

constexpr int kGT = dg::kT;     // tile edge (rows and problems)
constexpr int kGK = dg::kStep;  // K chunks are multiples of it

// the chunk-th 64 active problems, in index order; returns their count
// (128 threads)
__device__ __forceinline__ int active_tile(const ProbState* __restrict__ st, int gate, int B, int chunk, int* list) {
  __shared__ int s_cnt[4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lo = chunk * kGT;
  int base_rank = 0;
  for (int base = 0; base < B; base += 128) {
    const int b = base + (int)threadIdx.x;
    const bool on = b < B && gate_ok(st[b], gate);
    const unsigned int bal = __ballot_sync(0xffffffffu, on);
    if (lane == 0) s_cnt[warp] = __popc(bal);
    __syncthreads();
    int r = base_rank + __popc(bal & ((1u << lane) - 1u));
    for (int w = 0; w < 4; ++w) {
      if (w < warp) r += s_cnt[w];
      base_rank += s_cnt[w];
    }
    if (on && r >= lo && r < lo + kGT) list[r - lo] = b;
    __syncthreads();  // s_cnt is rewritten by the next round
  }
  return min(max(base_rank - lo, 0), kGT);
}

// az_part[b][chunk][m] = sum_{n in chunk} A[m + n M] z_b[n]; grid (row tiles,
// chunks, 64-problem tiles), 128 threads, dg::kSmem
__global__ void __launch_bounds__(128, 3) k_dft_az_gemm(DftGeom g, const double* __restrict__ zall, long xstride,
                                                        const ProbState* __restrict__ st, int gate, int B) {
  extern __shared__ __align__(16) double dft_smem[];
  __shared__ int s_list[kGT];
  const int nact = active_tile(st, gate, B, blockIdx.z, s_list);
  if (nact == 0) return;  // no problem of this tile: skip reading A
  const int m0 = blockIdx.x * kGT, c = blockIdx.y;
  const int n0 = c * g.chunk, n1 = min(g.N, n0 + g.chunk);
  const dg::Operand<false> X(g.A, g.M, m0, g.M, (g.M & 1) == 0);
  const dg::Operand<true> Z(zall, (size_t)xstride, 0, nact, (xstride & 1) == 0, s_list);
  dg::Acc acc;
  dg::clear(acc);
  dg::tile_product(X, Z, n0, n1, (nact + 7) >> 3, dft_smem, acc);
  dg::each(acc, [&](int r, int j, double v) {
    if (m0 + r < g.M && j < nact) g.az_part[((size_t)s_list[j] * g.nchunk + c) * g.M + m0 + r] = v;
  });
}

// atr_part[b][chunk][n] = sum_{m in chunk} A[m + n M] r_b[m]
__global__ void __launch_bounds__(128, 3) k_dft_atr_gemm(DftGeom g, double* __restrict__ atr_part, int mchunk,
                                                         int nmchunk, const ProbState* __restrict__ st, int gate,
                                                         int B) {
  extern __shared__ __align__(16) double dft_smem[];
  __shared__ int s_list[kGT];
  const int nact = active_tile(st, gate, B, blockIdx.z, s_list);
  if (nact == 0) return;
  const int nn0 = blockIdx.x * kGT, c = blockIdx.y;
  const int ms = c * mchunk, me = min(g.M, ms + mchunk);
  const bool vec = (g.M & 1) == 0;
  const dg::Operand<true> X(g.A, g.M, nn0, g.N, vec), R(g.resid, g.M, 0, nact, vec, s_list);
  dg::Acc acc;
  dg::clear(acc);
  dg::tile_product(X, R, ms, me, (nact + 7) >> 3, dft_smem, acc);
  dg::each(acc, [&](int r, int j, double v) {
    if (nn0 + r < g.N && j < nact) atr_part[((size_t)s_list[j] * nmchunk + c) * g.N + nn0 + r] = v;
  });
}

// dfdx[n] = beta dTSV(z)[n] + sum_chunks atr_part[b][c][n]
__global__ void k_dft_atr_finish(DftGeom g, const double* __restrict__ atr_part, int nmchunk,
                                 double* __restrict__ dall, long xstride, const double* __restrict__ zall,
                                 const ProbParams* __restrict__ prm, int tsvNX, int tsvNY,
                                 const ProbState* __restrict__ st, int gate) {
  int b = blockIdx.y;
  if (!gate_ok(st[b], gate)) return;
  int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= g.N) return;
  double s = 0.0;
  for (int c = 0; c < nmchunk; ++c) s += atr_part[((size_t)b * nmchunk + c) * g.N + n];
  const ProbParams& pp = prm[b];
  double* d = dall + (size_t)b * xstride;
  if (zall != nullptr && pp.lambda_tsv > 0.0) {
    const double* z = zall + (size_t)b * xstride;
    d[n] = dtsv_at(z, n, tsvNX, tsvNY) * (-pp.lambda_tsv) + s;
  } else {
    d[n] = s;
  }
}

}  // namespace mf

// ===========================================================================
// Split-BF16 tensor-core form (tc::k_gemm_bf16x3) with FP64 defect
// correction: for an anchor x_a (refreshed in FP64 every few outer
// iterations) with ax_a = A x_a, r_a = y - ax_a and g_a = A^T r_a,
//   A v   = ax_a + A (v - x_a)            (tensor-core part: A (v - x_a))
//   A^T r = g_a  + A^T (r - r_a)          (tensor-core part: A^T (r - r_a))
// so the low-precision products only carry the (small) departures from the
// anchor.  Partials arrive per K split as FP32 [nsplit][bpad][rows] and are
// summed in a fixed order in FP64.
// ===========================================================================
namespace mf {

// r = y - (ax_a + sum_s part[s]) ; chi^2 partials; r stored when `store`
__global__ void k_dft_tc_resid(const float* __restrict__ part, int nsplit, int bpad, int rows,
                               const double* __restrict__ axa, DftGeom g, const ProbState* __restrict__ st, int gate,
                               Partials pq, int qchi, int store) {
  __shared__ double sh[32];
  int b = blockIdx.y;
  if (!gate_ok(st[b], gate)) return;
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  double acc[1] = {0.0};
  if (m < g.M) {
    double s = axa[(size_t)b * g.M + m];
    for (int k = 0; k < nsplit; ++k) s += (double)part[((size_t)k * bpad + b) * rows + m];
    double r = g.y[m] - s;
    acc[0] = r * r;
    if (store) g.resid[(size_t)b * g.M + m] = r;
  }
  block_sum<1>(acc, sh);
  if (threadIdx.x == 0 && qchi >= 0) pq.at(qchi, b)[blockIdx.x] = acc[0];
}

// dfdx[n] = beta dTSV(z)[n] + g_a[n] + sum_s part[s][n]   (beta = -lambda_tsv or 0)
__global__ void k_dft_tc_atr_finish(const float* __restrict__ part, int nsplit, int bpad, int rows,
                                    const double* __restrict__ ga, int N, double* __restrict__ dall, long xstride,
                                    const double* __restrict__ zall, const ProbParams* __restrict__ prm, int tsvNX,
                                    int tsvNY, const ProbState* __restrict__ st, int gate) {
  int b = blockIdx.y;
  if (!gate_ok(st[b], gate)) return;
  int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  double s = ga[(size_t)b * N + n];
  for (int k = 0; k < nsplit; ++k) s += (double)part[((size_t)k * bpad + b) * rows + n];
  const ProbParams& pp = prm[b];
  double* d = dall + (size_t)b * xstride;
  if (zall != nullptr && pp.lambda_tsv > 0.0) {
    const double* z = zall + (size_t)b * xstride;
    d[n] = dtsv_at(z, n, tsvNX, tsvNY) * (-pp.lambda_tsv) + s;
  } else {
    d[n] = s;
  }
}

// anchor model from the FP64 GEMM partials: ax_a = sum_c az_part, r_a = y - ax_a
__global__ void k_dft_anchor(DftGeom g, const ProbState* __restrict__ st, int gate, double* __restrict__ axa,
                             double* __restrict__ ra) {
  int b = blockIdx.y;
  if (!gate_ok(st[b], gate)) return;
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= g.M) return;
  double s = 0.0;
  for (int c = 0; c < g.nchunk; ++c) s += g.az_part[((size_t)b * g.nchunk + c) * g.M + m];
  axa[(size_t)b * g.M + m] = s;
  ra[(size_t)b * g.M + m] = g.y[m] - s;
}

}  // namespace mf
