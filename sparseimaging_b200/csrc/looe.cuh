// Approximate leave-one-out error (LOOE) of DFT solutions on the GPU.
//
// The reference's c/looe_lib.c (compute_LOOE_L1 :190-226, compute_LOOE_L1_TSV
// :275-309, compute_LOOE_core :112-171; its call in c/mfista_dft_lib.c:506-529
// is commented out and its makefile does not build the file) scores a
// solution x of the DFT problem by
//   S = {j : |x_j| > 0},  A_S = A[:, S],
//   H = A_S^T A_S (+ lambda_tsv d2(j) on the diagonal, d2 = 8 / 6 / 4 inside /
//       on an edge / on a corner of the NX grid, d2_TSV :228-245),
//   d_i = (A_S H^-1 A_S^T)_ii,  t_i = (y - A x)_i / (1 - d_i),  s_i = t_i^2 / 2,
//   LOOE_m = mean s,  LOOE_std = sqrt(sum s^2 / (M-1) - LOOE_m^2 M / (M-1)),
// and reports a Hessian that is not positive definite (dposv info > 0).
//
// Here, all in FP64, per solution:
//   H = A_S^T A_S, lower tiles, by matrix products over the active columns
//   where they lie (dgemm_mma.cuh; K split so that the tiles fill the GPU);
//   blocked right-looking Cholesky H = L L^T in 64-wide panels: the diagonal
//   block and the inverse W_k of its factor in one CTA, the panel below as a
//   product with W_k^T, the trailing matrix by products;
//   Y = A_S L^-T by rows: a CTA takes 64 rows through all panels,
//   Y_k = (Z_k - sum_{j<k} Y_j L_kj^T) W_k^T, so that row i of Y is
//   (L^-1 a_i)^T and d_i = |row i|^2 (one triangular solve instead of the
//   reference's two: the same quantity, other rounding);
//   the residual, the t_i and the two sums with fixed-order reductions.
// A non-positive pivot sets an info word that every later kernel of the
// solution checks at entry.
//
// With one thread per row for the triangular solves (53 % of the time), a
// barrier per pivot, column and update in the diagonal block (14 %) and scalar
// 4 x 4 sums in the products (29 %, 13 TFLOP/s), a solution of 1261 active
// pixels, M = 8000, took 9.9 ms on B200; here 2.2 ms: the triangular solves
// 820 us (12.7 GFLOP, 125 CTAs), the diagonal blocks 20 x 27 us (a chain of
// pivots each), the Gram product 486 us, trailing updates 19 x 8 us, panels
// 19 x 7 us.  A call with three solutions: 32 ms -> 8.9 ms.
#pragma once

#include "column_runs.h"
#include "dgemm_mma.cuh"
#include "looe_rule.h"
#include "solver.cuh"

namespace mf {
namespace looe {

constexpr int kPanel = 64;  // Cholesky / triangular-solve block width (the products' tile)
constexpr int kSplitR = 16;  // column ranges of the residual's partial sums
static_assert(kPanel == dg::kT, "panels are tiles of the products");

// tile (ti, tj), ti >= tj, of the e-th lower tile in row order
__device__ __forceinline__ void lower_tile(int e, int& ti, int& tj) {
  ti = (int)((sqrtf(8.f * (float)e + 1.f) - 1.f) * 0.5f);
  while ((ti + 1) * (ti + 2) / 2 <= e) ++ti;
  while (ti * (ti + 1) / 2 > e) --ti;
  tj = e - ti * (ti + 1) / 2;
}

// lower tiles of A_S^T A_S over the K range of split blockIdx.y: split 0 into H,
// split q > 0 into part[q - 1], n_s x n_s each; grid (lower tiles, splits)
__global__ void __launch_bounds__(128, 3) k_looe_gram(const double* __restrict__ A, int M, const int* __restrict__ S,
                                                      int ns, int kchunk, double* __restrict__ H0, double* __restrict__ part) {
  extern __shared__ __align__(16) double looe_smem[];
  int ti, tj;
  lower_tile(blockIdx.x, ti, tj);
  const bool vec = (M & 1) == 0;
  dg::Operand<true> X(A, M, ti * kPanel, ns, vec, S), Y(A, M, tj * kPanel, ns, vec, S);
  dg::Acc acc;
  dg::clear(acc);
  const int k0 = blockIdx.y * kchunk;
  dg::tile_product_nb<8>(X, Y, k0, min(M, k0 + kchunk), looe_smem, acc);
  double* H = blockIdx.y ? part + (size_t)(blockIdx.y - 1) * ns * ns : H0;
  dg::each(acc, [&](int r, int c, double v) {
    const int i = ti * kPanel + r, j = tj * kPanel + c;
    if (i < ns && j < ns) H[(size_t)i + (size_t)j * ns] = v;
  });
}

// H += the splits behind the first (in order), lower triangle, plus lambda_tsv
// d2(S_j) on the diagonal (TSV form); grid: ns columns of cdiv(ns, blockDim.x) CTAs each,
// in x (y ends at 65535, and there may be more columns)
__global__ void k_looe_gram_sum(const double* __restrict__ part, int nsplit, double* __restrict__ H,
                                const int* __restrict__ S, int ns, int nx, double lam) {
  const int nb = (ns + (int)blockDim.x - 1) / (int)blockDim.x;
  const int j = blockIdx.x / nb, i = (blockIdx.x - j * nb) * blockDim.x + threadIdx.x;
  if (i >= ns || i < j) return;
  const size_t e = (size_t)i + (size_t)j * ns;
  double h = H[e];
  for (int q = 0; q < nsplit - 1; ++q) h += part[(size_t)q * ns * ns + e];
  if (i == j && lam != 0.0) {
    const int pix = S[j], r = pix % nx, c = pix / nx;
    const bool ri = r > 0 && r < nx - 1, ci = c > 0 && c < nx - 1;
    h += lam * (ri ? (ci ? 8.0 : 6.0) : (ci ? 6.0 : 4.0));
  }
  H[e] = h;
}

// partial sums of (A x)_i over a range of the active columns: part[split][M]
__global__ void k_looe_ax(const double* __restrict__ A, int M, const int* __restrict__ S, const double* __restrict__ xs,
                          int ns, double* __restrict__ part) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= M) return;
  const int per = (ns + kSplitR - 1) / kSplitR;
  const int j0 = blockIdx.y * per, j1 = min(ns, j0 + per);
  double s = 0.0;
#pragma unroll 8
  for (int j = j0; j < j1; ++j) s = fma(A[(size_t)S[j] * M + i], xs[j], s);
  part[(size_t)blockIdx.y * M + i] = s;
}

// Cholesky of the nb x nb diagonal block at (k0, k0) (lower triangle in and
// out) and the inverse of the factor, W [64][64] (zeros above its diagonal and
// beyond nb); info = k0 + j + 1 at a pivot that is not > 0.  One CTA, the
// block and the inverse in registers (a thread holds rows tx + 16 r and
// columns ty + 16 c of both); a step broadcasts pivot column and inverse row
// through shared memory, eliminates without square roots (L = U D^1/2) and
// costs one barrier.
__global__ void __launch_bounds__(256) k_looe_chol_diag(double* __restrict__ H, int ld, int k0, int nb,
                                                        double* __restrict__ W, int* __restrict__ info) {
  if (*info) return;
  __shared__ double s_col[2][kPanel], s_row[2][kPanel], s_d[kPanel];
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  double* blk = H + (size_t)k0 + (size_t)k0 * ld;
  double a[4][4], w[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = tx + 16 * r, j = ty + 16 * c;
      const double one = i == j ? 1.0 : 0.0;
      a[r][c] = (i < nb && j < nb) ? (i >= j ? blk[(size_t)i + (size_t)j * ld] : blk[(size_t)j + (size_t)i * ld]) : one;
      w[r][c] = one;
    }
#pragma unroll
  for (int jc = 0; jc < 4; ++jc)
    for (int jj = 0; jj < 16; ++jj) {
      const int j = 16 * jc + jj, buf = j & 1;
      if (ty == jj) {
#pragma unroll
        for (int r = 0; r < 4; ++r) s_col[buf][tx + 16 * r] = a[r][jc];
      }
      if (tx == jj) {
#pragma unroll
        for (int c = 0; c < 4; ++c) s_row[buf][ty + 16 * c] = w[jc][c];
      }
      __syncthreads();
      const double d = s_col[buf][j];
      if (!(d > 0.0)) {  // the same for every thread
        if (t == 0) *info = k0 + j + 1;
        return;
      }
      if (t == 0) s_d[j] = d;
      const double rd = 1.0 / d;
      double cj[4], wj[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int k = ty + 16 * c;
        cj[c] = k > j ? s_col[buf][k] : 0.0;
        wj[c] = s_row[buf][k];
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int i = tx + 16 * r;
        const double l = i > j ? s_col[buf][i] * rd : 0.0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          a[r][c] = fma(-l, cj[c], a[r][c]);
          w[r][c] = fma(-l, wj[c], w[r][c]);
        }
      }
    }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = tx + 16 * r, j = ty + 16 * c;
      const bool in = i < nb && j < nb && i >= j;
      if (in) blk[(size_t)i + (size_t)j * ld] = i == j ? sqrt(s_d[j]) : a[r][c] / sqrt(s_d[j]);
      W[i * kPanel + j] = in ? w[r][c] / sqrt(s_d[i]) : 0.0;
    }
}

// the panel below a factored diagonal block: H[k1 + i][k0 ..] := H[..] W^T, in
// place (a CTA reads its 64 rows whole before it writes them)
__global__ void __launch_bounds__(128, 3) k_looe_panel(double* __restrict__ H, int ld, int k0, int nb,
                                                       const double* __restrict__ W, const int* __restrict__ info) {
  if (*info) return;
  extern __shared__ __align__(16) double looe_smem[];
  const int i0 = blockIdx.x * kPanel, rows = ld - (k0 + nb);
  double* P = H + (size_t)(k0 + nb) + (size_t)k0 * ld;
  dg::Operand<false> X(P, ld, i0, rows, (ld & 1) == 0 && ((k0 + nb) & 1) == 0);
  dg::Operand<true> Y(W, kPanel, 0, nb, true);
  dg::Acc acc;
  dg::clear(acc);
  dg::tile_product_nb<8>(X, Y, 0, nb, looe_smem, acc);
  dg::each(acc, [&](int r, int c, double v) {
    if (i0 + r < rows && c < nb) P[(size_t)(i0 + r) + (size_t)c * ld] = v;
  });
}

// trailing matrix H[k1.., k1..] -= P P^T, lower tiles, P the panel below the
// block at k0; grid: the lower tiles
__global__ void __launch_bounds__(256, 2) k_looe_trail(double* __restrict__ H, int ld, int k0, int nb,
                                                       const int* __restrict__ info) {
  if (*info) return;
  extern __shared__ __align__(16) double looe_smem[];
  int ti, tj;
  lower_tile(blockIdx.x, ti, tj);
  const int k1 = k0 + nb, rows = ld - k1;
  const double* P = H + (size_t)k1 + (size_t)k0 * ld;
  const bool vec = (ld & 1) == 0 && (k1 & 1) == 0;
  dg::Operand<false, 256> X(P, ld, ti * kPanel, rows, vec), Y(P, ld, tj * kPanel, rows, vec);
  dg::AccNb<4> acc, old;
  dg::clear(acc);
  double* C = H + (size_t)k1 + (size_t)k1 * ld;
  auto at = [&](int r, int c) { return (size_t)(ti * kPanel + r) + (size_t)(tj * kPanel + c) * ld; };
  auto in = [&](int r, int c) { return ti * kPanel + r < rows && tj * kPanel + c < rows; };
  dg::each_of<4>(old, [&](int r, int c, double& v) { v = in(r, c) ? C[at(r, c)] : 0.0; });  // in flight behind the product
  dg::tile_product_nb<4>(X, Y, 0, nb, looe_smem, acc);
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) old[m][j][h] -= acc[m][j][h];
  dg::each_of<4>(old, [&](int r, int c, double v) {
    if (in(r, c)) C[at(r, c)] = v;
  });
}

// Y = A_S L^-T and the leverages d_i = |Y_i|^2 of 64 rows per CTA, panel by
// panel (each needs the CTA's own earlier panels only).  W: [panel][64][64].
constexpr int kRowLd = 68;  // row stride of the staged panel and of W
constexpr size_t kRowsSmem = dg::kSmem + sizeof(double) * kPanel * kRowLd;
static_assert(sizeof(double) * kPanel * kRowLd <= dg::kSmem, "a panel fits the products' stages");
__global__ void __launch_bounds__(256, 2) k_looe_rows(const double* __restrict__ A, int M, const int* __restrict__ S, int ns,
                                                   const double* __restrict__ H, const double* __restrict__ Wall,
                                                   double* __restrict__ Y, double* __restrict__ dlev,
                                                   const int* __restrict__ info) {
  if (*info) return;
  extern __shared__ __align__(16) double looe_smem[];
  double* s_t = looe_smem;                                  // [64][68], over the stages
  double* s_w = looe_smem + dg::kSmem / sizeof(double);     // [64][68]
  const int i0 = blockIdx.x * kPanel;
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) & 3, half = threadIdx.x >> 7, g = lane >> 2, t = lane & 3;
  double d[2] = {0.0, 0.0};
  const bool vy = (M & 1) == 0, vh = (ns & 1) == 0;
  for (int k0 = 0; k0 < ns; k0 += kPanel) {
    const int nb = min(kPanel, ns - k0);
    const double* W = Wall + (size_t)(k0 / kPanel) * kPanel * kPanel;
    for (int e = threadIdx.x; e < kPanel * kPanel / 2; e += 256)
      dg::copy2(s_w + (e >> 5) * kRowLd + 2 * (e & 31), W + 2 * e, 2, true);
    cp_async_commit();
    dg::AccNb<4> acc, rhs;
    dg::clear(acc);
    dg::each_of<4>(rhs, [&](int r, int c, double& v) {  // in flight behind the product
      v = (i0 + r < M && c < nb) ? A[(size_t)S[k0 + c] * M + i0 + r] : 0.0;
    });
    dg::Operand<false, 256> X(Y, M, i0, M, vy), L(H, ns, k0, ns, vh);
    dg::tile_product_nb<4>(X, L, 0, k0, looe_smem, acc);
    // the right-hand side into shared memory (beyond nb the product is not zero)
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) rhs[m][j][h] -= acc[m][j][h];
    dg::each_of<4>(rhs, [&](int r, int c, double v) {
      s_t[r * kRowLd + c] = (i0 + r < M && c < nb) ? v : 0.0;
    });
    cp_async_wait<0>();
    __syncthreads();
    dg::clear(acc);
#pragma unroll 2
    for (int kk = 0; kk < kPanel; kk += 4) {
      double a[2], b[4];
#pragma unroll
      for (int m = 0; m < 2; ++m) a[m] = s_t[(16 * warp + 8 * m + g) * kRowLd + kk + t];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = s_w[(32 * half + 8 * j + g) * kRowLd + kk + t];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        dmma_884(acc[0][j], a[0], b[j]);
        dmma_884(acc[1][j], a[1], b[j]);
      }
    }
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int i = i0 + 16 * warp + 8 * m + g, c = 32 * half + 8 * j + 2 * t + h;
          const double v = acc[m][j][h];
          d[m] = fma(v, v, d[m]);  // zero beyond nb and M
          if (i < M && c < nb) Y[(size_t)i + (size_t)(k0 + c) * M] = v;
        }
    __syncthreads();  // Y_k is read, and s_t and s_w are written, by the next panel
  }
  __shared__ double s_half[kPanel];
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    d[m] += __shfl_xor_sync(0xffffffffu, d[m], 1);
    d[m] += __shfl_xor_sync(0xffffffffu, d[m], 2);
    if (t == 0 && half) s_half[16 * warp + 8 * m + g] = d[m];
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int i = i0 + 16 * warp + 8 * m + g;
    if (t == 0 && !half && i < M) dlev[i] = d[m] + s_half[16 * warp + 8 * m + g];
  }
}

// per row i: t = (y - A x)_i / (1 - d_i), s = t^2 / 2; per-CTA partial sums of
// s and s^2
__global__ void __launch_bounds__(256) k_looe_terms(const double* __restrict__ y, const double* __restrict__ ax, int nax,
                                                    const double* __restrict__ dlev, int M, double* __restrict__ part,
                                                    const int* __restrict__ info) {
  __shared__ double sh[2][256];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double s = 0.0, s2 = 0.0;
  if (!*info && i < M) {
    double v = 0.0;
    for (int q = 0; q < nax; ++q) v += ax[(size_t)q * M + i];
    const double tt = (y[i] - v) / (1.0 - (nax > 0 ? dlev[i] : 0.0));
    s = tt * tt / 2;
    s2 = s * s;
  }
  sh[0][threadIdx.x] = s;
  sh[1][threadIdx.x] = s2;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      sh[0][threadIdx.x] += sh[0][threadIdx.x + o];
      sh[1][threadIdx.x] += sh[1][threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = sh[0][0];
    part[2 * blockIdx.x + 1] = sh[1][0];
  }
}

// out = (looe_m, looe_std, positive) from the partials, in block order
__global__ void k_looe_final(const double* __restrict__ part, int nblk, int M, const int* __restrict__ info,
                             double* __restrict__ out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  if (*info) {
    out[0] = 0.0;
    out[1] = 0.0;
    out[2] = 0.0;
    return;
  }
  double s = 0.0, s2 = 0.0;
  for (int b = 0; b < nblk; ++b) {
    s += part[2 * b];
    s2 += part[2 * b + 1];
  }
  const double m = s / M;
  const double var = s2 / (M - 1.0) - m * m * M / (M - 1.0);
  out[0] = m;
  out[1] = sqrt(var);
  out[2] = 1.0;
}

// Host driver: LOOE of B solutions X [B][N] of the DFT problem (y [M], A
// column-major M x N); lambda_tsv per solution (null: 0).  Kernels per
// solution: 6 + 3 ceil(n_s / 64).
//
// Only the columns of A that some solution uses go to the device, in runs
// (column_runs.h).
// Solutions run on up to kLanes streams (looe_rule.h), each with its own scratch: one
// solution's factorisation is a chain of small kernels (840 of 2190 us at 1261
// active pixels) and its other kernels leave SMs idle, which the next one's
// fill.  Lanes beyond the first are taken only while all scratch stays within
// kLaneBytes, and given up when their memory cannot be had; the results do
// not depend on them.
struct Looe {
  static constexpr int kLanes = 4;
  static constexpr size_t kLaneBytes = (size_t)1 << 30;

  struct Lane {
    cudaStream_t s = nullptr;
    double* mem = nullptr;   // its part of d_lanes
    std::vector<int> idx;    // of the solution in flight: pixels, then columns of the device's A
    std::vector<double> xs;  // its active values
    ~Lane() {
      if (s) cudaStreamDestroy(s);
    }
  };
  // a lane's scratch, in doubles from its start
  struct Layout {
    size_t xs, ax, Y, H, Hs, W, lev, part, out, info, idx, total;
  };

  const double* X;
  int M, N, NX, B;
  int most = 0;          // active pixels of a solution at most
  DevMem d_A, d_y, d_lanes;
  std::vector<int> col;  // pixel -> column of the device's A
  std::vector<std::unique_ptr<Lane>> lanes;
  int sms = 148;

  Looe(const double* y, const double* A, int M_, int N_, int NX_, const double* X_, int B_)
      : X(X_), M(M_), N(N_), NX(NX_), B(B_) {
    int dev = 0;
    MF_CK(cudaGetDevice(&dev));
    MF_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    std::vector<char> used(N, 0);
    for (int b = 0; b < B; ++b) {
      int n = 0;
      for (int j = 0; j < N; ++j)
        if (fabs(X[(size_t)b * N + j]) > 0) {
          used[j] = 1;
          ++n;
        }
      most = std::max(most, n);
    }
    const std::vector<ColumnRun> runs = column_runs(used, sizeof(double) * M);
    col.assign(N, 0);
    int nc = 0;
    for (const ColumnRun& r : runs)
      for (int j = r.first; j < r.last; ++j) col[j] = nc++;
    d_A.alloc(sizeof(double) * (size_t)M * nc);
    for (const ColumnRun& r : runs)
      MF_CK(cudaMemcpy(d_A.as<double>() + (size_t)col[r.first] * M, A + (size_t)r.first * M,
                       sizeof(double) * (size_t)(r.last - r.first) * M, cudaMemcpyHostToDevice));
    d_y.upload(y, (size_t)M);
    MF_CK(cudaStreamSynchronize(nullptr));  // the lanes' streams do not wait for the copies' last part
    set_smem(k_looe_gram, dg::kSmem);
    set_smem(k_looe_panel, dg::kSmem);
    set_smem(k_looe_trail, dg::kSmem);
    set_smem(k_looe_rows, kRowsSmem);
    // one allocation for all lanes: each of its own cost 0.1 ms, and 0.7 ms from a few MB on
    const size_t each = layout(most).total, bytes = sizeof(double) * each;
    int n = looe_lanes(B, cdiv(most, kPanel), M, kLanes);
    while (n > 1 && n * bytes > kLaneBytes) --n;
    for (; n > 1; --n) {
      if (cudaMalloc(&d_lanes.p, n * bytes) == cudaSuccess) break;
      cudaGetLastError();
    }
    if (n > 1) d_lanes.bytes = n * bytes;
    else d_lanes.alloc(bytes);
    for (int i = 0; i < n; ++i) {
      std::unique_ptr<Lane> l(new Lane);
      l->mem = d_lanes.as<double>() + i * each;
      MF_CK(cudaStreamCreateWithFlags(&l->s, cudaStreamNonBlocking));
      lanes.push_back(std::move(l));
    }
  }

  // K splits of the lower tiles: the fewest (at most 4) whose CTAs spread over
  // the SMs with the least idle time in the last round
  int gram_splits(int tiles) const {
    int best = 1;
    double load = 0.0;
    for (int q = 1; q <= 4 && M / q >= 512; ++q) {
      const double x = (double)tiles * q / sms, l = x / ceil(x);
      if (l > load + 0.05) {
        load = l;
        best = q;
      }
    }
    return best;
  }
  static int tiles_of(int ns) {
    const int np = cdiv(ns, kPanel);
    return np * (np + 1) / 2;
  }

  // room for every solution of at most ns active pixels
  Layout layout(int ns) const {
    Layout l;
    size_t at = 0;
    auto take = [&](size_t n) {
      const size_t p = at;
      at += (n + 31) & ~(size_t)31;  // 256 bytes
      return p;
    };
    int splits = 1;
    size_t hs = 0;
    // splits behind the first: none above 62 panels (3968 pixels) on 148 SMs, so
    // they take at most 0.4 GB beside H, which is held once.  (A smaller
    // solution may have more splits.)
    for (int n = 1, np = cdiv(ns, kPanel); n <= np; ++n) {
      const size_t m = std::min((size_t)n * kPanel, (size_t)ns);
      splits = gram_splits(n * (n + 1) / 2);
      hs = std::max(hs, (size_t)(splits - 1) * m * m);
    }
    l.xs = take(ns);
    l.ax = take(kSplitR * (size_t)M);
    l.Y = take((size_t)M * ns);
    l.H = take((size_t)ns * ns);
    l.Hs = take(hs);
    l.W = take((size_t)cdiv(ns, kPanel) * kPanel * kPanel);
    l.lev = take(M);
    l.part = take(2 * (size_t)cdiv(M, 256));
    l.out = take(3);
    l.info = take(1);
    l.idx = take(ns);  // 2 ns ints
    l.total = at;
    return l;
  }

  // the kernels of solution b on a lane; its results are in the lane's out
  void launch(Lane& L, int b, double lam_tsv) {
    const double* x = X + (size_t)b * N;
    cudaStream_t s = L.s;
    L.idx.clear();
    L.xs.clear();
    for (int j = 0; j < N; ++j)
      if (fabs(x[j]) > 0) {
        L.idx.push_back(j);
        L.xs.push_back(x[j]);
      }
    const int ns = (int)L.xs.size();
    for (int q = 0; q < ns; ++q) L.idx.push_back(col[L.idx[q]]);
    const int np = cdiv(ns, kPanel), tiles = tiles_of(ns);
    const Layout l = layout(most);
    double* m = L.mem;
    int* info = reinterpret_cast<int*>(m + l.info);
    int *pix = reinterpret_cast<int*>(m + l.idx), *S = pix + ns;
    MF_CK(cudaMemsetAsync(info, 0, sizeof(int), s));
    if (ns > 0) {
      const int nsplit = gram_splits(tiles);
      const int kchunk = cdiv(cdiv(M, nsplit), dg::kStep) * dg::kStep;
      MF_CK(cudaMemcpyAsync(pix, L.idx.data(), 2 * sizeof(int) * ns, cudaMemcpyHostToDevice, s));
      MF_CK(cudaMemcpyAsync(m + l.xs, L.xs.data(), sizeof(double) * ns, cudaMemcpyHostToDevice, s));
      double *H = m + l.H, *Hs = m + l.Hs;
      const double* A = d_A.as<double>();
      k_looe_ax<<<dim3(cdiv(M, 256), kSplitR), 256, 0, s>>>(A, M, S, m + l.xs, ns, m + l.ax);
      MF_LAUNCH_CK();
      k_looe_gram<<<dim3(tiles, nsplit), 128, dg::kSmem, s>>>(A, M, S, ns, kchunk, H, Hs);
      MF_LAUNCH_CK();
      if (nsplit > 1 || lam_tsv != 0.0) {
        k_looe_gram_sum<<<(unsigned int)cdiv(ns, 256) * ns, 256, 0, s>>>(Hs, nsplit, H, pix, ns, NX, lam_tsv);
        MF_LAUNCH_CK();
      }
      for (int k0 = 0; k0 < ns; k0 += kPanel) {
        const int nb = std::min(kPanel, ns - k0), nt = cdiv(ns - k0 - nb, kPanel);
        double* W = m + l.W + (size_t)(k0 / kPanel) * kPanel * kPanel;
        k_looe_chol_diag<<<1, 256, 0, s>>>(H, ns, k0, nb, W, info);
        MF_LAUNCH_CK();
        if (nt > 0) {
          k_looe_panel<<<nt, 128, dg::kSmem, s>>>(H, ns, k0, nb, W, info);
          MF_LAUNCH_CK();
          k_looe_trail<<<nt * (nt + 1) / 2, 256, dg::kSmem, s>>>(H, ns, k0, nb, info);
          MF_LAUNCH_CK();
        }
      }
      k_looe_rows<<<cdiv(M, kPanel), 256, kRowsSmem, s>>>(A, M, S, ns, H, m + l.W, m + l.Y, m + l.lev, info);
      MF_LAUNCH_CK();
    }
    const int nblk = cdiv(M, 256);
    k_looe_terms<<<nblk, 256, 0, s>>>(d_y.as<double>(), m + l.ax, ns > 0 ? kSplitR : 0, m + l.lev, M, m + l.part, info);
    MF_LAUNCH_CK();
    k_looe_final<<<1, 32, 0, s>>>(m + l.part, nblk, M, info, m + l.out);
    MF_LAUNCH_CK();
  }

  // f(b, {looe_m, looe_std, positive}) for every solution in order
  template <typename F> void all(const double* lambda_tsv, F f) {
    const int nl = (int)lanes.size();
    const Layout l = layout(most);
    auto finish = [&](int b) {
      Lane& L = *lanes[b % nl];
      double out[3];
      MF_CK(cudaMemcpyAsync(out, L.mem + l.out, sizeof(out), cudaMemcpyDeviceToHost, L.s));
      MF_CK(cudaStreamSynchronize(L.s));
      f(b, out);
    };
    for (int b = 0; b < B; ++b) {
      if (b >= nl) finish(b - nl);  // the lane's solution before
      launch(*lanes[b % nl], b, lambda_tsv ? lambda_tsv[b] : 0.0);
    }
    for (int b = std::max(0, B - nl); b < B; ++b) finish(b);
  }
};

}  // namespace looe
}  // namespace mf
