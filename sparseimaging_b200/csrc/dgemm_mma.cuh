// FP64 matrix products on mma.sync m8n8k4.f64: the tile loop shared by the
// batched DFT operator (dft_ops.cuh) and the leave-one-out error (looe.cuh).
//
// A CTA of 128 threads (or 256, below) forms a 64 x 64 tile of X Y^T, X and Y given by rows:
// an operand is stored either with K contiguous (kK) or with its rows
// contiguous (column-major, !kK).  K runs in steps of 16 through a ring of
// three shared-memory stages filled by cp.async (zeros outside the matrices);
// warp w multiplies rows 16 w .. 16 w + 15 with all 64 columns: per 4 of K two
// A and eight B fragments, 2.5 KB of shared memory for 16 products (64 cycles
// of the FP64 pipe).  A scalar loop over the same tiles with 4 x 4 sums a
// thread is bound by its shared-memory and issue slots at 9-13 TFLOP/s of 37.
// Row strides of 20 and 68 doubles put a half warp's 8-byte fragment loads on
// all banks.
#pragma once
#include "nufft_mma.cuh"

namespace mf {
namespace dg {

constexpr int kT = 64;       // tile edge
constexpr int kStep = 16;    // K per stage
constexpr int kStages = 3;
constexpr int kLdK = 20;     // stage row stride, K contiguous: [64][20]
constexpr int kLdM = 68;     // stage row stride, rows contiguous: [16][68]
constexpr int kOperand = kT * kLdK;  // doubles of one operand's stage (the larger of 64 x 20 and 16 x 68)
constexpr size_t kSmem = sizeof(double) * 2 * kStages * kOperand;

// 16 bytes (vec) or twice 8 bytes, the first `n` doubles valid, the others zero
__device__ __forceinline__ void copy2(double* dst, const double* src, int n, bool vec) {
  const unsigned int d = (unsigned int)__cvta_generic_to_shared(dst);
  if (vec) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(8 * n) : "memory");
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n > 0 ? 8 : 0) : "memory");
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d + 8), "l"(n > 1 ? src + 1 : src),
                 "r"(n > 1 ? 8 : 0)
                 : "memory");
  }
}

// One operand: 64 rows of the tile.  kK: row i of the matrix at base +
// (size_t)row(i) ld, K contiguous, row(i) = idx ? idx[i] : i; else element
// (i, k) at base + i + (size_t)k ld.  A thread keeps its four row pointers.
// vec: every row start (kK) or line start (!kK) is 16-byte aligned and K
// ranges and tiles begin at even offsets.
template <bool kK, int NT = 128> struct Operand {
  static constexpr int kRows = NT / 8, kLines = NT / 32;  // rows (kK) or K lines (!kK) staged per round
  const double* base;
  size_t ld;
  int i0, n;  // first row of the tile, rows of the matrix
  bool vec;
  const double* rp[kT / kRows];
  unsigned int ok;

  __device__ __forceinline__ Operand(const double* b, size_t l, int i0_, int n_, bool v, const int* idx = nullptr)
      : base(b), ld(l), i0(i0_), n(n_), vec(v), ok(0) {
#pragma unroll
    for (int q = 0; q < kT / kRows; ++q) {
      const int i = i0 + (int)(threadIdx.x >> 3) + kRows * q;
      rp[q] = base;
      if (kK && i < n) {
        rp[q] = base + (size_t)(idx ? idx[i] : i) * ld;
        ok |= 1u << q;
      }
    }
  }

  // K [k0, min(k0 + 16, k1)) into a stage; NT threads
  __device__ __forceinline__ void stage(double* s, int k0, int k1) const {
#pragma unroll
    for (int q = 0; q < (kK ? kT / kRows : kStep / kLines); ++q) {
      if (kK) {
        const int r = (int)(threadIdx.x >> 3) + kRows * q, kk = (int)(threadIdx.x & 7) * 2;
        const int m = ((ok >> q) & 1u) ? max(0, min(2, k1 - k0 - kk)) : 0;
        copy2(s + r * kLdK + kk, m ? rp[q] + k0 + kk : base, m, vec);
      } else {
        const int kk = (int)(threadIdx.x >> 5) + kLines * q, r = (int)(threadIdx.x & 31) * 2;
        const int m = k0 + kk < k1 ? max(0, min(2, n - i0 - r)) : 0;
        copy2(s + kk * kLdM + r, m ? base + (size_t)(k0 + kk) * ld + i0 + r : base, m, vec);
      }
    }
  }
};

// fragment element (row r, k) of a stage
template <bool kK> __device__ __forceinline__ double frag(const double* s, int r, int k) {
  return kK ? s[r * kLdK + k] : s[k * kLdM + r];
}

template <int NB> using AccNb = double[2][NB][2];
using Acc = AccNb<8>;

// acc[mb][nb] += the warp's 16 x 8 NB block of X Y^T over K [k0, k1): the
// first NB blocks of 8 columns (the rest of the tile is not needed), or, with
// eight warps, blocks 4 (warp / 4) .. + 3
template <int NB, bool kA, bool kB, int NT, int NA>
__device__ __forceinline__ void tile_product_nb(const Operand<kA, NT>& X, const Operand<kB, NT>& Y, int k0, int k1,
                                                double* smem, double (&acc)[2][NA][2]) {
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) & 3, cb = NT > 128 ? (threadIdx.x >> 7) * NB : 0;
  const int g = lane >> 2, t = lane & 3;
  const int ns = (max(0, k1 - k0) + kStep - 1) / kStep;
  auto load = [&](int s) {
    if (s < ns) {
      double* st = smem + (size_t)(s % kStages) * 2 * kOperand;
      X.stage(st, k0 + s * kStep, k1);
      Y.stage(st + kOperand, k0 + s * kStep, k1);
    }
    cp_async_commit();
  };
  for (int s = 0; s < kStages - 1; ++s) load(s);
  for (int s = 0; s < ns; ++s) {
    cp_async_wait<kStages - 2>();
    __syncthreads();  // stage s has landed, and everyone is done with stage s - 1
    load(s + kStages - 1);
    const double* sx = smem + (size_t)(s % kStages) * 2 * kOperand;
    const double* sy = sx + kOperand;
#pragma unroll
    for (int kk = 0; kk < kStep; kk += 4) {
      double a[2], b[NB];
#pragma unroll
      for (int m = 0; m < 2; ++m) a[m] = frag<kA>(sx, 16 * warp + 8 * m + g, kk + t);
#pragma unroll
      for (int j = 0; j < NB; ++j) b[j] = frag<kB>(sy, 8 * (cb + j) + g, kk + t);
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        dmma_884(acc[0][j], a[0], b[j]);
        dmma_884(acc[1][j], a[1], b[j]);
      }
    }
  }
  cp_async_wait<0>();
  __syncthreads();  // the stages may be reused
}

// the same with at least `nbl` (1..8) blocks formed.  Whole instances rather
// than a test per block: a matrix instruction whose predicate is off still
// takes its time on the pipe.
template <bool kA, bool kB>
__device__ __forceinline__ void tile_product(const Operand<kA>& X, const Operand<kB>& Y, int k0, int k1, int nbl,
                                             double* smem, Acc& acc) {
  if (nbl > 4) tile_product_nb<8, kA, kB>(X, Y, k0, k1, smem, acc);
  else if (nbl > 2) tile_product_nb<4, kA, kB>(X, Y, k0, k1, smem, acc);
  else if (nbl > 1) tile_product_nb<2, kA, kB>(X, Y, k0, k1, smem, acc);
  else tile_product_nb<1, kA, kB>(X, Y, k0, k1, smem, acc);
}

template <int NB> __device__ __forceinline__ void clear(double (&acc)[2][NB][2]) {
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int j = 0; j < NB; ++j) acc[m][j][0] = acc[m][j][1] = 0.0;
}

// f(row, column, value) for the thread's elements of the tile; the value may
// be changed where acc is not const
template <int NB, typename A, typename F> __device__ __forceinline__ void each_of(A& acc, F f) {
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) & 3, cb = NB < 8 ? (threadIdx.x >> 7) * NB : 0;
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) f(16 * warp + 8 * m + g, 8 * (cb + j) + 2 * t + h, acc[m][j][h]);
}
template <typename F> __device__ __forceinline__ void each(const Acc& acc, F f) { each_of<8>(acc, f); }

}  // namespace dg
}  // namespace mf
