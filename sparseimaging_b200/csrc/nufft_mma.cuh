// NUFFT interpolation and spreading (NUFFT2d2 / NUFFT2d1 of
// c/mfista_nufft_lib.c:123-243) on the FP64 matrix instruction
// (mma.sync m8n8k4.f64), for one problem, batches that share their points and
// batches with points of their own.
//
// Both are separable tap sums: a point's 576 weights are wx[24] x wy[24].
// Tap by tap they are bound by gathers and by address arithmetic (an FP64
// batch ran at 3 % of the FP64 rate).  Here a warp takes 16 points of one tile
// (interpolation) or 8 x 8 cells (spreading) through matrix products whose
// operands come from shared memory and registers, on "virtual" coordinates:
// grid rows and columns before the reference's row wrap and Hermitian fold,
// so that every point sees plain consecutive taps.
//
// FP64 products and sums throughout, also for the FP32 operators (whose grids
// and residuals stay FP32): m8n8k4.f64 runs at the rate of the FP64 pipe
// (37 TFLOP/s measured, with one shared-memory operand per 512 operations).
//
// Measured on B200, FP64, microseconds per launch, tap by tap -> here:
//   grid, points, problems          interpolation    spreading
//   64 x 64, 2016, 1                 40.1 -> 7.3      37.0 -> 10.4
//   128 x 128, 8100, 1               39.7 -> 10.2     60.6 -> 14.5
//   128 x 128, 8100, 64               489 -> 170       581 -> 142
//   256 x 256, 19998, 64             1130 -> 471      1710 -> 361
//   128 x 128, 102070 over 16 frames  163 -> 50        605 -> 117
// The products alone would take 60 us and 80 us at 128 x 128 with 64 problems;
// a copy of the interpolation without them takes 51 us.
#pragma once
#include "nufft_ops.cuh"

namespace mf {

__device__ __forceinline__ void dmma_884(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// asynchronous copy of one complex grid cell; valid = false writes zero
template <typename T>
__device__ __forceinline__ void cp_async_cell(cplx<T>* dst, const cplx<T>* src, bool valid) {
  const unsigned int d = (unsigned int)__cvta_generic_to_shared(dst);
  const unsigned int n = valid ? (unsigned int)sizeof(cplx<T>) : 0u;
  if (sizeof(cplx<T>) == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

// ---------------------------------------------------------------------------
// Interpolation.  The points are binned by their first tap (mx - 11, my - 11)
// into kImTile x kImTile tiles of virtual positions; all taps of a tile's
// points lie in a 39 x 39 window (kImWin = 40 staged).  A CTA takes up to 128
// points of a tile and a chunk of PB problems.  Per problem it stages the
// window (cp.async, the next problem's window in flight behind the products;
// dropped taps are staged as zeros), and each warp forms, for 16 points and 4
// window rows at a time,
//   T[p][row, re/im] = sum_c wy_p[c] G[row, c][re/im]      (K = columns)
//   y_p += sum_row wx_p[row] T[p][row]
// as m8n8k4 products: A = wy (in registers for all problems), B = the window's
// cells (one 8-byte shared load per lane serves both blocks of 8 points), so
// nothing of a matrix tile is idle for a single problem.  Only the rows and
// columns that the 16 points reach are walked, in four row groups whose
// sums are added as (0 + 1) + (2 + 3); a CTA with few points gives its warps
// one or two groups each.  Bound by the FP64 pipe where the chip is full and
// by the length of one CTA's chain where it is not, so the points per CTA
// (32, 64 or 128) and the problems per CTA follow the amount of work
// (NufftOp::build_im_tiles): 128-point CTAs of 8 problems throughout took 215
// us an iteration at 100 x 100 with 11 problems (166 here), 106 at 64 x 64
// with one (93).
// Signs: the reference negates the imaginary part of direct taps (NU_SIGN) and
// keeps that of mirrored ones; a tap is direct or mirrored by its column alone,
// so the imaginary parts of mirrored columns are flipped at the fragment (at
// the sum, when all columns of the unit are) and the sum is negated once.
// A problem's sums depend neither on its CTA's points nor on the other
// problems: groups and chi^2 slots (32 points) are the same for every cut.
//
// Problems with points of their own can make thousands of tiles of a few
// points, which stage a window each and leave most of eight warps idle.  Where
// there are many (NufftOp::build_im_tiles) a CTA has four warps, or two, and at
// most half as many points as threads, two to four times as many are resident,
// and only the cells that the points reach are read (the others are zeros, as
// their weights are): the same bits.  Microseconds per launch with eight, four
// and two warps (tap by tap before): 10 frames of 3000 random points at 256 x
// 256 125, 88, 83 (49; FP32 125, 88, 76 (45)), along tracks 49, 37, 37 (48); 16
// of 1000 at 128 x 128 53, 39, 37 (30) and 28, 23, 23 (30); 16 of 12000 98, 82,
// 102 (283) and 80, 74, 90 (280).
// ---------------------------------------------------------------------------
constexpr int kImTile = 16;
constexpr int kImWin = kImTile + kTaps;  // 40: 39 used, a multiple of 4
constexpr int kImPts = 128;              // points per CTA at most: 8 warps x 16
constexpr int kImSteps = kImWin / 4;     // column steps of 4

struct ImTileItem {
  int row0, col0;    // window origin, virtual
  int start, count;  // perm[start, start + count)
  int prob;          // its problem (points of its own), or -1 (shared points)
  int slot, nslot;   // first chi^2 slot (one per 32 points), slots of the problem
  int item, nitem;   // CTA of the problem, CTAs of the problem
  int box;           // cells of the window that its points reach: rows [r0, r1), columns [c0, c1), 8 bits each
};

// row stride of the staged window: the four rows of a B fragment hit all banks
template <typename T> struct ImWindow {
  static constexpr int kLd = sizeof(T) == 8 ? 44 : 52;
  static constexpr size_t kBytes = sizeof(cplx<T>) * (size_t)kImWin * kLd;
};
constexpr size_t im_red_bytes(int pb) { return sizeof(double2) * (size_t)pb * 8 * 16; }
constexpr int kImBuf = 2;   // staged windows
template <typename T, int PB> constexpr size_t im_smem() {
  return (PB > 1 ? kImBuf : 1) * ImWindow<T>::kBytes + im_red_bytes(PB);
}

__device__ __forceinline__ double2 im_add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }

// what a warp keeps of its unit of 16 points
struct ImUnit {
  const double* wx;           // row weights
  unsigned int oa, ob;        // first ones of points g and g + 8
  int dra, drb;               // their first rows, in the window
  bool va, vb, mixed;         // mixed: some lane of the warp has mirrored cells
  unsigned int mir;           // bit kk: this lane's imaginary cell of column step kk is mirrored
  double a0[kImSteps], a1[kImSteps];  // their column weights at the lane's columns
};

// row steps [s0, s1) of 4 window rows from rlo, NK column steps of 4 from w's
// column; TWO: the unit has a second block of 8 points.  Both are template
// arguments because a matrix instruction whose predicate is off still takes
// its time on the pipe.
template <int NK, bool TWO, typename T, int LD>
__device__ __forceinline__ void interp_rows(const ImUnit& u, const T* w, int rlo, int s0, int s1, int lane,
                                            double (&y0)[2], double (&y1)[2]) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll 1
  for (int s = s0; s < s1; ++s) {
    const int r = rlo + 4 * s;
    const int ja = r + t - u.dra, jb = r + t - u.drb;
    const double wa = (u.va && ja >= 0 && ja < kTaps) ? u.wx[(size_t)u.oa + ja] : 0.0;
    const double wb = (TWO && u.vb && jb >= 0 && jb < kTaps) ? u.wx[(size_t)u.ob + jb] : 0.0;
    const T* brow = w + 2 * ((r + (g >> 1)) * LD + t) + (g & 1);
    double d0[2][2] = {{0.0, 0.0}, {0.0, 0.0}}, d1[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    double b[NK];
#pragma unroll
    for (int kk = 0; kk < NK; ++kk) b[kk] = (double)brow[8 * kk];
    if (u.mixed) {
#pragma unroll
      for (int kk = 0; kk < NK; ++kk) b[kk] = ((u.mir >> kk) & 1u) ? -b[kk] : b[kk];
    }
#pragma unroll
    for (int kk = 0; kk < NK; ++kk) {
      dmma_884(d0[kk & 1], u.a0[kk], b[kk]);
      if (TWO) dmma_884(d1[kk & 1], u.a1[kk], b[kk]);
    }
    y0[0] = fma(wa, d0[0][0] + d0[1][0], y0[0]);
    y0[1] = fma(wa, d0[0][1] + d0[1][1], y0[1]);
    if (TWO) {
      y1[0] = fma(wb, d1[0][0] + d1[1][0], y1[0]);
      y1[1] = fma(wb, d1[0][1] + d1[1][1], y1[1]);
    }
  }
}

template <bool TWO, typename T, int LD>
__device__ __forceinline__ void interp_unit(const ImUnit& u, int nk, const T* w, int rlo, int s0, int s1, int lane,
                                            double (&y0)[2], double (&y1)[2]) {
  switch (nk) {  // 24 columns at least, 39 at most
    case 6: interp_rows<6, TWO, T, LD>(u, w, rlo, s0, s1, lane, y0, y1); break;
    case 7: interp_rows<7, TWO, T, LD>(u, w, rlo, s0, s1, lane, y0, y1); break;
    case 8: interp_rows<8, TWO, T, LD>(u, w, rlo, s0, s1, lane, y0, y1); break;
    case 9: interp_rows<9, TWO, T, LD>(u, w, rlo, s0, s1, lane, y0, y1); break;
    default: interp_rows<kImSteps, TWO, T, LD>(u, w, rlo, s0, s1, lane, y0, y1); break;
  }
}

template <typename T, int PB, int NT>
__global__ void __launch_bounds__(NT, 512 / NT)
    k_nufft_interp_mma(NufftGeom<T> geo, const double* __restrict__ wxd, const double* __restrict__ wyd,
                       const ImTileItem* __restrict__ tiles, const int2* __restrict__ perm,
                       const cplx<T>* __restrict__ gall, long gstride, int nx, int ny, double inv_mm,
                       const ProbState* __restrict__ st, int gate, Partials part, int qchi, int nslots,
                       cplx<T>* __restrict__ y2, int B, const double2* __restrict__ ax_base,
                       double2* __restrict__ ax_out) {
  constexpr int LD = ImWindow<T>::kLd;
  constexpr int kCells = (kImWin * kImWin + NT - 1) / NT, NW = NT / 32;
  extern __shared__ __align__(16) unsigned char im_smem_raw[];
  cplx<T>* win = reinterpret_cast<cplx<T>*>(im_smem_raw);
  double* s_red = reinterpret_cast<double*>(im_smem_raw + (PB > 1 ? kImBuf : 1) * ImWindow<T>::kBytes);
  __shared__ int s_list[PB];
  __shared__ int s_cnt[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const ImTileItem tl = tiles[blockIdx.x];
  int nact;
  if (PB > 1) {
    nact = active_share<PB>(st, gate, B, s_list, s_cnt, geo.act_lists);
  } else {
    const int b = tl.prob >= 0 ? tl.prob : (int)blockIdx.y;
    nact = gate_ok(st[b], gate) ? 1 : 0;
    if (threadIdx.x == 0) s_list[0] = b;
    __syncthreads();
  }
  if (nact == 0) return;
  // stored cell of each window cell this thread copies (-1: dropped tap)
  int cell[kCells];
#pragma unroll
  for (int i = 0; i < kCells; ++i) {
    const int v = threadIdx.x + NT * i;
    cell[i] = -1;
    const int r = v / kImWin, c = v % kImWin;
    if (v < kImWin * kImWin &&
        (NT == 256 || (r >= (tl.box & 255) && r < ((tl.box >> 8) & 255) && c >= ((tl.box >> 16) & 255) && c < tl.box >> 24))) {
      const int vr = tl.row0 + r, vc = tl.col0 + c;
      int col = half_col(vc, ny), row = -1;
      if (col >= 0) {
        row = wrap_row(vr, nx);
      } else {
        col = half_col(-vc, ny);
        row = wrap_row(-vr, nx);
      }
      if (col >= 0 && row >= 0) cell[i] = row * (ny + 1) + col;
    }
  }
  auto stage = [&](int slot, int buf) {
    const cplx<T>* gr = gall + (size_t)s_list[slot] * gstride;
    cplx<T>* w = win + (size_t)buf * kImWin * LD;
#pragma unroll
    for (int i = 0; i < kCells; ++i) {
      const int v = threadIdx.x + NT * i;
      if (v < kImWin * kImWin)
        cp_async_cell<T>(w + (v / kImWin) * LD + v % kImWin, gr + max(cell[i], 0), cell[i] >= 0);
    }
  };
  for (int i = 0; i < (PB > 1 ? kImBuf - 1 : 1); ++i) {
    if (i < nact) stage(i, i);
    cp_async_commit();
  }
  // chi^2 slots beyond this problem's: zero
  if ((int)threadIdx.x < nact && qchi >= 0)
    for (int sl = tl.nslot + tl.item; sl < nslots; sl += tl.nitem) part.at(qchi, s_list[threadIdx.x])[sl] = 0.0;

  // warps over (unit of 16 points, row groups): nu units, ng warps a unit
  const int nu = max(1, (tl.count + 15) >> 4), ng = 2 * nu > NW ? 1 : 4 * nu > NW ? 2 : 4;
  const int unit = warp % nu, grp = warp / nu;
  const bool on = grp < ng;
  const int p0 = tl.start + unit * 16;
  const int np = on ? min(16, tl.start + tl.count - p0) : 0;
  int kq = 0, drq = 0, dcq = 0;
  if (lane < np) {
    const int2 pk = perm[p0 + lane];
    kq = pk.x;
    drq = pk.y & 0xff;
    dcq = pk.y >> 8;
  }
  const unsigned int all = 0xffffffffu;
  const int ka = __shfl_sync(all, kq, g), kb = __shfl_sync(all, kq, g + 8);
  const int dra = __shfl_sync(all, drq, g), drb = __shfl_sync(all, drq, g + 8);
  const int dca = __shfl_sync(all, dcq, g), dcb = __shfl_sync(all, dcq, g + 8);
  const bool va = g < np, vb = g + 8 < np;
  const bool two = np > 8;
  // rows and columns of the window that the unit's points reach, in steps of 4
  int rlo = __reduce_min_sync(all, lane < np ? drq : kImWin), rhi = __reduce_max_sync(all, lane < np ? drq + kTaps : 0);
  int clo = __reduce_min_sync(all, lane < np ? dcq : kImWin), chi_ = __reduce_max_sync(all, lane < np ? dcq + kTaps : 0);
  if (np == 0) rlo = rhi = clo = chi_ = 0;
  const int ns = (rhi - rlo + 3) >> 2, nk = (chi_ - clo + 3) >> 2;
  rlo = min(rlo, kImWin - 4 * ns);
  clo = min(clo, kImWin - 4 * nk);
  ImUnit u;
  u.wx = wxd;
  u.oa = (unsigned int)ka * kTaps;
  u.ob = (unsigned int)kb * kTaps;
  u.dra = dra;
  u.drb = drb;
  u.va = va;
  u.vb = vb;
  u.mir = 0;
#pragma unroll
  for (int kk = 0; kk < kImSteps; ++kk) {
    const int c = clo + 4 * kk + t;
    const int ja = c - dca, jb = c - dcb;
    u.a0[kk] = (va && kk < nk && ja >= 0 && ja < kTaps) ? wyd[(size_t)ka * kTaps + ja] : 0.0;
    u.a1[kk] = (vb && kk < nk && jb >= 0 && jb < kTaps) ? wyd[(size_t)kb * kTaps + jb] : 0.0;
    if ((g & 1) && half_col(tl.col0 + c, ny) < 0) u.mir |= 1u << kk;
  }
  // mirrored as a whole (lanes of imaginary cells agree on all columns): the
  // sign goes to the sum
  const unsigned int cols = (1u << nk) - 1u;
  const bool flip = __all_sync(all, !(g & 1) || (u.mir & cols) == cols);
  u.mixed = !flip && __any_sync(all, (u.mir & cols) != 0);
  const int q0 = grp * (4 / ng), q1 = on ? q0 + 4 / ng : q0;
  for (int i = 0; i < nact; ++i) {
    if (PB > 1) cp_async_wait<kImBuf - 2>();
    else cp_async_wait<0>();
    __syncthreads();  // window i has landed for every thread, and everyone is done with window i - 1
    if (PB > 1) {
      if (i + kImBuf - 1 < nact) stage(i + kImBuf - 1, (i + kImBuf - 1) % kImBuf);
      cp_async_commit();
    }
    const T* w = reinterpret_cast<const T*>(win + (size_t)(PB > 1 ? i % kImBuf : 0) * kImWin * LD + clo);
    double tot = 0.0, even = 0.0;
    for (int q = q0; q < q1; ++q) {
      double y0[2] = {0.0, 0.0}, y1[2] = {0.0, 0.0};
      const int s0 = (q * ns) >> 2, s1 = ((q + 1) * ns) >> 2;  // 6 row steps at least
      {
        if (two) interp_unit<true, T, LD>(u, nk, w, rlo, s0, s1, lane, y0, y1);
        else interp_unit<false, T, LD>(u, nk, w, rlo, s0, s1, lane, y0, y1);
      }
      // over the four rows of a step (lanes t): lane t ends with component
      // t & 1 of point g + 8 (t >> 1)
      const bool im = (t & 1) != 0, hi = (t & 2) != 0;
      const double m0 = (im ? y0[1] : y0[0]) + __shfl_xor_sync(all, im ? y0[0] : y0[1], 1);
      const double m1 = (im ? y1[1] : y1[0]) + __shfl_xor_sync(all, im ? y1[0] : y1[1], 1);
      double v = (hi ? m1 : m0) + __shfl_xor_sync(all, hi ? m0 : m1, 2);
      if (im && flip) v = -v;
      if (ng == 4) tot = v;
      else if (q & 1) tot += even + v;  // (groups 0 + 1) + (groups 2 + 3)
      else even = v;
    }
    if (on) s_red[((i * 8 + warp) * 16 + 8 * (t >> 1) + g) * 2 + (t & 1)] = tot;
  }
  __syncthreads();
  // residual, chi^2 and models: a warp per (problem, 32 points)
  const int nq = (nu + 1) >> 1;
  for (int e0 = warp; e0 < nact * nq; e0 += NW) {
    const int i = e0 / nq, j0 = 32 * (e0 - i * nq);
    const int b = s_list[i];
    const int j = j0 + lane;
    double chi = 0.0;
    if (j < tl.count) {
      const double2* v = reinterpret_cast<const double2*>(s_red) + (i * 8 + (j >> 4)) * 16 + (j & 15);
      double2 f = v[0];
      if (ng == 2) f = im_add(f, v[nu * 16]);
      if (ng == 4) f = im_add(im_add(f, v[nu * 16]), im_add(v[2 * nu * 16], v[3 * nu * 16]));
      double fr = f.x, fi = f.y;
      const int k = perm[tl.start + j].x;
      const size_t e = (size_t)b * geo.y2_bstride + k;
      fr *= inv_mm;
      fi *= -inv_mm;
      if (ax_base) {
        const double2 ab = ax_base[e];
        fr += ab.x;
        fi += ab.y;
      }
      if (ax_out) ax_out[e] = make_double2(fr, fi);
      const double wgt = geo.weight[k];
      const double rr = (geo.vis_r[k] - fr) * wgt, ri = (geo.vis_i[k] - fi) * wgt;
      chi = rr * rr + ri * ri;
      if (y2) y2[e] = mk<T>((T)(rr * wgt), (T)(ri * wgt));
    }
    chi = warp_sum(chi);
    if (lane == 0 && qchi >= 0) part.at(qchi, b)[tl.slot + (j0 >> 5)] = chi;
  }
}

// ---------------------------------------------------------------------------
// Spreading, output-stationary: the stored half grid is cut into tiles of
// 8 rows x 16 columns, each with the list of the virtual points that have a
// tap on it (every uv point as itself, imaginary part negated, and mirrored,
// both weight vectors reversed, each with half the residual).  A tile is four
// 8 x 8 products over the list,
//   D[(row, re/im)][col] = sum_p (wx_p[row] y_p[re/im]) wy_p[col],
// four rows x {re, im} by eight columns, K = points, so a single problem fills
// the matrix tile.  A CTA takes up to kSmSeg list entries and up to PB
// problems: its warps go over (pair of problems, blocks, even or odd steps of
// 4 points).  A pair shares a warp's weights and their index arithmetic, and
// with half of the steps a warp needs few enough registers for three CTAs an
// SM: 146 us at 128 x 128 with 64 problems, against 199 with a problem and
// both parities to a warp and two CTAs.  Each block's sum is the even steps'
// plus the odd steps' whatever the mapping, and longer lists are cut into
// segments whose partial tiles the tile's last CTA adds in segment order, so
// neither the batch nor the order of the CTAs changes a result.  A segment is
// kSmSeg entries, or as many times that (staged one after another) as leave
// at most kSmSegMax partial tiles, 2 KB each, to a problem: the scratch stays
// within 8 MB a problem, where it would be 75 bytes a point and problem.
// The weights are read where they lie (48 values a point, shared by the tiles
// around it): cached, with the taps outside [0, 24) as zeros.
// Thinly spread points leave most tiles with a few entries, a CTA's chain of
// loads and barriers each.  Where one problem, or problems with points of their
// own, make many tiles (NufftOp::build_sm_items), those of at most kSmLight
// entries go eight to a CTA, one to a warp, entries in the lanes: the same sums
// without barriers.  Microseconds per launch with a CTA to every tile -> here
// (tap by tap before): 10 frames of 3000 random points at 256 x 256 86 -> 33
// (92), of 300 66 -> 12 (23), 16 of 12000 at 128 x 128 273 -> 195 (585); one
// problem of 3000 points at 512 x 512 31 -> 8 (220).  With at most 16 entries
// a light tile: 58, 12, 195 and 8.
// ---------------------------------------------------------------------------
constexpr int kSmRows = 8, kSmCols = 16;
constexpr int kSmSeg = 256;  // list entries staged at once
constexpr int kSmSegMax = 4096;  // partial tiles of a problem at most
constexpr int kSmLight = 32;     // entries of a tile that one warp takes at most

// nseg = 0: `count` light tiles, items[start] and following
struct SmItem {
  int tile;          // tile of the stored half grid, row-major
  int start, count;  // list entries; count a multiple of 8
  int seg, nseg;     // segment of the tile's list
  int scratch;       // scratch slot of the tile's segment 0
  int ticket;        // the tile's ticket
  int prob;          // its problem, or -1 (shared points)
};

struct SmPoint {
  unsigned int k24;  // first weight of the point
  int x0, y0;  // first tap, virtual
  int fl;      // mirrored
};

// a list entry's geometry; an empty one has no tap anywhere
template <typename T>
__device__ __forceinline__ SmPoint sm_point(const NufftGeom<T>& geo, unsigned int code) {
  SmPoint p{0, 1 << 29, 1 << 29, 0};
  if (code != 0xffffffffu) {
    const int k = (int)(code >> 1), fl = (int)(code & 1u);
    p.k24 = (unsigned int)k * kTaps;
    p.x0 = fl ? -geo.mx[k] - kMSP : geo.mx[k] - (kMSP - 1);
    p.y0 = fl ? -geo.my[k] - kMSP : geo.my[k] - (kMSP - 1);
    p.fl = fl;
  }
  return p;
}

// and its half residual, the imaginary part negated for a direct point
template <typename T>
__device__ __forceinline__ double2 sm_residual(const cplx<T>* __restrict__ y2, unsigned int code) {
  if (code == 0xffffffffu) return make_double2(0.0, 0.0);
  const cplx<T> r = y2[code >> 1];
  return make_double2(0.5 * (double)r.x, (code & 1u) ? 0.5 * (double)r.y : -0.5 * (double)r.y);
}

// (the exchange of the parities' sums reuses the residuals' space)
constexpr size_t sm_exchange(int pb) { return sizeof(double) * 64 * (pb > 1 ? 8 * 4 : 8); }
template <typename T, int PB> constexpr size_t sm_smem() {
  const size_t y = sizeof(double2) * (size_t)PB * kSmSeg;
  return (size_t)kSmSeg * sizeof(SmPoint) + (y > sm_exchange(PB) ? y : sm_exchange(PB));
}

constexpr int kSmOut = 1 << 28;  // no tap reaches it
// virtual row and column of a stored one
__device__ __forceinline__ int sm_row(int row, int nx) { return row < nx ? row : row < 2 * nx ? row - 2 * nx : kSmOut; }
__device__ __forceinline__ int sm_col(int col, int ny) { return col < ny ? col : col == ny ? -ny : kSmOut; }

// the products of NP problems' MB x NB blocks (from mb0, nb0) over the steps
// of parity ch0; problem p's residuals at s_yp + p kSmSeg
template <int MB, int NB, int NP>
__device__ __forceinline__ void spread_products(const SmPoint* s_pt, const double2* s_yp, int count, int mb0, int nb0,
                                                int ch0, int row_base, int col_base, int nx, int ny, int lane,
                                                const double* __restrict__ wxd, const double* __restrict__ wyd,
                                                double (&d)[2][4][2]) {
  const int g = lane >> 2, t = lane & 3;
  int mr[MB], mc[NB];
#pragma unroll
  for (int m = 0; m < MB; ++m) mr[m] = sm_row(row_base + 4 * (mb0 + m) + (g >> 1), nx);
#pragma unroll
  for (int n = 0; n < NB; ++n) mc[n] = sm_col(col_base + 8 * (nb0 + n) + g, ny);
  const SmPoint* pt = s_pt + 4 * ch0 + t;
  const double* yp = reinterpret_cast<const double*>(s_yp + 4 * ch0 + t) + (g & 1);
#pragma unroll 4
  for (int e = 0; e < count; e += 8) {
    const SmPoint p = pt[e];
    double a[MB], b[NB];
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      const int j = mr[m] - p.x0;
      a[m] = (unsigned)j < (unsigned)kTaps ? __ldg(wxd + p.k24 + (p.fl ? kTaps - 1 - j : j)) : 0.0;
    }
#pragma unroll
    for (int n = 0; n < NB; ++n) {
      const int j = mc[n] - p.y0;
      b[n] = (unsigned)j < (unsigned)kTaps ? __ldg(wyd + p.k24 + (p.fl ? kTaps - 1 - j : j)) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      const double y = yp[2 * (q * kSmSeg + e)];
#pragma unroll
      for (int m = 0; m < MB; ++m) {
        const double ay = a[m] * y;
#pragma unroll
        for (int n = 0; n < NB; ++n) dmma_884(d[q][m * NB + n], ay, b[n]);
      }
    }
  }
}

// block blk of a tile into the grid.  Lane (g, t): row g >> 1, re or im (g & 1),
// columns 2t, 2t + 1; lanes g and g ^ 1 exchange so that each writes one
// complex cell
template <typename T>
__device__ __forceinline__ void sm_store(cplx<T>* __restrict__ gr, int blk, double d0, double d1, int row_base,
                                         int col_base, int nx, int ny, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const double other = __shfl_xor_sync(0xffffffffu, (g & 1) ? d0 : d1, 4);
  const double re = (g & 1) ? other : d0, im = (g & 1) ? d1 : other;
  const int row = row_base + 4 * (blk >> 1) + (g >> 1), col = col_base + 8 * (blk & 1) + 2 * t + (g & 1);
  if (row < 2 * nx && col <= ny) gr[(size_t)row * (ny + 1) + col] = mk<T>((T)re, (T)im);
}

// a light tile, by a warp
template <typename T>
__device__ __forceinline__ void spread_light(const NufftGeom<T>& geo, const double* __restrict__ wxd,
                                             const double* __restrict__ wyd, const unsigned int* __restrict__ list,
                                             int count, const cplx<T>* __restrict__ y2, cplx<T>* __restrict__ gr,
                                             int row_base, int col_base, int nx, int ny, int lane) {
  const unsigned int all = 0xffffffffu;
  const int g = lane >> 2, t = lane & 3;
  const unsigned int code = lane < count ? list[lane] : all;
  const SmPoint p = sm_point<T>(geo, code);
  const double2 y = sm_residual<T>(y2, code);
  int mr[2], mc[2];
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    mr[m] = sm_row(row_base + 4 * m + (g >> 1), nx);
    mc[m] = sm_col(col_base + 8 * m + g, ny);
  }
  double acc[2][4][2];  // even and odd steps
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int m = 0; m < 4; ++m) acc[q][m][0] = acc[q][m][1] = 0.0;
  for (int e = 0; e < count; e += 8)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int src = e + 4 * q + t;
      const unsigned int k24 = __shfl_sync(all, p.k24, src);
      const int x0 = __shfl_sync(all, p.x0, src), y0 = __shfl_sync(all, p.y0, src), fl = __shfl_sync(all, p.fl, src);
      const double re = __shfl_sync(all, y.x, src), im = __shfl_sync(all, y.y, src);
      double a[2], b[2];
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int j = mr[m] - x0, i = mc[m] - y0;
        a[m] = (unsigned)j < (unsigned)kTaps ? __ldg(wxd + k24 + (fl ? kTaps - 1 - j : j)) : 0.0;
        b[m] = (unsigned)i < (unsigned)kTaps ? __ldg(wyd + k24 + (fl ? kTaps - 1 - i : i)) : 0.0;
      }
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const double ay = a[m] * ((g & 1) ? im : re);
#pragma unroll
        for (int n = 0; n < 2; ++n) dmma_884(acc[q][2 * m + n], ay, b[n]);
      }
    }
#pragma unroll
  for (int m = 0; m < 4; ++m)
    sm_store<T>(gr, m, acc[0][m][0] + acc[1][m][0], acc[0][m][1] + acc[1][m][1], row_base, col_base, nx, ny, lane);
}

// kLong: there are segments of more than kSmSeg entries (an instance of its
// own: with the loop the others take 2-5 % longer)
template <typename T, int PB, bool kLong>
__global__ void __launch_bounds__(256, 3)
    k_nufft_spread_mma(NufftGeom<T> geo, const double* __restrict__ wxd, const double* __restrict__ wyd,
                       const SmItem* __restrict__ items, const unsigned int* __restrict__ vlist,
                       const cplx<T>* __restrict__ y2, cplx<T>* __restrict__ gall, long gstride, int nx, int ny,
                       int ntcol, const ProbState* __restrict__ st, int gate, int B, double* __restrict__ scratch,
                       unsigned int* __restrict__ tickets) {
  extern __shared__ __align__(16) unsigned char sm_smem_raw[];
  SmPoint* s_pt = reinterpret_cast<SmPoint*>(sm_smem_raw);
  double2* s_y = reinterpret_cast<double2*>(sm_smem_raw + (size_t)kSmSeg * sizeof(SmPoint));  // [PB][kSmSeg]
  double* s_ex = reinterpret_cast<double*>(s_y);  // [warp][block][64], after the products
  __shared__ int s_list[PB];
  __shared__ int s_cnt[8];
  __shared__ unsigned int s_ticket;
  const SmItem it = items[blockIdx.x];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int nact;
  if (PB > 1) {
    nact = active_share<PB>(st, gate, B, s_list, s_cnt, geo.act_lists);
  } else {
    if (it.nseg == 0) {
      if (warp >= it.count) return;
      const SmItem l = items[it.start + warp];
      const int b = l.prob >= 0 ? l.prob : (int)blockIdx.y, tr = l.tile / ntcol;
      if (!gate_ok(st[b], gate)) return;
      spread_light<T>(geo, wxd, wyd, vlist + l.start, l.count, y2 + (size_t)b * geo.y2_bstride,
                      gall + (size_t)b * gstride, tr * kSmRows, (l.tile - tr * ntcol) * kSmCols, nx, ny, lane);
      return;
    }
    const int b = it.prob >= 0 ? it.prob : (int)blockIdx.y;
    nact = gate_ok(st[b], gate) ? 1 : 0;
    if (threadIdx.x == 0) s_list[0] = b;
    __syncthreads();
  }
  if (nact == 0) return;
  const int tr = it.tile / ntcol, tcl = it.tile - tr * ntcol;
  const int row_base = tr * kSmRows, col_base = tcl * kSmCols;
  // warps over (pair of problems, blocks of the tile, parity of the steps):
  // the fewer pairs, the fewer blocks a warp takes
  const int ch = warp & 1, groups = nact > 4 ? 1 : nact > 2 ? 2 : 4;
  const int pair = (warp >> 1) / groups, sub = (warp >> 1) - pair * groups;
  const int nblk_w = 4 / groups, blk0 = sub * nblk_w;
  const int np = min(2, nact - 2 * pair);  // problems of the warp (< 1: none)
  double acc[2][4][2];
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int m = 0; m < 4; ++m) acc[q][m][0] = acc[q][m][1] = 0.0;
  const double2* yp = s_y + (size_t)2 * pair * kSmSeg;
  for (int base = 0; base < (kLong ? it.count : 1); base += kSmSeg) {
    const int cnt = kLong ? min(kSmSeg, it.count - base) : it.count;
    if (base) __syncthreads();  // the entries before have been read
    for (int e = threadIdx.x; e < cnt * nact; e += blockDim.x) {
      const int i = e / cnt, q = e - i * cnt;
      const unsigned int code = vlist[it.start + base + q];
      s_y[(size_t)i * kSmSeg + q] = sm_residual<T>(y2 + (size_t)s_list[i] * geo.y2_bstride, code);
      if (i == 0) s_pt[q] = sm_point<T>(geo, code);
    }
    __syncthreads();
    if (PB > 1 && groups == 1) {
      if (np == 2)
        spread_products<2, 2, 2>(s_pt, yp, cnt, 0, 0, ch, row_base, col_base, nx, ny, lane, wxd, wyd, acc);
      else if (np == 1)
        spread_products<2, 2, 1>(s_pt, yp, cnt, 0, 0, ch, row_base, col_base, nx, ny, lane, wxd, wyd, acc);
    } else if (PB > 1 && groups == 2) {
      if (np == 2)
        spread_products<1, 2, 2>(s_pt, yp, cnt, sub, 0, ch, row_base, col_base, nx, ny, lane, wxd, wyd, acc);
      else if (np == 1)
        spread_products<1, 2, 1>(s_pt, yp, cnt, sub, 0, ch, row_base, col_base, nx, ny, lane, wxd, wyd, acc);
    } else {
      if (PB > 1 && np == 2)
        spread_products<1, 1, 2>(s_pt, yp, cnt, sub >> 1, sub & 1, ch, row_base, col_base, nx, ny, lane, wxd, wyd,
                                 acc);
      else if (np == 1)
        spread_products<1, 1, 1>(s_pt, yp, cnt, sub >> 1, sub & 1, ch, row_base, col_base, nx, ny, lane, wxd, wyd,
                                 acc);
    }
  }
  // even plus odd steps: warp c of the two parities keeps the pair's problem c
  // and hands over the other
  __syncthreads();  // the residuals have been read
  constexpr int kBlkW = PB > 1 ? 4 : 1;  // blocks per warp at most
#pragma unroll
  for (int m = 0; m < kBlkW; ++m)
    if (m < nblk_w)
      *reinterpret_cast<double2*>(s_ex + (warp * kBlkW + m) * 64 + 2 * lane) =
          ch ? make_double2(acc[0][m][0], acc[0][m][1]) : make_double2(acc[1][m][0], acc[1][m][1]);
  __syncthreads();
  const int prob = 2 * pair + ch;
  const int nblk = prob < nact ? nblk_w : 0;
  double d[4][2];  // the problem's blocks 2 mb + nb: [blk0, blk0 + nblk)
#pragma unroll
  for (int m = 0; m < kBlkW; ++m)
    if (m < nblk) {
      const double2 v = *reinterpret_cast<const double2*>(s_ex + ((warp ^ 1) * kBlkW + m) * 64 + 2 * lane);
      d[m][0] = (ch ? acc[1][m][0] : acc[0][m][0]) + v.x;
      d[m][1] = (ch ? acc[1][m][1] : acc[0][m][1]) + v.y;
    }
  constexpr int kPart = 4 * 64;  // doubles of one problem's tile
  if (it.nseg > 1) {
    const size_t cs = (size_t)gridDim.y * PB * kPart;
    double* mine = scratch + (size_t)(it.scratch + it.seg) * cs + ((size_t)blockIdx.y * PB + prob) * kPart;
#pragma unroll
    for (int q = 0; q < kBlkW; ++q)
      if (q < nblk) *reinterpret_cast<double2*>(mine + (blk0 + q) * 64 + 2 * lane) = make_double2(d[q][0], d[q][1]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_ticket = atomicAdd(&tickets[(size_t)it.ticket * gridDim.y + blockIdx.y], 1u);
    __syncthreads();
    if (s_ticket != (unsigned int)(it.nseg - 1)) return;
    __threadfence();
#pragma unroll
    for (int q = 0; q < kBlkW; ++q) d[q][0] = d[q][1] = 0.0;
    for (int sg = 0; sg < it.nseg; ++sg) {
      const double* p = scratch + (size_t)(it.scratch + sg) * cs + ((size_t)blockIdx.y * PB + prob) * kPart;
#pragma unroll
      for (int q = 0; q < kBlkW; ++q)
        if (q < nblk) {
          const double2 v = __ldcg(reinterpret_cast<const double2*>(p + (blk0 + q) * 64 + 2 * lane));
          d[q][0] += v.x;
          d[q][1] += v.y;
        }
    }
    if (threadIdx.x == 0) tickets[(size_t)it.ticket * gridDim.y + blockIdx.y] = 0u;  // for the next launch
  }
  if (nblk == 0) return;
  cplx<T>* gr = gall + (size_t)s_list[prob] * gstride;
#pragma unroll
  for (int q = 0; q < kBlkW; ++q)
    if (q < nblk) sm_store<T>(gr, blk0 + q, d[q][0], d[q][1], row_base, col_base, nx, ny, lane);
}

}  // namespace mf
