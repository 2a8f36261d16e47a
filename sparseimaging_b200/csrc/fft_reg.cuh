// FFT passes of the FP64 operators: a mixed-radix Stockham FFT through
// registers, and the row and column kernels of the NUFFT and of the gridded
// variant on it.
//
// `count` independent transforms of length n per CTA.  A stage of radix R takes
// R points a thread into registers, forms their butterfly and writes them in
// the auto-sorting order (no bit reversal).  The first stage reads its points
// with the caller's `load` (global memory, with the padding, grid correction
// or half-spectrum folding of the pass) and the last hands its results to the
// caller's `store`, so a transform of s stages crosses shared memory s - 1
// times.  Stages read one shared buffer and write the other, one barrier each.
//
// Powers of two in radices of at most 4 in the row passes and 8 in the column
// passes (fft_radices), 3 and 5 in closed form, 7, 11 and 13 as symmetric
// direct sums.  The twiddles of a stage lie
// together, [r - 1][k], so that a warp reads consecutive values (by index over
// the whole table, a warp's reads were scattered and L1 was 64 % busy).
// Forward sign is -1 (exp(-2 pi i jk/n)), unnormalised, matching FFTW's
// convention for the transforms the reference plans
// (c/mfista_nufft_lib.c:609-610, c/mfista_fft_lib.c:246-247).
//
// A thread's arithmetic does not depend on count or on the launch, so results
// do not either.  The FP32 operators keep the radix-4 passes of fft_smem.cuh:
// the corrected solves compare objectives at the level of their FP32 rounding,
// and another order of the same sums moves single accept decisions.
//
// Measured on B200, us per launch, radix 4 through shared memory -> here:
// 64 grids of 512 x 257, columns 172 / 184 -> 90 / 86 (forward / inverse), rows
// 84 / 115 -> 70 / 92; 256 x 129: columns 41 / 41 -> 23 / 21, rows 23 / 27 -> 20 / 23.
#pragma once
#include "common.cuh"
#include "fftvar_ops.cuh"
#include "nufft_ops.cuh"

namespace mf {

// w *= exp(sign i phi), phi given by its cosine and sine
template <typename T> __device__ __forceinline__ cplx<T> crot(cplx<T> a, T c, T s, int sign) {
  return cmul<T>(a, mk<T>(c, sign < 0 ? -s : s));
}

template <typename T, int R> struct Bfly;

template <typename T> struct Bfly<T, 2> {
  static __device__ __forceinline__ void run(cplx<T>* v, int) {
    cplx<T> a = v[0], b = v[1];
    v[0] = cadd<T>(a, b);
    v[1] = csub<T>(a, b);
  }
};

template <typename T> struct Bfly<T, 4> {
  static __device__ __forceinline__ void run(cplx<T>* v, int sign) {
    cplx<T> t0 = cadd<T>(v[0], v[2]), t1 = csub<T>(v[0], v[2]);
    cplx<T> t2 = cadd<T>(v[1], v[3]), t3 = cmul_si<T>(csub<T>(v[1], v[3]), sign);
    v[0] = cadd<T>(t0, t2);
    v[2] = csub<T>(t0, t2);
    v[1] = cadd<T>(t1, t3);
    v[3] = csub<T>(t1, t3);
  }
};

// even and odd halves, then the odd ones turned by w = exp(sign 2 pi i k / R)
template <typename T> struct Bfly<T, 8> {
  static __device__ __forceinline__ void run(cplx<T>* v, int sign) {
    const T h = T(0.7071067811865475244008);
    cplx<T> e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    Bfly<T, 4>::run(e, sign);
    Bfly<T, 4>::run(o, sign);
    o[1] = crot<T>(o[1], h, h, sign);
    o[2] = cmul_si<T>(o[2], sign);
    o[3] = crot<T>(o[3], -h, h, sign);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = cadd<T>(e[k], o[k]);
      v[k + 4] = csub<T>(e[k], o[k]);
    }
  }
};

template <typename T> struct Bfly<T, 3> {
  static __device__ __forceinline__ void run(cplx<T>* v, int sign) {
    const T c3 = T(-0.5), s3 = T(0.86602540378443864676);
    cplx<T> t1 = cadd<T>(v[1], v[2]);
    cplx<T> t2 = csub<T>(v[1], v[2]);
    cplx<T> m1 = mk<T>(v[0].x + c3 * t1.x, v[0].y + c3 * t1.y);
    cplx<T> m2 = cmul_si<T>(mk<T>(s3 * t2.x, s3 * t2.y), sign);
    v[0] = cadd<T>(v[0], t1);
    v[1] = cadd<T>(m1, m2);
    v[2] = csub<T>(m1, m2);
  }
};

template <typename T> struct Bfly<T, 5> {
  static __device__ __forceinline__ void run(cplx<T>* v, int sign) {
    const T c1 = T(0.30901699437494742410), c2 = T(-0.80901699437494742410);
    const T s1 = T(0.95105651629515357212), s2 = T(0.58778525229247312917);
    cplx<T> a1 = cadd<T>(v[1], v[4]), b1 = csub<T>(v[1], v[4]);
    cplx<T> a2 = cadd<T>(v[2], v[3]), b2 = csub<T>(v[2], v[3]);
    cplx<T> r1 = mk<T>(v[0].x + c1 * a1.x + c2 * a2.x, v[0].y + c1 * a1.y + c2 * a2.y);
    cplx<T> r2 = mk<T>(v[0].x + c2 * a1.x + c1 * a2.x, v[0].y + c2 * a1.y + c1 * a2.y);
    cplx<T> i1 = cmul_si<T>(mk<T>(s1 * b1.x + s2 * b2.x, s1 * b1.y + s2 * b2.y), sign);
    cplx<T> i2 = cmul_si<T>(mk<T>(s2 * b1.x - s1 * b2.x, s2 * b1.y - s1 * b2.y), sign);
    v[0] = mk<T>(v[0].x + a1.x + a2.x, v[0].y + a1.y + a2.y);
    v[1] = cadd<T>(r1, i1);
    v[4] = csub<T>(r1, i1);
    v[2] = cadd<T>(r2, i2);
    v[3] = csub<T>(r2, i2);
  }
};

// odd prime R: X_q and X_{R-q} from the sums and differences of v_r and v_{R-r}
template <typename T, int R> struct BflyOdd {
  static __device__ __forceinline__ void run(cplx<T>* v, int sign, const double (&co)[R], const double (&si)[R]) {
    constexpr int H = (R - 1) / 2;
    cplx<T> a[H], b[H], out[R];
    out[0] = v[0];
#pragma unroll
    for (int r = 1; r <= H; ++r) {
      a[r - 1] = cadd<T>(v[r], v[R - r]);
      b[r - 1] = csub<T>(v[r], v[R - r]);
      out[0] = cadd<T>(out[0], a[r - 1]);
    }
#pragma unroll
    for (int q = 1; q <= H; ++q) {
      cplx<T> m = v[0], d = mk<T>(0, 0);
#pragma unroll
      for (int r = 1; r <= H; ++r) {
        const T c = T(co[(r * q) % R]), s = T(si[(r * q) % R]);
        m = mk<T>(m.x + c * a[r - 1].x, m.y + c * a[r - 1].y);
        d = mk<T>(d.x + s * b[r - 1].x, d.y + s * b[r - 1].y);
      }
      d = cmul_si<T>(d, sign);
      out[q] = cadd<T>(m, d);
      out[R - q] = csub<T>(m, d);
    }
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = out[q];
  }
};
template <typename T> struct Bfly<T, 7> {
  static __device__ __forceinline__ void run(cplx<T>* v, int sign) {
    constexpr double c[7] = {1.0, 0.623489801858733530525, -0.2225209339563144042889, -0.9009688679024191262361,
                             -0.9009688679024191262361, -0.2225209339563144042889, 0.623489801858733530525};
    constexpr double s[7] = {0.0, 0.7818314824680298087084, 0.9749279121818236070181, 0.4338837391175581204758,
                             -0.4338837391175581204758, -0.9749279121818236070181, -0.7818314824680298087084};
    BflyOdd<T, 7>::run(v, sign, c, s);
  }
};
template <typename T> struct Bfly<T, 11> {
  static __device__ __forceinline__ void run(cplx<T>* v, int sign) {
    constexpr double c[11] = {1.0, 0.8412535328311811688618, 0.4154150130018864255293, -0.1423148382732851404438,
                              -0.6548607339452850640569, -0.9594929736144973898904, -0.9594929736144973898904,
                              -0.6548607339452850640569, -0.1423148382732851404438, 0.4154150130018864255293,
                              0.8412535328311811688618};
    constexpr double s[11] = {0.0, 0.5406408174555975821076, 0.9096319953545183714117, 0.9898214418809327323761,
                              0.755749574354258283774, 0.2817325568414296977114, -0.2817325568414296977114,
                              -0.755749574354258283774, -0.9898214418809327323761, -0.9096319953545183714117,
                              -0.5406408174555975821076};
    BflyOdd<T, 11>::run(v, sign, c, s);
  }
};
template <typename T> struct Bfly<T, 13> {
  static __device__ __forceinline__ void run(cplx<T>* v, int sign) {
    constexpr double c[13] = {1.0, 0.8854560256532098959004, 0.5680647467311558025118, 0.1205366802553230533491,
                              -0.3546048870425356259696, -0.7485107481711010986346, -0.970941817426052027157,
                              -0.970941817426052027157, -0.7485107481711010986346, -0.3546048870425356259696,
                              0.1205366802553230533491, 0.5680647467311558025118, 0.8854560256532098959004};
    constexpr double s[13] = {0.0, 0.464723172043768545656, 0.8229838658936563945796, 0.9927088740980539928008,
                              0.9350162426854148234398, 0.6631226582407952023768, 0.2393156642875577671488,
                              -0.2393156642875577671488, -0.6631226582407952023768, -0.9350162426854148234398,
                              -0.9927088740980539928008, -0.8229838658936563945796, -0.464723172043768545656};
    BflyOdd<T, 13>::run(v, sign, c, s);
  }
};

// quotient and remainder by a length that is mostly a power of two
struct LenDiv {
  int n, sh;
  __device__ __forceinline__ explicit LenDiv(int m) {
    n = m;
    sh = (m & (m - 1)) == 0 ? __popc(m - 1) : -1;
  }
  __device__ __forceinline__ int div(int t) const { return sh >= 0 ? t >> sh : t / n; }
};

// One radix-R stage: thread items over (transform, j), the transforms running
// fastest with kCols (neighbouring lanes on neighbouring columns), else j.
template <typename T, int R, bool kCols, class Load, class Store>
__device__ __forceinline__ void fft_stage(int n, int count, int Ns, const cplx<T>* __restrict__ tw, int sign, Load load,
                                          Store store) {
  const int nR = n / R;
  const LenDiv inner(kCols ? count : nR), dn(Ns);
  for (int t = threadIdx.x; t < count * nR; t += blockDim.x) {
    const int hi = inner.div(t), lo = t - hi * inner.n;
    const int tr = kCols ? lo : hi, j = kCols ? hi : lo;
    const int jq = dn.div(j), k = j - jq * Ns;
    cplx<T> v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = load(tr, j + r * nR);
    if (Ns > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) {
        cplx<T> w = tw[(r - 1) * Ns + k];
        if (sign > 0) w.y = -w.y;
        v[r] = cmul<T>(v[r], w);
      }
    }
    Bfly<T, R>::run(v, sign);
    const int base = jq * Ns * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) store(tr, base + r * Ns, v[r]);
  }
}

// Where the transforms lie in a shared buffer: transform tr, element i at
// tr ld + i + (i >> psh).  Rows (j fastest) are padded by one element in 128
// bytes where the buffers allow it (psh < 31): a first stage writes with a
// stride of R.  Columns need none: neighbouring lanes are ld apart.
struct FftLay {
  int ld, psh;
  __device__ __forceinline__ int at(int tr, int i) const { return tr * ld + i + (i >> psh); }
};

// radices whose first or last stage exchanges with global memory
__host__ __device__ __forceinline__ bool fft_fused(int r) { return r == 8 || r == 5 || r == 4; }

// All stages.  With kToSmem the result stays in the returned buffer (after a
// barrier); else every element goes to `store`, and the returned pointer is
// null.  `a` and `b` may be read and written by the whole CTA; no barrier is
// needed before the call when they have not been used yet.
template <typename T, bool kCols, bool kToSmem, class Load, class Store>
__device__ __forceinline__ cplx<T>* fft_run(const FftDev<T>& p, int count, int sign, cplx<T>* a, cplx<T>* b, FftLay lay,
                                            Load load, Store store) {
  const int n = p.n;
  cplx<T>*src = a, *dst = b;
  const cplx<T>* tw = p.tw;
  auto from = [&](int tr, int i) { return src[lay.at(tr, i)]; };
  auto to = [&](int tr, int i, cplx<T> v) { dst[lay.at(tr, i)] = v; };
  auto swap = [&]() {
    __syncthreads();
    cplx<T>* q = src;
    src = dst;
    dst = q;
  };
  auto move = [&](auto&& f) {  // f(tr, i) for every element
    const LenDiv inner(kCols ? count : n);
    for (int t = threadIdx.x; t < count * n; t += blockDim.x) {
      const int hi = inner.div(t), lo = t - hi * inner.n;
      if (kCols) f(lo, hi);
      else f(hi, lo);
    }
  };
  int s = 0, Ns = 1, last = p.nst;
  // first stage from global memory, if its radix has a fused instance
  switch (p.nst > 1 ? p.radix[0] : 0) {
    case 8:
      if constexpr (kCols) fft_stage<T, 8, kCols>(n, count, 1, tw, sign, load, to);  // rows have none
      s = 1;
      break;
    case 5: fft_stage<T, 5, kCols>(n, count, 1, tw, sign, load, to); s = 1; break;
    case 4: fft_stage<T, 4, kCols>(n, count, 1, tw, sign, load, to); s = 1; break;
    default: move([&](int tr, int i) { to(tr, i, load(tr, i)); });
  }
  swap();
  if (s) {
    Ns = p.radix[0];
    tw += Ns - 1;
  }
  if (!kToSmem && s && fft_fused(p.radix[p.nst - 1])) last = p.nst - 1;
  for (; s < last; ++s) {
    const int R = p.radix[s];
    switch (R) {
      case 8:
        if constexpr (kCols) fft_stage<T, 8, kCols>(n, count, Ns, tw, sign, from, to);
        break;
      case 4: fft_stage<T, 4, kCols>(n, count, Ns, tw, sign, from, to); break;
      case 2: fft_stage<T, 2, kCols>(n, count, Ns, tw, sign, from, to); break;
      case 3: fft_stage<T, 3, kCols>(n, count, Ns, tw, sign, from, to); break;
      case 5: fft_stage<T, 5, kCols>(n, count, Ns, tw, sign, from, to); break;
      case 7: fft_stage<T, 7, kCols>(n, count, Ns, tw, sign, from, to); break;
      case 11: fft_stage<T, 11, kCols>(n, count, Ns, tw, sign, from, to); break;
      default: fft_stage<T, 13, kCols>(n, count, Ns, tw, sign, from, to); break;
    }
    swap();
    tw += (R - 1) * Ns;
    Ns *= R;
  }
  if (kToSmem) return src;
  if (last == p.nst) {
    move([&](int tr, int i) { store(tr, i, from(tr, i)); });
    return nullptr;
  }
  switch (p.radix[last]) {
    case 8:
      if constexpr (kCols) fft_stage<T, 8, kCols>(n, count, Ns, tw, sign, from, store);
      break;
    case 5: fft_stage<T, 5, kCols>(n, count, Ns, tw, sign, from, store); break;
    default: fft_stage<T, 4, kCols>(n, count, Ns, tw, sign, from, store); break;
  }
  return nullptr;
}

// The radices of length n in stage order (0: a prime factor above 13; no int
// has more than kMaxStages of them): powers of two in as few radices up to
// 2^log2max as possible and as even as possible; the two largest with an
// instance that exchanges with global memory (fft_fused) go first and last.
// Columns take radices up to 8 and rows up to 4.  Larger ones make fewer trips
// through shared memory but leave a CTA's few transforms to fewer threads, each
// with a longer chain: an iteration of one problem took 115 / 119 us at 64 /
// 128 pixels a side with 16 and 8, 107 / 111 with 8 and 4; 32 problems at 256
// took 312 either way.  (The lengths decide alone: a problem's values may not
// depend on its batch.)
constexpr int kColsLog2Max = 3, kRowsLog2Max = 2;

inline int fft_radices(int n, int (&radix)[kMaxStages], int log2max) {
  int list[64], m = 0, p2 = 0;
  while (n % 2 == 0) {
    ++p2;
    n /= 2;
  }
  if (p2) {
    const int k = (p2 + log2max - 1) / log2max;
    for (int i = 0; i < k; ++i) list[m++] = 1 << (p2 / k + (i < p2 % k ? 1 : 0));
  }
  for (int f : {3, 5, 7, 11, 13})
    while (n % f == 0) {
      list[m++] = f;
      n /= f;
    }
  if (n > 1) return 0;
  auto key = [](int r) { return (fft_fused(r) ? 100 : 0) + r; };
  for (int i = 1; i < m; ++i)  // fused first, by falling radix
    for (int j = i; j > 0 && key(list[j]) > key(list[j - 1]); --j) {
      const int t = list[j];
      list[j] = list[j - 1];
      list[j - 1] = t;
    }
  if (m > 1 && fft_fused(list[1])) {  // the second of them to the end
    const int t = list[1];
    for (int i = 1; i + 1 < m; ++i) list[i] = list[i + 1];
    list[m - 1] = t;
  }
  for (int i = 0; i < m; ++i) radix[i] = list[i];
  return m;
}

constexpr size_t kRowsPadMax = 96 * 1024;  // larger row buffers go without padding

// Shared layouts of the FFT passes.  Rows are padded (FftLay) where both
// buffers then take at most kRowsPadMax (a single row: half of it, so that no
// length loses its place in the default shared memory), the host sizing them
// alike.
constexpr int kRowsPsh = 3;  // an element in eight of 16 bytes
template <typename T> __host__ __device__ __forceinline__ size_t rows_bytes(int h, int rows, int psh) {
  return 2 * sizeof(cplx<T>) * (size_t)rows * (h + 1 + (h >> psh));
}
template <typename T> __host__ __device__ __forceinline__ FftLay rows_lay(int h, int rows) {
  const size_t most = rows == 1 ? kRowsPadMax / 2 : kRowsPadMax;
  const int psh = rows_bytes<T>(h, rows, kRowsPsh) <= most ? kRowsPsh : 31;
  return FftLay{h + 1 + (h >> psh), psh};
}
template <typename T> __host__ __device__ __forceinline__ size_t rows_smem_bytes(int h, int rows) {
  return 2 * sizeof(cplx<T>) * (size_t)rows * rows_lay<T>(h, rows).ld;
}
template <typename T> __host__ __device__ __forceinline__ FftLay cols_lay(int n) {
  return FftLay{n + 1, 31};
}
template <typename T> __host__ __device__ __forceinline__ size_t cols_smem_bytes(int n, int cols) {
  return 2 * sizeof(cplx<T>) * (size_t)cols * cols_lay<T>(n).ld;
}


// k_nufft_rows_fwd
template <typename T>
__global__ void __launch_bounds__(256, 2) k_nufft_rows_fwd_reg(const double* __restrict__ xall, long xstride, const double* __restrict__ e4,
                                 cplx<T>* __restrict__ gall, long gstride, int nx, int ny, const __grid_constant__ FftDev<T> fh,
                                 const cplx<T>* __restrict__ tw2h, const ProbState* __restrict__ st, int gate,
                                 int rows_per_cta, const double* __restrict__ suball, DynUnits dyn) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FftWork w;
  if (!fft_work(dyn, st, gate, nx, rows_per_cta, w)) return;
  const int b = w.b;
  const int h = ny;
  const FftLay lay = rows_lay<T>(h, rows_per_cta);
  cplx<T>* A = reinterpret_cast<cplx<T>*>(smem_raw);
  cplx<T>* Bf = A + (size_t)rows_per_cta * lay.ld;
  const double* x = xall + (size_t)b * xstride;
  // defect correction: transform x - x_anchor (the anchor's model is added
  // back in FP64 at the interpolation)
  const double* sub = suball ? suball + (size_t)b * xstride : nullptr;
  cplx<T>* g = gall + (size_t)b * gstride;
  int i0 = w.u0;
  int nrows = min(w.units, nx - i0);
  auto pixel = [&](int i, int m) -> T {
    const int j = uncentre_index(m, ny);
    if (j < 0) return T(0);
    const size_t f = (size_t)i * ny + j;
    return (T)((sub ? x[f] - sub[f] : x[f]) * e4[f]);
  };
  cplx<T>* Z = fft_run<T, false, true>(
      fh, nrows, -1, A, Bf, lay, [&](int rr, int m) { return mk<T>(pixel(i0 + rr, 2 * m), pixel(i0 + rr, 2 * m + 1)); },
      [](int, int, cplx<T>) {});
  // X[k] = 1/2[(Z_k + conj Z_{h-k}) - i W^k (Z_k - conj Z_{h-k})], W = exp(-2 pi i / 2h)
  // a warp per row, lanes along its h + 1 outputs (no division by h + 1)
  for (int rr = (int)(threadIdx.x >> 5); rr < nrows; rr += (int)(blockDim.x >> 5))
    for (int k = (int)(threadIdx.x & 31); k <= h; k += 32) {
    cplx<T> zk = Z[lay.at(rr, k == h ? 0 : k)];
    cplx<T> zc = cconj<T>(Z[lay.at(rr, k == 0 ? 0 : h - k)]);
    cplx<T> e = cadd<T>(zk, zc);
    cplx<T> o = csub<T>(zk, zc);
    cplx<T> wo = cmul_si<T>(cmul<T>(tw2h[k], o), -1);
    cplx<T> X = mk<T>(T(0.5) * (e.x + wo.x), T(0.5) * (e.y + wo.y));
    int row = centre_index(i0 + rr, nx);
    g[(size_t)row * (ny + 1) + k] = X;
  }
}

// k_nufft_cols
template <typename T>
__global__ void __launch_bounds__(256, 2) k_nufft_cols_reg(cplx<T>* __restrict__ gall, long gstride, int nx, int ny, const __grid_constant__ FftDev<T> f2x, int sign,
                             int cols_per_cta, int load_pruned, int store_pruned,
                             const ProbState* __restrict__ st, int gate, DynUnits dyn) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FftWork w;
  if (!fft_work(dyn, st, gate, ny + 1, cols_per_cta, w)) return;
  const int b = w.b;
  const int ncol = ny + 1;
  const FftLay lay = cols_lay<T>(2 * nx);
  cplx<T>* A = reinterpret_cast<cplx<T>*>(smem_raw);
  cplx<T>* Bf = A + (size_t)cols_per_cta * lay.ld;
  const int c0 = w.u0;
  cplx<T>* g = gall + (size_t)b * gstride + c0;
  fft_run<T, true, false>(
      f2x, min(w.units, ncol - c0), sign, A, Bf, lay,
      [&](int cc, int r) {
        return (!load_pruned || uncentre_index(r, nx) >= 0) ? g[(size_t)r * ncol + cc] : mk<T>(0, 0);
      },
      [&](int cc, int r, cplx<T> v) {
        if (!store_pruned || uncentre_index(r, nx) >= 0) g[(size_t)r * ncol + cc] = v;
      });
}

// k_nufft_rows_inv
template <typename T>
__global__ void __launch_bounds__(256, 2) k_nufft_rows_inv_reg(const cplx<T>* __restrict__ gall, long gstride, double* __restrict__ dall,
                                 long xstride, const double* __restrict__ e4, int nx, int ny, double inv_mm,
                                 const __grid_constant__ FftDev<T> fh, const cplx<T>* __restrict__ tw2h, TsvFuse tf, Partials part,
                                 int qtsv, const ProbState* __restrict__ st, int gate, int rows_per_cta,
                                 DynUnits dyn) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double sh[32];
  FftWork w;
  if (!fft_work(dyn, st, gate, nx, rows_per_cta, w)) return;
  const int b = w.b;
  const int h = ny;
  const FftLay lay = rows_lay<T>(h, rows_per_cta);
  cplx<T>* A = reinterpret_cast<cplx<T>*>(smem_raw);
  cplx<T>* Bf = A + (size_t)rows_per_cta * lay.ld;
  const cplx<T>* g = gall + (size_t)b * gstride;
  double* dfdx = dall + (size_t)b * xstride;
  // (the spread mapping only without TSV partials: their slots are the grid's x)
  int i0 = w.u0;
  int nrows = min(w.units, nx - i0);
  const ProbParams& pp = tf.prm[b];
  bool fuse = tf.z != nullptr && pp.lambda_tsv > 0.0;
  const double* z = fuse ? tf.z + (size_t)b * xstride : nullptr;
  double acc[1] = {0.0};
  auto pixel = [&](int i, int c, T v) {  // padded column c of image row i
    const int j = uncentre_index(c, ny);
    if (j < 0) return;
    const int f = i * ny + j;
    double d = (double)v * e4[f] * inv_mm;
    if (fuse) {
      d = d + dtsv_at(z, f, tf.NX, tf.NY) * (-pp.lambda_tsv);
      acc[0] += tsv_terms_at(z, f, tf.NX, tf.NY);
    }
    dfdx[f] = d;
  };
  // Z[k] = (X_k + conj X_{h-k}) + i conj(W^k) (X_k - conj X_{h-k}); DC/Nyquist real parts only
  fft_run<T, false, false>(
      fh, nrows, +1, A, Bf, lay,
      [&](int rr, int k) {
        const cplx<T>* grow = g + (size_t)centre_index(i0 + rr, nx) * (ny + 1);
        cplx<T> xk = grow[k];
        cplx<T> xc = grow[h - k];
        if (k == 0) {
          xk.y = 0;
          xc.y = 0;
        }
        xc = cconj<T>(xc);
        cplx<T> o = cmul_si<T>(cmul<T>(cconj<T>(tw2h[k]), csub<T>(xk, xc)), 1);
        return cadd<T>(cadd<T>(xk, xc), o);
      },
      [&](int rr, int c, cplx<T> v) {
        pixel(i0 + rr, 2 * c, v.x);
        pixel(i0 + rr, 2 * c + 1, v.y);
      });
  if (qtsv >= 0) {
    block_sum<1>(acc, sh);
    if (threadIdx.x == 0) part.at(qtsv, b)[blockIdx.x] = acc[0];
  }
}

// k_fftv_rows_fwd (fftvar_ops.cuh)
template <typename T>
__global__ void __launch_bounds__(256, 2) k_fftv_rows_fwd_reg(const double* __restrict__ xall, long xstride, cplx<T>* __restrict__ hall,
                                long hstride, int nx, int ny, const __grid_constant__ FftDev<T> fh, const cplx<T>* __restrict__ tw2h,
                                const ProbState* __restrict__ st, int gate, int rows_per_cta,
                                const double* __restrict__ suball) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int b = blockIdx.y;
  if (!gate_ok(st[b], gate)) return;
  const int h = ny / 2, nyh = h + 1;
  const FftLay lay = rows_lay<T>(h, rows_per_cta);
  cplx<T>* A = reinterpret_cast<cplx<T>*>(smem_raw);
  cplx<T>* Bf = A + (size_t)rows_per_cta * lay.ld;
  const double* x = xall + (size_t)b * xstride;
  cplx<T>* H = hall + (size_t)b * hstride;
  int i0 = blockIdx.x * rows_per_cta;
  int nrows = min(rows_per_cta, nx - i0);
  const double* sub = suball ? suball + (size_t)b * xstride : nullptr;
  cplx<T>* Z = fft_run<T, false, true>(
      fh, nrows, -1, A, Bf, lay,
      [&](int rr, int m) {
        const size_t f = (size_t)(i0 + rr) * ny + 2 * m;
        double x0 = x[f], x1 = x[f + 1];
        if (sub) {
          x0 -= sub[f];
          x1 -= sub[f + 1];
        }
        return mk<T>((T)x0, (T)x1);
      },
      [](int, int, cplx<T>) {});
  for (int t = threadIdx.x; t < nrows * nyh; t += blockDim.x) {
    int rr = t / nyh, k = t - rr * nyh;
    cplx<T> zk = Z[lay.at(rr, k == h ? 0 : k)];
    cplx<T> zc = cconj<T>(Z[lay.at(rr, k == 0 ? 0 : h - k)]);
    cplx<T> e = cadd<T>(zk, zc);
    cplx<T> wo = cmul_si<T>(cmul<T>(tw2h[k], csub<T>(zk, zc)), -1);
    H[(size_t)(i0 + rr) * nyh + k] = mk<T>(T(0.5) * (e.x + wo.x), T(0.5) * (e.y + wo.y));
  }
}

// k_fftv_cols
template <typename T>
__global__ void __launch_bounds__(256, 2) k_fftv_cols_reg(cplx<T>* __restrict__ hall, long hstride, int nx, int nyh, const __grid_constant__ FftDev<T> fnx, int sign,
                            int cols_per_cta, FftVarGeom geo, double sqrtn, const ProbState* __restrict__ st,
                            int gate, Partials part, int qchi, int store_grad, const double2* __restrict__ base,
                            double2* __restrict__ raw_out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double sh[32];
  int b = blockIdx.y;
  if (!gate_ok(st[b], gate)) return;
  const FftLay lay = cols_lay<T>(nx);
  cplx<T>* A = reinterpret_cast<cplx<T>*>(smem_raw);
  cplx<T>* Bf = A + (size_t)cols_per_cta * lay.ld;
  cplx<T>* H = hall + (size_t)b * hstride;
  int c0 = blockIdx.x * cols_per_cta;
  double acc[1] = {0.0};
  const double* mask = geo.mask_h + (size_t)b * geo.geo_stride;
  const double2* yf = geo.yf_h + (size_t)b * geo.geo_stride;
  fft_run<T, true, false>(
      fnx, min(cols_per_cta, nyh - c0), sign, A, Bf, lay, [&](int cc, int r) { return H[(size_t)r * nyh + c0 + cc]; },
      [&](int cc, int r, cplx<T> v) {
        const int k = c0 + cc;
        const size_t e = (size_t)r * nyh + k;
        if (raw_out) {
          raw_out[(size_t)b * hstride + e] = make_double2((double)v.x, (double)v.y);
        } else if (qchi >= 0) {
          const double mk_ = mask[e];
          const double2 y = yf[e];
          double vx = (double)v.x, vy = (double)v.y;
          if (base) {
            const double2 a = base[(size_t)b * hstride + e];
            vx += a.x;
            vy += a.y;
          }
          const double rr = y.x - mk_ * vx / sqrtn;
          const double ri = y.y - mk_ * vy / sqrtn;
          const double w = (k == 0 || k == nyh - 1) ? 1.0 : 2.0;
          acc[0] += w * (rr * rr + ri * ri);
          if (store_grad) {
            const double s = mk_ / (2 * sqrtn);
            H[e] = mk<T>((T)(rr * s), (T)(ri * s));
          }
        } else {
          H[e] = v;
        }
      });
  if (qchi >= 0) {
    block_sum<1>(acc, sh);
    if (threadIdx.x == 0) part.at(qchi, b)[blockIdx.x] = acc[0];
  }
}

// k_fftv_rows_inv
template <typename T>
__global__ void __launch_bounds__(256, 2) k_fftv_rows_inv_reg(const cplx<T>* __restrict__ hall, long hstride, double* __restrict__ dall,
                                long xstride, int nx, int ny, const __grid_constant__ FftDev<T> fh, const cplx<T>* __restrict__ tw2h,
                                const double* __restrict__ zall, const ProbParams* __restrict__ prm,
                                int tsvNX, int tsvNY, Partials part, int qtsv, const ProbState* __restrict__ st,
                                int gate, int rows_per_cta) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double sh[32];
  int b = blockIdx.y;
  if (!gate_ok(st[b], gate)) return;
  const int h = ny / 2, nyh = h + 1;
  const FftLay lay = rows_lay<T>(h, rows_per_cta);
  cplx<T>* A = reinterpret_cast<cplx<T>*>(smem_raw);
  cplx<T>* Bf = A + (size_t)rows_per_cta * lay.ld;
  const cplx<T>* H = hall + (size_t)b * hstride;
  double* dfdx = dall + (size_t)b * xstride;
  int i0 = blockIdx.x * rows_per_cta;
  int nrows = min(rows_per_cta, nx - i0);
  const ProbParams& pp = prm[b];
  bool fuse = zall != nullptr && pp.lambda_tsv > 0.0;
  const double* z = fuse ? zall + (size_t)b * xstride : nullptr;
  double acc[1] = {0.0};
  auto pixel = [&](int f, T v) {
    double d = (double)v;
    if (fuse) {
      d = d + dtsv_at(z, f, tsvNX, tsvNY) * (-pp.lambda_tsv);
      acc[0] += tsv_terms_at(z, f, tsvNX, tsvNY);
    }
    dfdx[f] = d;
  };
  fft_run<T, false, false>(
      fh, nrows, +1, A, Bf, lay,
      [&](int rr, int k) {
        const cplx<T>* hr = H + (size_t)(i0 + rr) * nyh;
        cplx<T> xk = hr[k];
        cplx<T> xc = hr[h - k];
        if (k == 0) {
          xk.y = 0;
          xc.y = 0;
        }
        xc = cconj<T>(xc);
        cplx<T> o = cmul_si<T>(cmul<T>(cconj<T>(tw2h[k]), csub<T>(xk, xc)), 1);
        return cadd<T>(cadd<T>(xk, xc), o);
      },
      [&](int rr, int c, cplx<T> v) {
        const int f = (i0 + rr) * ny + 2 * c;
        pixel(f, v.x);
        pixel(f + 1, v.y);
      });
  if (qtsv >= 0) {
    block_sum<1>(acc, sh);
    if (threadIdx.x == 0) part.at(qtsv, b)[blockIdx.x] = acc[0];
  }
}

}  // namespace mf
