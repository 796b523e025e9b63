// Persistent, TMA-pipelined batched FFT pass for compile-time line lengths.
//
// Same tile as fft.cu -- one grid line of N points times W consecutive states,
// 256-byte rows (or W consecutive columns of a flattened view; whole z-lines in fftz_kernel) -- but:
//   * tiles stream through an NS-stage shared-memory ring: one elected thread
//     issues cp.async.bulk.tensor (TMA) loads NS tiles ahead and a TMA store per
//     finished tile, so HBM traffic overlaps the arithmetic of the other stages;
//   * the line DFT is a two-level Cooley-Tukey N = N1 x N2 done in registers
//     (N1- and N2-point codelets, composite ones from radix 2,3,4,5,8 with
//     twiddles from a shared-memory copy of the line's table), with one
//     shared-memory exchange instead of one per radix;
//   * all index arithmetic is compile-time except the per-tile line decomposition.
// Every mbarrier wait is bounded (about 2 s by %globaltimer); on expiry the CTA
// raises the context's error flag and leaves its tile loop.

#pragma once

#include <cuda.h>

#include "fft2_lengths.h"
#include "fft_common.cuh"
#include "ptx.cuh"

namespace inqb {
namespace v2 {

enum Variant {
  FWD_STORE = 0, INV_STORE = 1, MID_KIN = 2, INV_FINAL = 3, FWD_VPSI = 4, FWD_LAPLADD = 5,
  // the same passes with the frequencies along the pass axis in digit-reversed order (position
  // k2 + N2 k1 holds frequency k1 + N1 k2): forward output, inverse input
  FWD_PERM = 6, INV_PERM = 7, INV_FINAL_PERM = 8
};

constexpr int base_var(int v) { return v == FWD_PERM ? FWD_STORE : (v == INV_PERM ? INV_STORE : (v == INV_FINAL_PERM ? INV_FINAL : v)); }
constexpr bool is_perm(int v) { return v >= FWD_PERM; }
constexpr bool has_aux(int v) { return base_var(v) == INV_FINAL || v == FWD_LAPLADD; }

template <int N> struct Split { static constexpr int N1 = 0, N2 = 0; };
#define INQB_X(N, A, B) \
  template <> struct Split<N> { static constexpr int N1 = A, N2 = B; };
INQB_FFT2_LENGTHS(INQB_X)
#undef INQB_X

constexpr int first_factor(int M) {
  const int f[6] = {8, 4, 2, 3, 5, 7};
  for (int i = 0; i < 6; i++)
    if (M % f[i] == 0 && M != f[i]) return f[i];
  return M;
}

// ------------------------------------------------------------------ PTX helpers

using ptx::global_ns;
using ptx::mbar_init;
using ptx::mbar_init_fence;
using ptx::mbar_try_wait;
using ptx::smem_u32;
using ptx::mbar_expect_tx;
__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, uint64_t *bar, int c0, int c1, int c2,
                                            int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::
          "r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap *map, const void *src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
using ptx::bulk_commit;
using ptx::bulk_wait0;
using ptx::bulk_wait_read0;
using ptx::fence_proxy_async;

// ------------------------------------------------------------------ register codelets (compile-time size)

template <int DIR, typename T> __device__ __forceinline__ T mmi(T a) {  // a * (-i * DIR)
  if constexpr (DIR > 0) return mk<T>(a.y, -a.x);
  else return mk<T>(-a.y, a.x);
}
template <int DIR, typename T> __device__ __forceinline__ T twid(T t) {
  if constexpr (DIR < 0) t.y = -t.y;
  return t;
}

// cos(2 pi m / r) and sin(2 pi m / r), m = 1..(r-1)/2, for the odd prime codelets
// Single-precision products by a constant or a twiddle factor.  The float roundings of sqrt(1/2),
// sin(pi/3) and of many table twiddles fall on the same side often enough to shrink every transform
// by ~2e-8 (an energy bias that reaches ~1e-6 Ha in <psi|H|psi>).  With c = c_hi + c_lo (c_lo the
// float rounding remainder), fma(x, c_hi, x * c_lo) leaves only an unbiased rounding; double products
// need no correction.
template <typename T> __device__ __forceinline__ T kscale(T a, double c) {
  using R = decltype(T::x);
  if constexpr (sizeof(R) == 4) {
    const float hi = float(c), lo = float(c - double(float(c)));
    if (lo == 0.0f) return mk<T>(a.x * hi, a.y * hi);
    return mk<T>(__fmaf_rn(a.x, hi, a.x * lo), __fmaf_rn(a.y, hi, a.y * lo));
  } else {
    return mk<T>(a.x * R(c), a.y * R(c));
  }
}
// a times twiddle `idx` of the line table; single-precision tables interleave each twiddle's float
// part and float remainder (one 16-byte load).
template <int DIR, int N, typename T> __device__ __forceinline__ T twmul(T a, const T *__restrict__ tw, int idx) {
  using R = decltype(T::x);
  if constexpr (sizeof(R) == 4) {
    const float4 q = reinterpret_cast<const float4 *>(tw)[idx];
    const T h = twid<DIR>(mk<T>(q.x, q.y)), l = twid<DIR>(mk<T>(q.z, q.w));
    const R lr = __fmaf_rn(-a.y, l.y, a.x * l.x), li = __fmaf_rn(a.y, l.x, a.x * l.y);
    return mk<T>(__fmaf_rn(a.x, h.x, __fmaf_rn(-a.y, h.y, lr)), __fmaf_rn(a.x, h.y, __fmaf_rn(a.y, h.x, li)));
  } else {
    return cmul(a, twid<DIR>(tw[idx]));
  }
}
// entries of the line's twiddle table in shared memory: N, or 2N for single precision
template <typename R> constexpr int tw_entries(int N) { return sizeof(R) == 4 ? 2 * N : N; }

template <int RR> __host__ __device__ constexpr double odd_cos(int m) {
  if (RR == 3) return -0.5;
  if (RR == 5) return m == 1 ? 0.30901699437494742410229341718281905886 : -0.80901699437494742410229341718281905886;
  return m == 1 ? 0.62348980185873353052500488400423981063
                : (m == 2 ? -0.22252093395631440428890256449679475947 : -0.90096886790241912623610231950744505117);
}
template <int RR> __host__ __device__ constexpr double odd_sin(int m) {
  if (RR == 3) return 0.86602540378443864676372317075293618347;
  if (RR == 5) return m == 1 ? 0.95105651629515357211643933337938214341 : 0.58778525229247312916870595463907276860;
  return m == 1 ? 0.78183148246802980870844452667405775023
                : (m == 2 ? 0.97492791218182360701813168299393121723 : 0.43388373911755812047576833284835875461);
}

// cos and sin of 2 pi p / q, evaluated at compile time: the angle is folded into [0, pi/4] by exact
// integer reflections, multiples of 30 and 45 degrees take exact values, the rest a Taylor series
// (x <= pi/4, terms to x^27).
struct CosSin {
  double c, s;
};
__host__ __device__ constexpr double taylor_sin(double x) {
  double term = x, sum = x;
  for (int n = 1; n < 14; n++) {
    term = -term * x * x / double((2 * n) * (2 * n + 1));
    sum += term;
  }
  return sum;
}
__host__ __device__ constexpr double taylor_cos(double x) {
  double term = 1.0, sum = 1.0;
  for (int n = 1; n < 14; n++) {
    term = -term * x * x / double((2 * n - 1) * (2 * n));
    sum += term;
  }
  return sum;
}
__host__ __device__ constexpr CosSin cos_sin_turn(long long p, long long q) {
  p %= q;
  if (p < 0) p += q;
  bool neg_s = false, neg_c = false, swap = false;
  if (2 * p > q) { p = q - p; neg_s = true; }              // 2 pi - theta
  if (4 * p > q) { p = q - 2 * p; q = 2 * q; neg_c = true; }  // pi - theta
  if (8 * p > q) { p = q - 4 * p; q = 4 * q; swap = true; }   // pi / 2 - theta
  double c = taylor_cos(6.283185307179586476925286766559 * double(p) / double(q));
  double s = taylor_sin(6.283185307179586476925286766559 * double(p) / double(q));
  if (p == 0) { c = 1.0; s = 0.0; }
  if (8 * p == q) c = s = 0.70710678118654752440084436210484903928;
  if (12 * p == q) { c = 0.86602540378443864676372317075293618347; s = 0.5; }
  if (swap) { const double t = c; c = s; s = t; }
  if (neg_c) c = -c;
  if (neg_s) s = -s;
  return CosSin{c, s};
}

// a times the compile-time twiddle W_M^TT = exp(-2 pi i TT DIR / M).  Single precision: the same
// compensated product as twmul (twiddle = float part + float remainder), with the terms of exact
// parts dropped; unit twiddles are sign changes and swaps.
template <int DIR, int M, int TT, typename T> __device__ __forceinline__ T tw_const(T a) {
  using R = decltype(T::x);
  constexpr CosSin cs = cos_sin_turn(TT, M);
  constexpr double tx = cs.c, ty = -double(DIR) * cs.s;
  if constexpr (ty == 0.0) {
    if constexpr (tx > 0.0) return a;
    else return mk<T>(-a.x, -a.y);
  } else if constexpr (tx == 0.0) {
    if constexpr (ty > 0.0) return mk<T>(-a.y, a.x);
    else return mk<T>(a.y, -a.x);
  } else if constexpr (sizeof(R) == 4) {
    constexpr float hx = float(tx), hy = float(ty);
    constexpr float lx = float(tx - double(hx)), ly = float(ty - double(hy));
    R lr, li;
    if constexpr (lx == 0.0f && ly == 0.0f) {
      lr = R(0);
      li = R(0);
      return mk<T>(__fmaf_rn(a.x, hx, -a.y * hy), __fmaf_rn(a.x, hy, a.y * hx));
    } else if constexpr (ly == 0.0f) {
      lr = a.x * lx;
      li = a.y * lx;
    } else if constexpr (lx == 0.0f) {
      lr = -a.y * ly;
      li = a.x * ly;
    } else {
      lr = __fmaf_rn(-a.y, ly, a.x * lx);
      li = __fmaf_rn(a.y, lx, a.x * ly);
    }
    return mk<T>(__fmaf_rn(a.x, hx, __fmaf_rn(-a.y, hy, lr)), __fmaf_rn(a.x, hy, __fmaf_rn(a.y, hx, li)));
  } else {
    return mk<T>(a.x * R(tx) - a.y * R(ty), a.x * R(ty) + a.y * R(tx));
  }
}
// tw_const with the exponent known only after unrolling (folds to one product once t is constant)
template <int DIR, int M, int TT = 1, typename T> __device__ __forceinline__ T tw_const_at(T a, int t) {
  if constexpr (TT >= M) return a;
  else return t == TT ? tw_const<DIR, M, TT>(a) : tw_const_at<DIR, M, TT + 1>(a, t);
}

// M-point DFT in registers.  Composite sizes take their inner twiddles as compile-time constants, or
// from the line's table when TABLE is set (the faster choice measured for the single-precision
// forward streaming passes; the constants win everywhere else).
template <int M, int DIR, int N, bool TABLE = false, typename T>
__device__ __forceinline__ void dft(T (&v)[M], const T *__restrict__ tw) {
  using R = decltype(T::x);
  if constexpr (M == 1) {
  } else if constexpr (M == 2) {
    T a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (M == 4) {
    T t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
    T t2 = cadd(v[1], v[3]), t3 = mmi<DIR>(csub(v[1], v[3]));
    v[0] = cadd(t0, t2);
    v[2] = csub(t0, t2);
    v[1] = cadd(t1, t3);
    v[3] = csub(t1, t3);
  } else if constexpr (M == 8) {
    constexpr double h = 0.70710678118654752440084436210484903928;
    T e[4] = {v[0], v[2], v[4], v[6]};
    T o[4] = {v[1], v[3], v[5], v[7]};
    dft<4, DIR, N>(e, tw);
    dft<4, DIR, N>(o, tw);
    T w1, w3;
    if constexpr (DIR > 0) {
      w1 = kscale(mk<T>(o[1].x + o[1].y, o[1].y - o[1].x), h);
      w3 = kscale(mk<T>(o[3].y - o[3].x, -o[3].x - o[3].y), h);
    } else {
      w1 = kscale(mk<T>(o[1].x - o[1].y, o[1].y + o[1].x), h);
      w3 = kscale(mk<T>(-o[3].x - o[3].y, o[3].x - o[3].y), h);
    }
    T w2 = mmi<DIR>(o[2]);
    v[0] = cadd(e[0], o[0]);
    v[4] = csub(e[0], o[0]);
    v[1] = cadd(e[1], w1);
    v[5] = csub(e[1], w1);
    v[2] = cadd(e[2], w2);
    v[6] = csub(e[2], w2);
    v[3] = cadd(e[3], w3);
    v[7] = csub(e[3], w3);
  } else if constexpr (M == 3 || M == 5 || M == 7) {
    constexpr int H = (M - 1) / 2;
    T a[H], b[H];
#pragma unroll
    for (int m = 1; m <= H; m++) {
      a[m - 1] = cadd(v[m], v[M - m]);
      b[m - 1] = csub(v[m], v[M - m]);
    }
    const T x0 = v[0];
    T s = x0;
#pragma unroll
    for (int m = 0; m < H; m++) s = cadd(s, a[m]);
    T y[M];
    y[0] = s;
#pragma unroll
    for (int k = 1; k <= H; k++) {
      T re = x0, im = mk<T>(R(0), R(0));
#pragma unroll
      for (int m = 1; m <= H; m++) {
        const int idx = (m * k) % M;
        const double c = idx <= H ? odd_cos<M>(idx) : odd_cos<M>(M - idx);
        const double sn = idx <= H ? odd_sin<M>(idx) : -odd_sin<M>(M - idx);
        re = cadd(re, kscale(a[m - 1], c));
        im = cadd(im, kscale(b[m - 1], sn));
      }
      const T t = mmi<DIR>(im);
      y[k] = cadd(re, t);
      y[M - k] = csub(re, t);
    }
#pragma unroll
    for (int k = 0; k < M; k++) v[k] = y[k];
  } else {
    // composite: Cooley-Tukey M = A * B, twiddles W_M^t = constants or tw[t * N / M]
    constexpr int A = first_factor(M);
    constexpr int B = M / A;
    T tmp[M];
#pragma unroll
    for (int j2 = 0; j2 < B; j2++) {
      T s[A];
#pragma unroll
      for (int j1 = 0; j1 < A; j1++) s[j1] = v[j2 + B * j1];
      dft<A, DIR, N, TABLE>(s, tw);
#pragma unroll
      for (int k1 = 0; k1 < A; k1++) {
        if (j2 * k1 == 0) tmp[k1 * B + j2] = s[k1];
        else if constexpr (TABLE) tmp[k1 * B + j2] = twmul<DIR, N>(s[k1], tw, (j2 * k1) * (N / M));
        else tmp[k1 * B + j2] = tw_const_at<DIR, M>(s[k1], j2 * k1);
      }
    }
#pragma unroll
    for (int k1 = 0; k1 < A; k1++) {
      T s[B];
#pragma unroll
      for (int j2 = 0; j2 < B; j2++) s[j2] = tmp[k1 * B + j2];
      dft<B, DIR, N, TABLE>(s, tw);
#pragma unroll
      for (int k2 = 0; k2 < B; k2++) v[k1 + A * k2] = s[k2];
    }
  }
}

// Two-level in-place transform of a [N][W] tile (rows = points, natural order in and out).
template <typename TO, typename TI> __device__ __forceinline__ TO conv(TI x) { return mk<TO>(decltype(TO::x)(x.x), decltype(TO::x)(x.y)); }

// Barrier of the CTA's NT compute threads (named barrier 1).  A kernel with a producer warp runs it
// after the NT compute threads; that warp never joins, so the compute threads synchronise among
// themselves.  Without a producer warp NT is the whole CTA.
template <int NT> __device__ __forceinline__ void csync() { asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory"); }
// the same barrier, returning whether any compute thread passed a nonzero value (uniform result)
template <int NT> __device__ __forceinline__ bool csync_or(int v) {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
               : "=r"(r)
               : "r"(v), "n"(NT)
               : "memory");
  return r != 0;
}
using ptx::mbar_arrive;

// The tile transforms below end without a barrier: their last step writes only addresses the
// writing thread owns in that step, and the kernel's fence + barrier before the TMA store (or an
// explicit barrier before another sweep) orders those writes for the other threads.

// Two-level transform of one [N][W] tile.
//   step A: N1-point DFTs down the columns j2 (points j2 + N2 j1), twiddle W_N^{j2 k1};
//   step B: N2-point DFTs along the rows k1, outputs in natural order m = k1 + N1 k2.
// Step A reads `asrc` (times an optional per-point factor `pre`, applied on load) and writes
// `adst`; step B reads `adst` and hands every output value to `put(m, w, value)`.  When
// HOLD is set (step B writes into the buffer it reads), all step-B inputs are read into
// registers before a barrier and only then stored.
template <int N, int DIR, int W, int NT, bool HOLD, typename TC, typename SA, typename DA, typename Put>
__device__ __forceinline__ void tile_dft(const SA *asrc, DA *adst, const TC *__restrict__ tw,
                                         const decltype(TC::x) *pre, Put put) {
  constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2;
  for (int it = threadIdx.x; it < W * N2; it += NT) {
    const int w = it % W, j2 = it / W;
    TC s[N1];
#pragma unroll
    for (int j1 = 0; j1 < N1; j1++) {
      s[j1] = conv<TC>(asrc[(j2 + N2 * j1) * W + w]);
      if (pre) s[j1] = cscale(s[j1], pre[j2 + N2 * j1]);
    }
    dft<N1, DIR, N>(s, tw);
#pragma unroll
    for (int k1 = 1; k1 < N1; k1++) s[k1] = twmul<DIR, N>(s[k1], tw, j2 * k1);
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) adst[(j2 + N2 * k1) * W + w] = conv<DA>(s[k1]);
  }
  csync<NT>();
  if constexpr (HOLD) {
    constexpr int IB = (W * N1 + NT - 1) / NT;
    TC r[IB][N2];
#pragma unroll
    for (int b = 0; b < IB; b++) {
      const int it = threadIdx.x + b * NT;
      if (it < W * N1) {
        const int w = it % W, k1 = it / W;
#pragma unroll
        for (int j2 = 0; j2 < N2; j2++) r[b][j2] = conv<TC>(adst[(j2 + N2 * k1) * W + w]);
        dft<N2, DIR, N>(r[b], tw);
      }
    }
    csync<NT>();
#pragma unroll
    for (int b = 0; b < IB; b++) {
      const int it = threadIdx.x + b * NT;
      if (it < W * N1) {
        const int w = it % W, k1 = it / W;
#pragma unroll
        for (int k2 = 0; k2 < N2; k2++) put(k1 + N1 * k2, w, r[b][k2]);
      }
    }
  } else {
    for (int it = threadIdx.x; it < W * N1; it += NT) {
      const int w = it % W, k1 = it / W;
      TC r[N2];
#pragma unroll
      for (int j2 = 0; j2 < N2; j2++) r[j2] = conv<TC>(adst[(j2 + N2 * k1) * W + w]);
      dft<N2, DIR, N>(r, tw);
#pragma unroll
      for (int k2 = 0; k2 < N2; k2++) put(k1 + N1 * k2, w, r[k2]);
    }
  }
}

// The in-place transforms below take the tile through one restrict-qualified pointer, so the compiler
// may overlap one item's shared-memory loads with the previous item's stores, and hand every output
// value to epi(m, w, value), which returns what is stored at row m (scaling, epilogue terms, Taylor
// accumulators; the identity for a plain pass).  None ends with a barrier: the last step writes only
// rows its thread read in that step, and the kernel's fence + barrier before the TMA store orders them.

struct Identity {
  template <typename T> __device__ __forceinline__ T operator()(int, int, T v) const { return v; }
};

// Natural order in and out: step A (N1-point DFTs down the columns j2, twiddle W_N^{j2 k1}), step B
// (N2-point DFTs along the rows k1, outputs m = k1 + N1 k2).  Step B reads all its inputs before a
// barrier and stores after it (it writes other rows than it reads).  `pre`: per-point factors applied on load;
// `scale` likewise (in the first step: a second form of the last one doubles the registers of long FP64 lines).
template <int N, int DIR, int W, int NT, typename T, typename Epi>
__device__ __forceinline__ void tile_dft_inplace(T *__restrict__ buf, const T *__restrict__ tw, Epi epi,
                                                 const decltype(T::x) *pre = nullptr, bool scaled = false,
                                                 double scale = 1.0) {
  constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2;
  for (int it = threadIdx.x; it < W * N2; it += NT) {
    const int w = it % W, j2 = it / W;
    T s[N1];
#pragma unroll
    for (int j1 = 0; j1 < N1; j1++) {
      s[j1] = buf[(j2 + N2 * j1) * W + w];
      if (pre) s[j1] = cscale(s[j1], pre[j2 + N2 * j1]);
    }
    if (scaled) {
#pragma unroll
      for (int j1 = 0; j1 < N1; j1++) s[j1] = kscale(s[j1], scale);
    }
    dft<N1, DIR, N>(s, tw);
#pragma unroll
    for (int k1 = 1; k1 < N1; k1++) s[k1] = twmul<DIR, N>(s[k1], tw, j2 * k1);
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) buf[(j2 + N2 * k1) * W + w] = s[k1];
  }
  csync<NT>();
  constexpr int IB = (W * N1 + NT - 1) / NT;
  T r[IB][N2];
#pragma unroll
  for (int b = 0; b < IB; b++) {
    const int it = threadIdx.x + b * NT;
    if (it < W * N1) {
      const int w = it % W, k1 = it / W;
#pragma unroll
      for (int j2 = 0; j2 < N2; j2++) r[b][j2] = buf[(j2 + N2 * k1) * W + w];
      dft<N2, DIR, N, (sizeof(decltype(T::x)) == 4 && DIR > 0)>(r[b], tw);
    }
  }
  csync<NT>();
#pragma unroll
  for (int b = 0; b < IB; b++) {
    const int it = threadIdx.x + b * NT;
    if (it < W * N1) {
      const int w = it % W, k1 = it / W;
#pragma unroll
      for (int k2 = 0; k2 < N2; k2++) buf[(k1 + N1 * k2) * W + w] = epi(k1 + N1 * k2, w, r[b][k2]);
    }
  }
}

// forward column step in place: N1-point DFT down column j2, twiddle W_N^{j2 k1}
template <int N, int W, int NT, typename T>
__device__ __forceinline__ void col_forward_inplace(T *__restrict__ buf, const T *__restrict__ tw) {
  constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2;
  for (int it = threadIdx.x; it < W * N2; it += NT) {
    const int w = it % W, j2 = it / W;
    T s[N1];
#pragma unroll
    for (int j1 = 0; j1 < N1; j1++) s[j1] = buf[(j2 + N2 * j1) * W + w];
    dft<N1, +1, N>(s, tw);
#pragma unroll
    for (int k1 = 1; k1 < N1; k1++) s[k1] = twmul<+1, N>(s[k1], tw, j2 * k1);
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) buf[(j2 + N2 * k1) * W + w] = s[k1];
  }
}

// inverse column step in place: inverse N1-point DFT down column j2, x[j2 + N2 j1] in natural order
template <int N, int W, int NT, typename T, typename Epi>
__device__ __forceinline__ void col_inverse_inplace(T *__restrict__ buf, const T *__restrict__ tw, Epi epi) {
  constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2;
  for (int it = threadIdx.x; it < W * N2; it += NT) {
    const int w = it % W, j2 = it / W;
    T s[N1];
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) s[k1] = buf[(j2 + N2 * k1) * W + w];
    dft<N1, -1, N>(s, tw);
#pragma unroll
    for (int j1 = 0; j1 < N1; j1++) buf[(j2 + N2 * j1) * W + w] = epi(j2 + N2 * j1, w, s[j1]);
  }
}

// The x pass of the real-space operator in place: forward transform, per-frequency factor f[m],
// inverse transform.  The inverse runs the forward's two steps transposed (step B first, with
// conjugate twiddles, then step A), so it starts from the forward's k1-major output and every step
// writes the rows it read: three shared-memory sweeps and two barriers, no transposition.
//   forward A: N1-point DFTs down the columns j2, twiddle W_N^{j2 k1}
//   forward B, factor, inverse B: N2-point DFT along row k1, times f[k1 + N1 k2], inverse
//     N2-point DFT, twiddle W_N^{-j2 k1} (rows of up to 12 points batched two items at a time)
//   inverse A: inverse N1-point DFTs down the columns j2, natural order
// `f` holds the factors of the thread's column: W divides NT, so a thread keeps one column through all steps.
// Rows batched per thread in the middle step: 24 points at most (two transforms per row; more would spill).
template <int N, int W, int NT> constexpr int kin_batch() {
  static_assert(NT % W == 0, "a thread works on one column of the tile");
  constexpr int n = (W * Split<N>::N1 + NT - 1) / NT, most = 24 / Split<N>::N2;
  return n < most ? n : (most > 1 ? most : 1);
}
template <int N, int W, int NT, typename T, typename Epi>
__device__ __forceinline__ void tile_kin_inplace(T *__restrict__ buf, const T *__restrict__ tw,
                                                 const decltype(T::x) *__restrict__ f, Epi epi) {
  constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2;
  constexpr int IB = kin_batch<N, W, NT>();
  col_forward_inplace<N, W, NT, T>(buf, tw);
  csync<NT>();
  for (int it0 = threadIdx.x; it0 < W * N1; it0 += IB * NT) {
    T r[IB][N2];
#pragma unroll
    for (int b = 0; b < IB; b++) {
      const int it = it0 + b * NT;
      if (it < W * N1) {
        const int w = it % W, k1 = it / W;
#pragma unroll
        for (int j2 = 0; j2 < N2; j2++) r[b][j2] = buf[(j2 + N2 * k1) * W + w];
      }
    }
#pragma unroll
    for (int b = 0; b < IB; b++) {
      const int it = it0 + b * NT;
      if (it < W * N1) {
        const int w = it % W, k1 = it / W;
        dft<N2, +1, N>(r[b], tw);
#pragma unroll
        for (int k2 = 0; k2 < N2; k2++) r[b][k2] = cscale(r[b][k2], f[k1 + N1 * k2]);
        dft<N2, -1, N>(r[b], tw);
        if (k1 > 0) {
#pragma unroll
          for (int j2 = 1; j2 < N2; j2++) r[b][j2] = twmul<-1, N>(r[b][j2], tw, j2 * k1);
        }
#pragma unroll
        for (int j2 = 0; j2 < N2; j2++) buf[(j2 + N2 * k1) * W + w] = r[b][j2];
      }
    }
  }
  csync<NT>();
  col_inverse_inplace<N, W, NT, T>(buf, tw, epi);
}

// Forward transform in place with the output in digit-reversed order: row k2 + N2 k1 receives
// frequency k1 + N1 k2.  Step B writes the rows it read, so no second barrier is needed.
template <int N, int W, int NT, typename T, typename Epi>
__device__ __forceinline__ void tile_fwd_perm_inplace(T *__restrict__ buf, const T *__restrict__ tw, Epi epi) {
  constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2, IB = (W * N1 + NT - 1) / NT;
  col_forward_inplace<N, W, NT, T>(buf, tw);
  csync<NT>();
  T r[IB][N2];
#pragma unroll
  for (int b = 0; b < IB; b++) {
    const int it = threadIdx.x + b * NT;
    if (it < W * N1) {
      const int w = it % W, k1 = it / W;
#pragma unroll
      for (int j2 = 0; j2 < N2; j2++) r[b][j2] = buf[(j2 + N2 * k1) * W + w];
    }
  }
#pragma unroll
  for (int b = 0; b < IB; b++) {
    const int it = threadIdx.x + b * NT;
    if (it < W * N1) {
      const int w = it % W, k1 = it / W;
      dft<N2, +1, N, (sizeof(decltype(T::x)) == 4)>(r[b], tw);
#pragma unroll
      for (int k2 = 0; k2 < N2; k2++) buf[(k2 + N2 * k1) * W + w] = epi(k2 + N2 * k1, w, r[b][k2]);
    }
  }
}

// Inverse transform in place of a tile whose rows are in digit-reversed order (row k2 + N2 k1 holds
// frequency k1 + N1 k2): the forward's steps transposed, conjugate twiddles; natural order out.
template <int N, int W, int NT, typename T, typename Epi>
__device__ __forceinline__ void tile_inv_perm_inplace(T *__restrict__ buf, const T *__restrict__ tw, Epi epi) {
  constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2, IB = (W * N1 + NT - 1) / NT;
  T r[IB][N2];
#pragma unroll
  for (int b = 0; b < IB; b++) {
    const int it = threadIdx.x + b * NT;
    if (it < W * N1) {
      const int w = it % W, k1 = it / W;
#pragma unroll
      for (int k2 = 0; k2 < N2; k2++) r[b][k2] = buf[(k2 + N2 * k1) * W + w];
    }
  }
#pragma unroll
  for (int b = 0; b < IB; b++) {
    const int it = threadIdx.x + b * NT;
    if (it < W * N1) {
      const int w = it % W, k1 = it / W;
      dft<N2, -1, N>(r[b], tw);
      if (k1 > 0) {
#pragma unroll
        for (int j2 = 1; j2 < N2; j2++) r[b][j2] = twmul<-1, N>(r[b][j2], tw, j2 * k1);
      }
#pragma unroll
      for (int j2 = 0; j2 < N2; j2++) buf[(j2 + N2 * k1) * W + w] = r[b][j2];
    }
  }
  csync<NT>();
  col_inverse_inplace<N, W, NT, T>(buf, tw, epi);
}

// Column and row steps of the two-level transforms below.
//   column step: item (j2, w), N1 values at rows j2 + N2 j1; a runtime loop over the thread's items
//   row step:    item (k1, w), N2 values at rows j2 + N2 k1; the thread's IB items are batched (all
//                loads first, then the arithmetic, then the stores) so their loads are in flight
//                together and their arithmetic interleaves
// Both write only the rows they read, so no barrier separates a step's loads from its stores.

// forward column step: N1-point DFT down column j2, twiddle W_N^{j2 k1}  (asrc -> work)
template <int N, int W, int NT, typename TC, typename SA>
__device__ __forceinline__ void col_forward(const SA *asrc, TC *work, const TC *__restrict__ tw) {
  constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2;
  for (int it = threadIdx.x; it < W * N2; it += NT) {
    const int w = it % W, j2 = it / W;
    TC s[N1];
#pragma unroll
    for (int j1 = 0; j1 < N1; j1++) s[j1] = conv<TC>(asrc[(j2 + N2 * j1) * W + w]);
    dft<N1, +1, N>(s, tw);
#pragma unroll
    for (int k1 = 1; k1 < N1; k1++) s[k1] = twmul<+1, N>(s[k1], tw, j2 * k1);
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) work[(j2 + N2 * k1) * W + w] = s[k1];
  }
}

// inverse column step: inverse N1-point DFT down column j2; x[j2 + N2 j1] to put (natural order)
template <int N, int W, int NT, typename TC, typename Put>
__device__ __forceinline__ void col_inverse(const TC *work, const TC *__restrict__ tw, Put put) {
  constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2;
  for (int it = threadIdx.x; it < W * N2; it += NT) {
    const int w = it % W, j2 = it / W;
    TC s[N1];
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) s[k1] = work[(j2 + N2 * k1) * W + w];
    dft<N1, -1, N>(s, tw);
#pragma unroll
    for (int j1 = 0; j1 < N1; j1++) put(j2 + N2 * j1, w, s[j1]);
  }
}

// Forward transform, per-frequency factor f[m], inverse transform of one [N][W] tile (the x pass of
// the real-space operator), with the arithmetic in a separate buffer `work` (wider type than the
// tile); the in-place form for equal types is tile_kin_inplace.  The inverse runs the forward's two steps transposed (step B first, with
// conjugate twiddles, then step A), so it starts from the forward's k1-major output and every step
// writes the addresses it read: three shared-memory sweeps and two barriers, no transposition.
//   forward A: N1-point DFTs down the columns j2, twiddle W_N^{j2 k1}           (asrc -> work)
//   forward B, factor, inverse B: N2-point DFT along row k1, times f[k1 + N1 k2], inverse
//     N2-point DFT, twiddle W_N^{-j2 k1}                                      (work, in place)
//   inverse A: inverse N1-point DFTs down the columns j2; x[j2 + N2 j1] goes to put(m, w, value)
// `asrc` may be `work` itself.  No barrier follows the last step.
template <int N, int W, int NT, typename TC, typename SA, typename Put>
__device__ __forceinline__ void tile_dft_kin(const SA *asrc, TC *work, const TC *__restrict__ tw,
                                             const decltype(TC::x) *f, Put put) {
  constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2;
  constexpr int IB = kin_batch<N, W, NT>();
  col_forward<N, W, NT, TC>(asrc, work, tw);
  csync<NT>();
  for (int it0 = threadIdx.x; it0 < W * N1; it0 += IB * NT) {
    TC r[IB][N2];
#pragma unroll
    for (int b = 0; b < IB; b++) {
      const int it = it0 + b * NT;
      if (it < W * N1) {
        const int w = it % W, k1 = it / W;
#pragma unroll
        for (int j2 = 0; j2 < N2; j2++) r[b][j2] = work[(j2 + N2 * k1) * W + w];
      }
    }
#pragma unroll
    for (int b = 0; b < IB; b++) {
      const int it = it0 + b * NT;
      if (it < W * N1) {
        const int w = it % W, k1 = it / W;
        dft<N2, +1, N>(r[b], tw);
#pragma unroll
        for (int k2 = 0; k2 < N2; k2++) r[b][k2] = cscale(r[b][k2], f[k1 + N1 * k2]);
        dft<N2, -1, N>(r[b], tw);
        if (k1 > 0) {
#pragma unroll
          for (int j2 = 1; j2 < N2; j2++) r[b][j2] = twmul<-1, N>(r[b][j2], tw, j2 * k1);
        }
#pragma unroll
        for (int j2 = 0; j2 < N2; j2++) work[(j2 + N2 * k1) * W + w] = r[b][j2];
      }
    }
  }
  csync<NT>();
  col_inverse<N, W, NT, TC>(work, tw, put);
}

struct Geom2 {
  Geom g;           // grid and line decomposition (point strides)
  int axis;
  int nsb;          // state blocks per line
  long long ntiles;
  int stages;
  int cwords;       // 32-bit words per complex element
  int aux_single;   // second input tiles single-buffered (1) or one set per ring stage (0)
  int cpa;          // rows that are not 16-byte multiples: the compute threads move tiles with 8-byte
                    // cp.async loads and plain stores instead of TMA (two stages, second tiles per stage)
  int flat;         // y and x passes over flattened columns (below); nsb is then the column blocks per row
  long long ncols;  // flat: columns per row, nz*S (y pass) or ny*nz*S (x pass)
  int flines;       // lines whose factors a tile may need (an even number: what follows stays 8-byte aligned)
};

// Flattened columns.  A y (x) transform acts on every column of the [nx][ny][nz*S] ([nx][ny*nz*S]) view
// of the set alike, so a tile may take any W consecutive columns of that view: the (z, state) or
// (y, z, state) pairs follow one another in memory.  Rows are then W full elements for every state count
// (odd counts too, whose point rows are not 16-byte multiples, and counts that leave the last state block
// of a line part-empty), and only the last tile of each row runs past its end (TMA fills the loads with
// zeros and clips the stores).  With S a multiple of W the tiles, and their order, are those of the
// (line, state block) decomposition.  The kinetic factor of a column depends on its (y, z) line; a tile's
// columns lie on at most (W - 1) / S + 2 lines, two when S >= W.

template <int VAR> constexpr int dir_first() { return (base_var(VAR) == INV_STORE || base_var(VAR) == INV_FINAL) ? -1 : +1; }

// Tiles of 256-byte rows, or 128-byte rows when the butterflies run in a wider type than the storage
// (the tile then also needs an exchange buffer of that type, and smaller tiles let several CTAs share
// an SM to cover the double-precision latency).
template <typename R, typename CR, int WIDE = 0> constexpr int tile_w() {
  return WIDE ? 512 / int(2 * sizeof(R)) : (sizeof(CR) > sizeof(R) ? 128 : 256) / int(2 * sizeof(R));
}
// Threads per CTA.  The two steps of a tile transform have W*N2 and W*N1 independent line pieces; with
// 128 threads and 16-state tiles (N1 = 8) the first step of N = 72, 96, 120, 128 takes two rounds in
// which part of the CTA idles at the next barrier, so those tiles get one thread per first-step piece.
// The kinetic pass (two transforms, the second with two idle thirds in its second step either way)
// keeps 128 threads and more CTAs per SM.  The single-precision final passes of 96- to 128-point
// lines (two tiles per stage: two stages, and 8 warps per SM at 128 threads for 96 points, 4 for
// 120) run one thread per column item: 384 threads for 96 points (measured: 1.06 ms against 1.15 ms
// at 96^3 x 256), 480 for 120.
template <typename R, typename CR, int N, int VAR, int WIDE = 0> constexpr int threads_of() {
  constexpr int W = tile_w<R, CR, WIDE>();
  constexpr int A = W * Split<N>::N2, B = W * Split<N>::N1;
  constexpr int M = A > B ? A : B;
  if constexpr (WIDE) return 256;
  if constexpr (base_var(VAR) == INV_FINAL && W == 32 && N >= 96 && sizeof(CR) == 4) return (A + 31) / 32 * 32;
  return (VAR != MID_KIN && W == 16 && M > 128 && M <= 256) ? (M + 31) / 32 * 32 : 128;
}

// Whether the kernel runs a producer warp: one extra warp whose lane 0 issues every TMA load and
// store and waits for the stores to drain, so no compute thread stalls on the copies.  Measured at
// 96^3 x 256: the single-precision passes gain 8-15 % (final pass 0.80 ms against 0.93, kinetic pass
// 0.68 against 0.73); the FP64 passes, already at the HBM limit, lose (forward 1.29 against 1.11).
template <typename R, typename CR, int N, int VAR> constexpr bool ws_of() {
  return sizeof(R) == 4 && sizeof(CR) == 4;
}
template <typename R, typename CR, int N, int VAR, int WIDE = 0> constexpr int block_threads_of() {
  return threads_of<R, CR, N, VAR, WIDE>() + (ws_of<R, CR, N, VAR>() ? 32 : 0);
}

// CTAs per SM the register allocation must allow: four for the single-precision kinetic pass of lines
// up to 96 points (two transforms per tile, latency-bound with fewer warps; longer lines would spill);
// 0 (no constraint: the compiler's own register choice) otherwise.
template <typename R, typename CR, int N, int VAR, int WIDE = 0> constexpr int min_ctas_of() {
  if constexpr (WIDE) return 0;
  return (VAR == MID_KIN && sizeof(R) == 4 && sizeof(CR) == 4 && N <= 96) ? 4 : 0;
}

template <typename R, typename CR, int N, int VAR, int WIDE>
__global__ void __launch_bounds__(block_threads_of<R, CR, N, VAR, WIDE>(), min_ctas_of<R, CR, N, VAR, WIDE>()) fft2_kernel(const __grid_constant__ CUtensorMap map_in,
                                                   const __grid_constant__ CUtensorMap map_out,
                                                   const __grid_constant__ CUtensorMap map_aux,
                                                   const __grid_constant__ CUtensorMap map_base, PassArgs<R> a, Geom2 gg,
                                                   const C2<CR> *__restrict__ twg, int *err) {
  using T = C2<R>;
  using TC = C2<CR>;
  constexpr int NT = threads_of<R, CR, N, VAR, WIDE>();   // compute threads
  constexpr bool WS = ws_of<R, CR, N, VAR>();             // plus a producer warp
  constexpr int NTT = block_threads_of<R, CR, N, VAR, WIDE>();
  constexpr bool SPLIT = sizeof(CR) > sizeof(R);          // exchange buffer in the arithmetic type
  constexpr int W = tile_w<R, CR, WIDE>();
  constexpr int TILE = N * W;                       // complex elements per tile
  constexpr uint32_t TILE_BYTES = TILE * sizeof(T);
  constexpr bool AUX = has_aux(VAR);
  const int NS = gg.stages;
  // a Horner step (final pass of the real-space operator): a third tile per stage holds the base
  const bool horner = AUX && a.hbase != nullptr;

  // The second input tile (psi of V psi or of the Laplacian term) and the Horner base are needed only in
  // the last step of a tile's transform.  Either every ring stage holds them beside its tile (loaded with
  // it), or, when that would leave one CTA per SM (gg.aux_single), they are single-buffered: loaded for
  // the CTA's next tile as soon as its current one is computed, so that they land during the next tile's
  // first steps, while the ring stages hold one tile each.
  const int naux = AUX ? (horner ? 2 : 1) : 0;
  const bool aux1 = AUX && gg.aux_single;

  extern __shared__ __align__(1024) unsigned char smem[];
  T *stage_in = reinterpret_cast<T *>(smem);                         // NS tiles
  T *aux_ring = stage_in + size_t(NS) * TILE;                        // naux tiles, or NS x naux
  TC *exch = reinterpret_cast<TC *>(aux_ring + size_t(aux1 ? 1 : NS) * naux * TILE);  // one tile when SPLIT
  constexpr int TWN = tw_entries<CR>(N);
  TC *tw = exch + (SPLIT ? TILE : 0);                                // twiddles (high, then low parts)
  CR *linev = reinterpret_cast<CR *>(tw + TWN);                      // N per-point factors per line of the tile
  uint64_t *bar = reinterpret_cast<uint64_t *>(linev + gg.flines * N);  // NS "tile loaded" barriers (8-byte aligned)
  uint64_t *done = bar + NS;                                         // NS "tile computed" barriers (producer warp)
  uint64_t *abar = done + NS;                                        // "second input tiles loaded"
  volatile int *abort_flag = reinterpret_cast<volatile int *>(abar + 1);

  const Geom &g = gg.g;
  for (int i = threadIdx.x; i < TWN; i += NTT) tw[i] = twg[i];
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < NS; s++) {
      mbar_init(&bar[s], 1);
      if constexpr (WS) mbar_init(&done[s], NT);
    }
    mbar_init(abar, 1);
    mbar_init_fence();
  }
  __syncthreads();
  ptx::grid_wait();
  ptx::grid_release();

  auto coords = [&](long long t, int &c0, int &c1, int &c2, int &c3) {
    if (gg.flat) {
      c0 = int((t % gg.nsb) * W) * gg.cwords;
      c1 = 0;
      c2 = gg.axis == 1 ? int(t / gg.nsb) : 0;
      c3 = 0;
      return;
    }
    const long long L = t / gg.nsb;
    const int s0 = int(t % gg.nsb) * W;
    const int la = int(L / g.nb), lb = int(L % g.nb);
    c0 = s0 * gg.cwords;
    if (gg.axis == 2) { c1 = 0; c2 = lb; c3 = la; }        // z-lines: (x, y) fixed
    else if (gg.axis == 1) { c1 = lb; c2 = 0; c3 = la; }   // y-lines: (x, z) fixed
    else { c1 = lb; c2 = la; c3 = 0; }                     // x-lines: (y, z) fixed
  };
  auto issue = [&](int st, long long t) {
    int c0, c1, c2, c3;
    coords(t, c0, c1, c2, c3);
    mbar_expect_tx(&bar[st], uint32_t(aux1 ? 1 : 1 + naux) * TILE_BYTES);
    tma_load_4d(stage_in + size_t(st) * TILE, &map_in, &bar[st], c0, c1, c2, c3);
    if (AUX && !aux1) {
      T *ax = aux_ring + size_t(st) * naux * TILE;
      tma_load_4d(ax, &map_aux, &bar[st], c0, c1, c2, c3);
      if (horner) tma_load_4d(ax + TILE, &map_base, &bar[st], c0, c1, c2, c3);
    }
  };
  // single-buffered: the second input tile (and the Horner base) of tile t; the k-th such load completes
  // phase k of abar
  auto issue_aux = [&](long long t) {
    int c0, c1, c2, c3;
    coords(t, c0, c1, c2, c3);
    mbar_expect_tx(abar, uint32_t(naux) * TILE_BYTES);
    tma_load_4d(aux_ring, &map_aux, abar, c0, c1, c2, c3);
    if (horner) tma_load_4d(aux_ring + TILE, &map_base, abar, c0, c1, c2, c3);
  };

  // bounded wait on an mbarrier phase; false (and the error flag raised) on expiry or abort
  auto wait_bar = [&](uint64_t *b, uint32_t parity) -> bool {
    const uint64_t t0 = global_ns();
    while (!mbar_try_wait(b, parity)) {
      if (*abort_flag) return false;
      if (global_ns() - t0 > 2000000000ull) {
        *abort_flag = 1;
        atomicExch(err, 1);
        return false;
      }
    }
    return true;
  };

  // tiles whose loads the issuing thread has started (the i-th goes to stage i % NS, phase i / NS);
  // before the CTA ends, that thread waits (bounded) for the last NS of them, so that after an aborted
  // wait no load still lands in shared memory (on the normal path those phases are complete already)
  int nissued = 0, naux_issued = 0;
  auto drain = [&]() {
    for (int i = nissued - NS < 0 ? 0 : nissued - NS; i < nissued; i++)
      ptx::mbar_wait_bounded(&bar[i % NS], uint32_t(i / NS) & 1u, 2000000000ull);
    if (naux_issued > 0) ptx::mbar_wait_bounded(abar, uint32_t(naux_issued - 1) & 1u, 2000000000ull);
  };
  if (threadIdx.x == (WS ? NT : 0) && !gg.cpa) {
    for (int s = 0; s < NS; s++) {
      const long long t = blockIdx.x + (long long)s * gridDim.x;
      if (t < gg.ntiles) issue(s, t), nissued++;
    }
    if (aux1 && blockIdx.x < gg.ntiles) issue_aux(blockIdx.x), naux_issued++;
  }
  if constexpr (WS) {
    // rows that TMA cannot move: the compute threads copy them (below); the producer warp has no work
    if (threadIdx.x >= NT && gg.cpa) return;
    if (threadIdx.x >= NT) {
      // producer warp: lane 0 stores every computed tile, waits for the store to read the stage and
      // refills it with the tile NS steps ahead
      if (threadIdx.x == NT) {
        int k = 0;
        for (long long t = blockIdx.x; t < gg.ntiles; t += gridDim.x, k++) {
          const int st = k % NS;
          if (!wait_bar(&done[st], uint32_t(k / NS) & 1u)) break;
          int c0, c1, c2, c3;
          coords(t, c0, c1, c2, c3);
          tma_store_4d(&map_out, stage_in + size_t(st) * TILE, c0, c1, c2, c3);
          bulk_commit();
          // the second input tiles were read by the finished tile's epilogue: load the next tile's
          if (aux1 && t + gridDim.x < gg.ntiles) issue_aux(t + gridDim.x), naux_issued++;
          bulk_wait_read0();
          const long long tn = t + (long long)NS * gridDim.x;
          if (tn < gg.ntiles) issue(st, tn), nissued++;
        }
        drain();
        bulk_wait0();
      }
      return;
    }
  }

  const bool scaled = a.scale != 1.0;
  // 8-byte copies by the compute threads (rows that are not 16-byte multiples, gg.cpa): tile t's rows of
  // `src` into dst, consecutive threads on consecutive states; with the second input tiles of the stage
  auto cpa_rows = [&](long long t, long long &pbase, int &s0, int &ws) {
    const long long L = t / gg.nsb;
    s0 = int(t % gg.nsb) * W;
    ws = a.S - s0 < W ? a.S - s0 : W;
    pbase = (L / g.nb) * g.sa + (L % g.nb) * g.sb;
  };
  auto cpa_load = [&](T *dst, const T *src, long long t) {
    long long pbase;
    int s0, ws;
    cpa_rows(t, pbase, s0, ws);
    for (int e = threadIdx.x; e < TILE; e += NT) {
      const int r = e / W, c = e % W;
      if (c < ws) ptx::cp_async8(dst + e, src + (pbase + r * g.sp) * a.S + s0 + c);
    }
  };
  auto cpa_load_stage = [&](int st, long long t) {
    cpa_load(stage_in + size_t(st) * TILE, a.in, t);
    if constexpr (AUX) {
      cpa_load(aux_ring + size_t(st) * naux * TILE, a.psi, t);
      if (horner) cpa_load(aux_ring + size_t(st) * naux * TILE + TILE, a.hbase, t);
    }
  };
  if (gg.cpa) {
    if (blockIdx.x < gg.ntiles) cpa_load_stage(0, blockIdx.x);
    ptx::cp_async_commit();
  }
  // V of a tile's line: in double requested one tile ahead (raw, so that nothing waits for it before the next
  // tile; 120^3 x 64 final pass 872 -> 826 us); single-precision passes lose by it (96^3 x 256 816 -> 877)
  constexpr bool LINEV = base_var(VAR) == INV_FINAL || VAR == FWD_VPSI;
  constexpr bool AHEAD = LINEV && sizeof(R) == 8;
  constexpr int VB = LINEV ? (N + NT - 1) / NT : 1;
  R nextv[VB];
  int nexth[VAR == FWD_VPSI ? VB : 1];  // sphere hits of the point
  auto request_v = [&](long long t) {
    if constexpr (LINEV) {
      const long long L = t / gg.nsb, pb = (L / g.nb) * g.sa + (L % g.nb) * g.sb;
#pragma unroll
      for (int k = 0; k < VB; k++) {
        const int m = threadIdx.x + k * NT;
        const long long pt = pb + (m < N ? m : 0) * g.sp;
        nextv[k] = a.V[pt * a.nspin + a.spin];
        if constexpr (VAR == FWD_VPSI) nexth[k] = a.nl_offs ? a.nl_offs[pt + 1] - a.nl_offs[pt] : 0;
      }
    }
  };
  if (AHEAD && blockIdx.x < gg.ntiles) request_v(blockIdx.x);
  int i = 0;
  for (long long t = blockIdx.x; t < gg.ntiles; t += gridDim.x, i++) {
    const int st = i % NS;
    const uint32_t par = uint32_t(i / NS) & 1u;
    if (gg.cpa) {
      // two stages: the next tile's copies are issued before this tile's are awaited
      if (t + gridDim.x < gg.ntiles) cpa_load_stage((i + 1) % NS, t + gridDim.x);
      ptx::cp_async_commit();
      ptx::cp_async_wait<1>();
      csync<NT>();
    } else {
      // bounded wait for this stage's TMA load; every compute thread takes the same decision
      const bool ok = wait_bar(&bar[st], par);
      if (csync_or<NT>(!ok || *abort_flag)) break;
    }

    T *buf = stage_in + size_t(st) * TILE;
    const T *aux = aux_ring + (aux1 ? 0 : size_t(st) * naux * TILE);
    const T *base = aux + TILE;
    bool aux_ready = !aux1;  // this thread has waited for the tile's second input (phase i of abar)
    long long L;
    int s0, la, lb;
    if constexpr (VAR == MID_KIN) {
      // the issue-bound kinetic pass: 32-bit divisions (the host keeps the tile count below 2^31)
      const int ti = int(t), Li = ti / gg.nsb;
      L = Li;
      s0 = (ti - Li * gg.nsb) * W;
      la = Li / g.nb;
      lb = Li - la * g.nb;
    } else {
      L = t / gg.nsb;
      s0 = int(t % gg.nsb) * W;
      la = int(L / g.nb);
      lb = int(L % g.nb);
    }
    const long long pbase = la * g.sa + lb * g.sb;

    // per-point factors of this line (consumed after the first barrier of the transform); flattened
    // columns: of every line the tile's columns lie on, one after the other; lv: those of the thread's column
    const CR *lv = linev;
    if constexpr (VAR == MID_KIN || VAR == FWD_LAPLADD) {
      if (gg.flat) {
        // 32-bit divisions: a view row has fewer than 2^31 words (the host checks it).  With S >= W a tile's columns
        // lie on at most two lines, and comparisons do for the two divisions per column (issue-bound: 72^3 x 99 single
        // 137 -> 135.5 us, 96^3 x 110 305 -> 302).  o0: columns of line l0 before the tile's
        const int col0 = int(t % gg.nsb) * W, l0 = col0 / a.S, o0 = col0 - l0 * a.S;
        const int left = int(gg.ncols) - 1 - col0, last = left < W - 1 ? left : W - 1;  // last column of the tile
        const int w = int(threadIdx.x % W), mine = w < last ? w : last;
        const bool few = a.S < W;
        const int nl = few ? (o0 + last) / a.S + 1 : (o0 + last >= a.S ? 2 : 1);
        lv = linev + N * (few ? (o0 + mine) / a.S : (o0 + mine >= a.S ? 1 : 0));
        for (int e = threadIdx.x; e < nl * N; e += NT) {
          const int l = l0 + e / N;  // x-line (y, z) = (l / nz, l % nz)
          const int ly = l / g.n[2];
          int ix, iy, iz;
          line_coords(gg.axis, ly, l - ly * g.n[2], e % N, ix, iy, iz);
          if (a.perm_n2[1]) iy = iy / a.perm_n2[1] + (g.n[1] / a.perm_n2[1]) * (iy % a.perm_n2[1]);
          if (a.perm_n2[2]) iz = iz / a.perm_n2[2] + (g.n[2] / a.perm_n2[2]) * (iz % a.perm_n2[2]);
          linev[e] = CR(lapl_value(g, ix, iy, iz, a.lap_factor, a.gc));
        }
      } else
      for (int m = threadIdx.x; m < N; m += NT) {
        int ix, iy, iz;
        line_coords(gg.axis, la, lb, m, ix, iy, iz);
        // axes held in digit-reversed frequency order: position k2 + N2 k1 is frequency k1 + N1 k2
        if (a.perm_n2[1]) iy = iy / a.perm_n2[1] + (g.n[1] / a.perm_n2[1]) * (iy % a.perm_n2[1]);
        if (a.perm_n2[2]) iz = iz / a.perm_n2[2] + (g.n[2] / a.perm_n2[2]) * (iz % a.perm_n2[2]);
        linev[m] = CR(lapl_value(g, ix, iy, iz, a.lap_factor, a.gc));
      }
    } else if constexpr (AHEAD) {
#pragma unroll
      for (int k = 0; k < VB; k++) {
        const int m = threadIdx.x + k * NT;
        // Fourier form: points with sphere hits already hold (V + shift) psi + nonlocal
        bool masked = false;
        if constexpr (VAR == FWD_VPSI) masked = nexth[k] > 0;
        if (m < N) linev[m] = masked ? CR(1) : CR(nextv[k]) + CR(a.vshift);
      }
      if (t + gridDim.x < gg.ntiles) request_v(t + gridDim.x);
    } else if constexpr (LINEV) {
      for (int m = threadIdx.x; m < N; m += NT) {
        const long long pt = pbase + m * g.sp;
        const bool masked = VAR == FWD_VPSI && a.nl_offs && a.nl_offs[pt + 1] > a.nl_offs[pt];
        linev[m] = masked ? CR(1) : CR(a.V[pt * a.nspin + a.spin]) + CR(a.vshift);
      }
    }
    if constexpr (VAR == FWD_VPSI) csync<NT>();  // the transform's first step reads the factors

    // final value of one output element: scaling, epilogue term, Horner step (base + c * value, the
    // value rounded to the storage type first, as the operator's output would be)
    auto epi_out = [&](int m, int w, TC v) -> T {
      if constexpr (AUX) {
        if (!aux_ready) {
          wait_bar(abar, uint32_t(i) & 1u);  // on expiry the error flag is raised and the tile loop ends
          aux_ready = true;
        }
      }
      if (scaled) v = kscale(v, a.scale);
      if constexpr (base_var(VAR) == INV_FINAL || VAR == FWD_LAPLADD) v = cadd(v, cscale(conv<TC>(aux[m * W + w]), lv[m]));
      if constexpr (AUX) {
        if (horner) return cadd(base[m * W + w], cmul(a.hc, conv<T>(v)));
      }
      return conv<T>(v);
    };
    auto put_out = [&](int m, int w, TC v) { buf[m * W + w] = epi_out(m, w, v); };
    const CR *pre = VAR == FWD_VPSI ? linev : nullptr;  // per-point factors of the input
    constexpr int D = dir_first<VAR>();
    const T *twt = reinterpret_cast<const T *>(tw);

    if constexpr (SPLIT) {
      static_assert(!is_perm(VAR), "digit-reversed passes run with equal storage and arithmetic types");
      if constexpr (VAR == MID_KIN) {
        // forward, multiply by the kinetic factor, backward
        tile_dft_kin<N, W, NT, TC>(buf, exch, tw, lv, put_out);
      } else {
        tile_dft<N, D, W, NT, false, TC>(buf, exch, tw, pre, put_out);
      }
    } else {
      // plain passes (no scaling, no accumulators) store the transform's values as they are
      const bool plain = !AUX && !scaled;
      if constexpr (VAR == MID_KIN) {
        if (plain) tile_kin_inplace<N, W, NT, T>(buf, twt, lv, Identity());
        else tile_kin_inplace<N, W, NT, T>(buf, twt, lv, epi_out);
      } else if constexpr (VAR == INV_FINAL_PERM) {
        tile_inv_perm_inplace<N, W, NT, T>(buf, twt, epi_out);
      } else if constexpr (VAR == FWD_PERM || VAR == INV_PERM) {
        if constexpr (VAR == FWD_PERM) tile_fwd_perm_inplace<N, W, NT, T>(buf, twt, Identity());
        else tile_inv_perm_inplace<N, W, NT, T>(buf, twt, Identity());
        if (!plain) {
          csync<NT>();
          for (int e = threadIdx.x; e < TILE; e += NT) put_out(e / W, e % W, buf[e]);
        }
      } else if constexpr (AUX) {
        // the epilogue (V psi or the Laplacian term, Taylor accumulators) in the transform's last step
        tile_dft_inplace<N, D, W, NT, T>(buf, twt, epi_out);
      } else if constexpr (VAR == INV_STORE) {
        tile_dft_inplace<N, D, W, NT, T>(buf, twt, Identity(), nullptr, scaled, a.scale);
      } else {
        tile_dft_inplace<N, D, W, NT, T>(buf, twt, Identity(), pre);
        if (!plain) {
          csync<NT>();
          for (int e = threadIdx.x; e < TILE; e += NT) put_out(e / W, e % W, buf[e]);
        }
      }
    }

    if (gg.cpa) {
      // plain stores of the computed tile; the barrier after them frees the stage for the copies of the
      // tile two steps ahead
      csync<NT>();
      long long pbase;
      int s0, ws;
      cpa_rows(t, pbase, s0, ws);
      for (int e = threadIdx.x; e < TILE; e += NT) {
        const int r = e / W, c = e % W;
        if (c < ws) a.out[(pbase + r * g.sp) * a.S + s0 + c] = buf[e];
      }
      csync<NT>();
      continue;
    }
    fence_proxy_async();
    if constexpr (WS) {
      mbar_arrive(&done[st]);  // the producer warp stores the tile and refills the stage
    } else {
      csync<NT>();
      if (threadIdx.x == 0) {
        int c0, c1, c2, c3;
        coords(t, c0, c1, c2, c3);
        tma_store_4d(&map_out, buf, c0, c1, c2, c3);
        bulk_commit();
        if (aux1 && t + gridDim.x < gg.ntiles) issue_aux(t + gridDim.x), naux_issued++;
        bulk_wait_read0();  // the stage may be refilled once the store has read it
        const long long tn = t + (long long)NS * gridDim.x;
        if (tn < gg.ntiles) issue(st, tn), nissued++;
      }
    }
  }
  if (gg.cpa) ptx::cp_async_wait_all();
  if (!WS && threadIdx.x == 0) {
    drain();
    bulk_wait0();
  }
}


// ------------------------------------------------------------------ z passes over whole lines

// A z-line's points follow one another in memory, so `lpt` whole lines with all their states are one
// contiguous chunk, whatever the state count: one bulk copy loads it, odd counts (whose point rows no
// tensor map describes) and few states included, and no tile slot is empty.  The tiles of fft2_kernel
// leave up to a whole state block of each line empty, and move odd single-precision counts with 8-byte
// copies of the compute threads.
//
// In the chunk [line][point][state] the first step's items (j2, s) and the second step's (k1, s) of a line
// are consecutive too: item i of a column step touches i + j1 N2 S, so consecutive threads read consecutive
// elements and only the twiddles need the item's (j2, s), one multiplication by a reciprocal.  The first
// step works in shared memory in place, the second goes straight to global memory with its epilogue (a
// warp stores consecutive elements); the second inputs of an epilogue are read there the same way, before
// the step's shared-memory loads, so they need no tile of their own.
//
// Bound by HBM: one transit in and one out (and the second inputs).  Measured: 72^3 x 99 single, forward 206 -> 95 us
// (6.2 TB/s) and final 354 -> 183 us against the 8-byte copies; 40^3 x 33 double, forward 22.8 -> 12.4 and final
// Horner pass 46.7 -> 31.0 us against 16-state tiles (48 slots for 33 states).  zlines_of has the chunk and thread
// counts, which follow shared memory alone.  The forward and plain inverse kernels (48 to 108 registers a thread)
// come close to its 10 to 18 warps per SM; the final ones do not: in double they take 99 to 168 registers, so 40^3 x 33
// (224 threads) runs one CTA per SM where its shared memory would hold three, 54 x 60 x 45 x 50 (288) one of two, and the
// CTAs beyond those resident follow when they end; natural-order final passes in double spill besides (300 bytes at 75,
// 105 and 120 points, 104 to 324 at 84, 96, 98, 108, 112, 126 and 128).  Rows that are whole 256-byte tiles keep the
// TMA tiles of fft2_kernel, which leave nothing empty either, and so do the final passes of final_tiles.
struct GeomZ {
  long long lines;           // nx * ny
  int lpt, stages;
  int ntiles;
  uint32_t mag_s, mag_a, mag_b;  // reciprocals of S, N2 S (items per line of a column step), N1 S
};
// floor(i / d) for i d < 2^32 with m = ceil(2^32 / d); m = 0 stands for d = 1
__device__ __forceinline__ int div_by(int i, uint32_t m) { return m ? int(__umulhi(uint32_t(i), m)) : i; }

template <typename R> constexpr int zl_max_threads() { return (sizeof(R) == 8 ? 320 : 480) + 32; }

template <typename R, int N, int VAR>
__global__ void __launch_bounds__(zl_max_threads<R>()) fftz_kernel(PassArgs<R> a, GeomZ gz,
                                                                  const C2<R> *__restrict__ twg, int *err) {
  using T = C2<R>;
  constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2;
  constexpr int TWN = tw_entries<R>(N);
  constexpr int D = dir_first<VAR>();
  constexpr bool FINAL = base_var(VAR) == INV_FINAL;
  constexpr bool LINEV = FINAL || VAR == FWD_VPSI;
  const int NT = int(blockDim.x) - 32;  // compute threads; the last warp's lane 0 issues the loads
  const int S = a.S, NS = gz.stages;
  const int line = N * S;               // elements per line
  const int chunk = gz.lpt * line;

  extern __shared__ __align__(1024) unsigned char smem[];
  T *ring = reinterpret_cast<T *>(smem);
  T *tw = ring + size_t(NS) * chunk;
  R *linev = reinterpret_cast<R *>(tw + TWN);  // V + shift of the chunk's points
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + ((size_t(NS) * chunk * sizeof(T) + TWN * sizeof(T) +
                                                         size_t(gz.lpt) * N * sizeof(R) + 15) & ~size_t(15)));
  uint64_t *done = full + NS;
  volatile int *abort_flag = reinterpret_cast<volatile int *>(done + NS);

  for (int i = threadIdx.x; i < TWN; i += blockDim.x) tw[i] = twg[i];
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < NS; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&done[s], NT);
    }
    mbar_init_fence();
  }
  __syncthreads();
  ptx::grid_wait();
  ptx::grid_release();

  auto wait_bar = [&](uint64_t *b, uint32_t parity) -> bool {
    const uint64_t t0 = global_ns();
    while (!mbar_try_wait(b, parity)) {
      if (*abort_flag) return false;
      if (global_ns() - t0 > 2000000000ull) {
        *abort_flag = 1;
        atomicExch(err, 1);
        return false;
      }
    }
    return true;
  };
  auto lines_of = [&](int t) {
    const long long left = gz.lines - (long long)t * gz.lpt;
    return left < gz.lpt ? int(left) : gz.lpt;
  };

  if (int(threadIdx.x) >= NT) {
    if (int(threadIdx.x) == NT) {
      int k = 0;
      for (int t = blockIdx.x; t < gz.ntiles; t += gridDim.x, k++) {
        const int st = k % NS;
        if (k >= NS && !wait_bar(&done[st], uint32_t(k / NS - 1) & 1u)) break;
        const uint32_t bytes = uint32_t(lines_of(t)) * uint32_t(line) * uint32_t(sizeof(T));
        mbar_expect_tx(&full[st], bytes);
        ptx::bulk_load(ring + size_t(st) * chunk, a.in + (long long)t * chunk, bytes, &full[st]);
      }
      // after an aborted wait the compute threads may leave early: no load may still land in the CTA's
      // shared memory then (on the normal path these phases are complete)
      for (int i = k - NS < 0 ? 0 : k - NS; i < k; i++)
        ptx::mbar_wait_bounded(&full[i % NS], uint32_t(i / NS) & 1u, 2000000000ull);
    }
    return;
  }

  auto sync = [&]() { asm volatile("bar.sync 1, %0;" ::"r"(NT) : "memory"); };
  auto sync_or = [&](int v) -> bool {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(r)
                 : "r"(v), "r"(NT)
                 : "memory");
    return r != 0;
  };
  const bool horner = FINAL && a.hbase != nullptr;
  const bool scaled = a.scale != 1.0;
  const int tid = threadIdx.x, colS = N2 * S, rowS = N1 * S;
  // V of the chunk's point tid: in double requested one chunk ahead
  constexpr bool AHEAD = LINEV && sizeof(R) == 8;
  // psi of an item of the last step one item ahead: in double (54 x 60 x 45 x 50 87 -> 76 us) while the registers
  // last (80^3 x 40: H 717 -> 765 us with spills); single precision loses by it (72^3 x 99 181 -> 199 us)
  constexpr bool PSI_AHEAD = FINAL && sizeof(R) == 8 && N1 + N2 <= 16;
  R nextv = R(0);
  int nexth = 0;
  auto request_v = [&](int t) {
    if constexpr (LINEV) {
      const long long pt = (long long)t * gz.lpt * N + tid;
      if (tid < lines_of(t) * N) {
        nextv = a.V[pt * a.nspin + a.spin];
        if (VAR == FWD_VPSI && a.nl_offs) nexth = a.nl_offs[pt + 1] - a.nl_offs[pt];
      }
    }
  };
  if (AHEAD && int(blockIdx.x) < gz.ntiles) request_v(blockIdx.x);
  int i = 0;
  for (int t = blockIdx.x; t < gz.ntiles; t += gridDim.x, i++) {
    const int st = i % NS;
    const bool ok = wait_bar(&full[st], uint32_t(i / NS) & 1u);
    if (sync_or(!ok || *abort_flag)) break;
    T *__restrict__ buf = ring + size_t(st) * chunk;
    const int nl = lines_of(t);
    const long long g0 = (long long)t * chunk;  // the chunk's first element
    T *__restrict__ out = a.out + g0;
    if constexpr (LINEV) {
      const long long p0 = (long long)t * gz.lpt * N;
      const bool hits = VAR == FWD_VPSI && a.nl_offs != nullptr;
      // points with sphere hits already hold (V + shift) psi + nonlocal
      if (AHEAD && tid < nl * N) linev[tid] = hits && nexth > 0 ? R(1) : nextv + a.vshift;
      for (int m = AHEAD ? tid + NT : tid; m < nl * N; m += NT) {
        const long long pt = p0 + m;
        linev[m] = hits && a.nl_offs[pt + 1] > a.nl_offs[pt] ? R(1) : a.V[pt * a.nspin + a.spin] + a.vshift;
      }
      if (AHEAD && t + int(gridDim.x) < gz.ntiles) request_v(t + gridDim.x);
      if constexpr (VAR == FWD_VPSI) sync();
    }

    if constexpr (VAR == INV_PERM || VAR == INV_FINAL_PERM) {
      // rows first (digit-reversed input), then columns in natural order; the first column item's psi is
      // requested before the rows, each further one an item ahead
      T xn[PSI_AHEAD ? N1 : 1];
      auto request_psi = [&](int it) {
        if constexpr (PSI_AHEAD) {
          if (it < nl * colS) {
            const int l = nl > 1 ? div_by(it, gz.mag_a) : 0;
            const T *src = a.psi + g0 + it + (long long)l * (line - colS);
#pragma unroll
            for (int j1 = 0; j1 < N1; j1++) xn[j1] = src[j1 * colS];
          }
        }
      };
      request_psi(tid);
      for (int it = tid; it < nl * rowS; it += NT) {
        const int l = nl > 1 ? div_by(it, gz.mag_b) : 0, r = it - l * rowS;
        const int k1 = div_by(r, gz.mag_s);
        T *p = buf + l * line + k1 * colS + (r - k1 * S);
        T v[N2];
#pragma unroll
        for (int k2 = 0; k2 < N2; k2++) v[k2] = p[k2 * S];
        dft<N2, -1, N>(v, tw);
        if (k1 > 0) {
#pragma unroll
          for (int j2 = 1; j2 < N2; j2++) v[j2] = twmul<-1, N>(v[j2], tw, j2 * k1);
        }
#pragma unroll
        for (int j2 = 0; j2 < N2; j2++) p[j2 * S] = v[j2];
      }
      sync();
      for (int it = tid; it < nl * colS; it += NT) {
        const int l = nl > 1 ? div_by(it, gz.mag_a) : 0, r = it - l * colS;
        const int e0 = l * line + r;
        T x[FINAL ? N1 : 1], h[FINAL ? N1 : 1];
        if constexpr (FINAL) {
#pragma unroll
          for (int j1 = 0; j1 < N1; j1++) x[j1] = PSI_AHEAD ? xn[PSI_AHEAD ? j1 : 0] : a.psi[g0 + e0 + j1 * colS];
          request_psi(it + NT);  // the next item's, while this one is transformed
          if (horner) {
#pragma unroll
            for (int j1 = 0; j1 < N1; j1++) h[j1] = a.hbase[g0 + e0 + j1 * colS];
          }
        }
        T v[N1];
#pragma unroll
        for (int k1 = 0; k1 < N1; k1++) v[k1] = buf[e0 + k1 * colS];
        dft<N1, -1, N>(v, tw);
        if constexpr (FINAL) {
          const R *lv = linev + l * N + div_by(r, gz.mag_s);
#pragma unroll
          for (int j1 = 0; j1 < N1; j1++) {
            T o = scaled ? kscale(v[j1], a.scale) : v[j1];
            o = cadd(o, cscale(x[j1], lv[j1 * N2]));
            if (horner) o = cadd(h[j1], cmul(a.hc, o));
            out[e0 + j1 * colS] = o;
          }
        } else {
#pragma unroll
          for (int j1 = 0; j1 < N1; j1++) out[e0 + j1 * colS] = scaled ? kscale(v[j1], a.scale) : v[j1];
        }
      }
    } else {
      // columns first, then rows: natural order, or rows of digit-reversed frequencies
      for (int it = tid; it < nl * colS; it += NT) {
        const int l = nl > 1 ? div_by(it, gz.mag_a) : 0, r = it - l * colS;
        const int j2 = div_by(r, gz.mag_s);
        T *p = buf + l * line + r;
        T v[N1];
#pragma unroll
        for (int j1 = 0; j1 < N1; j1++) v[j1] = p[j1 * colS];
        if constexpr (VAR == FWD_VPSI) {
          const R *lv = linev + l * N + j2;
#pragma unroll
          for (int j1 = 0; j1 < N1; j1++) v[j1] = cscale(v[j1], lv[j1 * N2]);
        }
        dft<N1, D, N>(v, tw);
#pragma unroll
        for (int k1 = 1; k1 < N1; k1++) v[k1] = twmul<D, N>(v[k1], tw, j2 * k1);
#pragma unroll
        for (int k1 = 0; k1 < N1; k1++) p[k1 * colS] = v[k1];
      }
      sync();
      for (int it = tid; it < nl * rowS; it += NT) {
        const int l = nl > 1 ? div_by(it, gz.mag_b) : 0, r = it - l * rowS;
        const int k1 = div_by(r, gz.mag_s), s = r - k1 * S;
        const int e0 = l * line + s;
        const T *p = buf + e0 + k1 * colS;
        T x[FINAL ? N2 : 1], h[FINAL ? N2 : 1];
        if constexpr (FINAL) {
#pragma unroll
          for (int k2 = 0; k2 < N2; k2++) x[k2] = a.psi[g0 + e0 + (k1 + N1 * k2) * S];
          if (horner) {
#pragma unroll
            for (int k2 = 0; k2 < N2; k2++) h[k2] = a.hbase[g0 + e0 + (k1 + N1 * k2) * S];
          }
        }
        T v[N2];
#pragma unroll
        for (int j2 = 0; j2 < N2; j2++) v[j2] = p[j2 * S];
        dft<N2, D, N, (sizeof(R) == 4 && D > 0)>(v, tw);
#pragma unroll
        for (int k2 = 0; k2 < N2; k2++) {
          const int m = VAR == FWD_PERM ? k2 + N2 * k1 : k1 + N1 * k2;
          T o = scaled ? kscale(v[k2], a.scale) : v[k2];
          if constexpr (FINAL) {
            o = cadd(o, cscale(x[k2], linev[l * N + m]));
            if (horner) o = cadd(h[k2], cmul(a.hc, o));
          }
          out[e0 + m * S] = o;
        }
      }
    }
    fence_proxy_async();
    mbar_arrive(&done[st]);  // every read of the stage is done: it may be refilled
  }
}

}  // namespace v2
}  // namespace inqb

// ------------------------------------------------------------------ host side
#include <cudaTypedefs.h>

#include <mutex>

namespace inqb {
namespace v2 {

inline PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  INQB_REQUIRE(fn != nullptr, INQB_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable");
  return fn;
}

// 4-D map of a [nx][ny][nz][S] complex array as 32-bit words; box = W states x N points along `axis`.
inline CUtensorMap orbital_map(const void *base, const Basis &b, int S, int cwords, int axis, int W) {
  CUtensorMap m;
  const cuuint64_t row = cuuint64_t(S) * cwords * 4;
  cuuint64_t dims[4] = {cuuint64_t(S) * cwords, cuuint64_t(b.n[2]), cuuint64_t(b.n[1]), cuuint64_t(b.n[0])};
  cuuint64_t strides[3] = {row, row * b.n[2], row * b.n[2] * b.n[1]};
  cuuint32_t box[4] = {cuuint32_t(W * cwords), cuuint32_t(axis == 2 ? b.n[2] : 1), cuuint32_t(axis == 1 ? b.n[1] : 1),
                       cuuint32_t(axis == 0 ? b.n[0] : 1)};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = tensor_map_encoder()(&m, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, const_cast<void *>(base), dims, strides, box,
                                    estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  INQB_REQUIRE(r == CUDA_SUCCESS, INQB_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string(int(r)) + ")");
  return m;
}

// 4-D map of the flattened-column view of a [nx][ny][nz][S] complex array as 32-bit words: y pass
// [nx][ny][nz*S], x pass [nx][ny*nz*S]; box = W columns x N points along `axis`.
inline CUtensorMap flat_map(const void *base, const Basis &b, long long ncols, int cwords, int axis, int W) {
  CUtensorMap m;
  const cuuint64_t roww = cuuint64_t(ncols) * cwords;
  const cuuint64_t d1 = cuuint64_t(axis == 1 ? b.n[1] : b.n[0]), d2 = cuuint64_t(axis == 1 ? b.n[0] : 1);
  cuuint64_t dims[4] = {roww, d1, d2, 1};
  cuuint64_t strides[3] = {roww * 4, roww * 4 * d1, roww * 4 * d1 * d2};
  cuuint32_t box[4] = {cuuint32_t(W * cwords), cuuint32_t(d1), 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = tensor_map_encoder()(&m, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, const_cast<void *>(base), dims, strides, box,
                                    estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  INQB_REQUIRE(r == CUDA_SUCCESS, INQB_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string(int(r)) + ")");
  return m;
}

template <typename R, typename CR, int N, int VAR, int WIDE = 0>
void launch_kernel(Ctx &ctx, const Basis &b, const PassArgs<R> &a, Geom2 gg) {
  using T = C2<R>;
  using TC = C2<CR>;
  constexpr int W = tile_w<R, CR, WIDE>();
  constexpr size_t TILE_BYTES = size_t(N) * W * sizeof(T);
  const int naux = has_aux(VAR) ? (a.hbase ? 2 : 1) : 0;
  constexpr bool SPLIT = sizeof(CR) > sizeof(R);
  constexpr int NT = block_threads_of<R, CR, N, VAR, WIDE>();
  // lines whose factors a flattened tile needs: at most (W - 1) / S + 2 consecutive ones
  gg.flines = ((VAR == MID_KIN || VAR == FWD_LAPLADD) && gg.flat && a.S < W) ? ((W - 1) / a.S + 3) / 2 * 2 : 2;
  const size_t fixed = (SPLIT ? size_t(N) * W * sizeof(TC) : 0) + size_t(tw_entries<CR>(N)) * sizeof(TC) +
                       size_t(gg.flines) * N * sizeof(CR) + 64 + 16 * 8;
  // second input tiles beside every ring stage when two stages of them leave room for two CTAs per SM,
  // else single-buffered (96^3 x 256: 0.80 against 0.92 ms for the single-precision final pass beside
  // every stage; 120^3 x 256 double: 3.1 against 5.35 ms single-buffered, at two CTAs per SM against one)
  gg.cpa = !gg.flat && (size_t(a.S) * sizeof(T)) % 16 != 0;
  gg.aux_single = !gg.cpa && naux > 0 && size_t(2) * (1 + naux) * TILE_BYTES + fixed > 113 * 1024;
  const size_t per_stage = TILE_BYTES * (gg.aux_single ? 1 : 1 + naux);
  const size_t fixed_aux = gg.aux_single ? naux * TILE_BYTES : 0;
  // Ring depth.  What counts is the warps per SM that cover the arithmetic's latency, then the bytes in flight;
  // measured per pass (us, one transit in and out at 6.4 TB/s in brackets):
  //  * double: two stages, so that four to six CTAs share an SM (fwd/inv y pass 120^3 x 64 630/622 -> 576/564 [549];
  //    final pass, two tiles per stage, 64^3 x 128 345 -> 252, 48^3 x 128 183 -> 113); three where the first step has
  //    exactly one item per thread (50, 60, 64, 70, 80, 84, 90, 96, 98, 100, 108, 112, 126 and 128 points: 96^3 x 128
  //    554/547 with three, 604/597 with two), and in the kinetic pass of 64 points of sets beyond L2.  A transform alone
  //    is 1 to 2 % faster with six at 40 and 48 points beyond L2 (48^3 x 128 253 against 247), H slower (497 against 502);
  //  * single, 512-byte rows: three stages for sets that stay in L2 (two to three CTAs per SM up to 72 points:
  //    48^3 x 97 37/36 with six stages, 26/24 with three [27]), four for larger ones while they fit 150 KB
  //    (72^3 x 250 276/269 with three, 240/248 with four [232]), three up to 204 KB (120^3 x 64 350/336 with
  //    two, 274/286 with three [274]); two where the steps leave part of the CTA idle in their last round
  //    (N1 no multiple of 4: 90^3 x 128 255/270 with three, 244/244 with two [232]);
  //  * other single-precision passes and wider arithmetic: about 56 KB per CTA (four per SM), two stages for sets
  //    that stay in L2 (as fast alone, and the CTAs find room beside the previous pass's last ones).
  constexpr int NTC = threads_of<R, CR, N, VAR, WIDE>();
  const bool in_l2 = stays_in_l2(b, a.S, int(sizeof(T)));
  auto bytes = [&](int n) { return per_stage * n + fixed_aux + fixed; };
  int ns;
  if (WIDE) {
    if ((W * Split<N>::N1) % NTC != 0 && bytes(2) <= 110 * 1024) ns = 2;
    else {
      ns = in_l2 ? 3 : 4;
      if (ns == 4 && bytes(4) > 150 * 1024) ns = 3;
      if (ns == 3 && bytes(3) > 204 * 1024) ns = 2;
    }
  } else if (sizeof(R) == 8) {
    constexpr bool exact = W * Split<N>::N2 == NTC;
    ns = naux == 0 && exact && (VAR != MID_KIN || !in_l2) ? 3 : 2;
  } else {
    ns = 56 * 1024 > fixed + fixed_aux ? int((56 * 1024 - fixed - fixed_aux) / per_stage) : 0;
    ns = ns < 2 || in_l2 ? 2 : (ns > 6 ? 6 : ns);
  }
  if (ctx.fft_stages > 0) {
    ns = ctx.fft_stages < 2 ? 2 : ctx.fft_stages;
    // the lengths of has_wide_arith with at least a 256-byte row of states refuse a ring that does not fit (below);
    // other sets, which ran the generic kernel whatever the depth before they had a pass of their own, take the
    // deepest ring that fits
    if (!has_wide_arith(N) || a.S < 256 / int(sizeof(T)))
      while (ns > 2 && bytes(ns) > ctx.max_smem_optin) ns--;
  }
  if (gg.cpa) ns = 2;
  gg.stages = ns;
  if (gg.flat) {
    gg.nsb = (gg.ncols + W - 1) / W;
    gg.ntiles = gg.axis == 1 ? (long long)b.n[0] * gg.nsb : gg.nsb;
  } else {
    gg.nsb = (a.S + W - 1) / W;
    gg.ntiles = (b.npoints / b.n[gg.axis]) * gg.nsb;
  }
  const size_t smem = per_stage * ns + fixed_aux + fixed;
  INQB_REQUIRE(smem <= ctx.max_smem_optin, INQB_ERR_UNSUPPORTED, "FFT tile does not fit in shared memory");
  INQB_REQUIRE(gg.ntiles < (1LL << 31), INQB_ERR_UNSUPPORTED, "FFT pass has more than 2^31 tiles");
  auto kern = fft2_kernel<R, CR, N, VAR, WIDE>;
  // per instantiation: shared-memory attribute and occupancy, computed under a lock (several host
  // threads may drive contexts at once); the attribute only ever grows
  static std::mutex mtx;
  static int occ_smem = -1, occ_per_sm = 1;
  int per_sm;
  ensure_smem_attr(reinterpret_cast<const void *>(kern), smem);
  {
    std::lock_guard<std::mutex> lock(mtx);
    if (occ_smem != int(smem)) {
      INQB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_per_sm, kern, NT, smem));
      occ_smem = int(smem);
    }
    per_sm = occ_per_sm;
  }
  long long grid = (long long)(per_sm < 1 ? 1 : per_sm) * ctx.num_sms;
  if (grid > gg.ntiles) grid = gg.ntiles;
  const int cwords = int(sizeof(T) / 4);
  // rows that are not 16-byte multiples have no tensor map; the compute threads copy them (gg.cpa)
  constexpr bool has_producer = ws_of<R, CR, N, VAR>();
  INQB_REQUIRE(!gg.cpa || has_producer, INQB_ERR_UNSUPPORTED,
               "FFT pass rows that are not 16-byte multiples need the producer-warp kernel");
  CUtensorMap mi{}, mo{}, mx{}, mb{};
  if (gg.flat) {
    mi = flat_map(a.in, b, gg.ncols, cwords, gg.axis, W);
    mo = flat_map(a.out, b, gg.ncols, cwords, gg.axis, W);
    mx = has_aux(VAR) ? flat_map(a.psi, b, gg.ncols, cwords, gg.axis, W) : mi;
    mb = mi;
  } else if (!gg.cpa) {
    mi = orbital_map(a.in, b, a.S, cwords, gg.axis, W);
    mo = orbital_map(a.out, b, a.S, cwords, gg.axis, W);
    mx = has_aux(VAR) ? orbital_map(a.psi, b, a.S, cwords, gg.axis, W) : mi;
    mb = (has_aux(VAR) && a.hbase) ? orbital_map(a.hbase, b, a.S, cwords, gg.axis, W) : mi;
  }
  const TC *tw = reinterpret_cast<const TC *>(sizeof(CR) == 8 ? b.tw64[gg.axis] : b.tw32[gg.axis]);
  // sets beyond L2 start their passes the ordinary way: CTAs that come early settle unevenly in the room the
  // previous pass leaves, and these passes are long enough for that to cost more than the launch gap (H at
  // 64^3 x 128 FP64 1202 -> 1072 us, 96^3 x 120 single 1625 -> 1592)
  pdl_launch(in_l2, kern, dim3(unsigned(grid)), NT, smem, ctx.stream, mi, mo, mx, mb, a, gg, tw, ctx.d_err);
  ctx.launches++;
}

// The plain streaming passes of single-precision sets run with 512-byte rows (64 states or flattened columns; context
// option fft_wide, default 1; launch_n says when) in two to four stages, one to three CTAs per SM (launch_kernel).
// Measured at 96^3 x 256, three stages, one CTA: 0.571 ms per pass against 0.633 ms with 256-byte rows at four CTAs per
// SM (6.35 against 5.72 TB/s).  The same shape made the kinetic pass slower, and double-precision passes (32 states,
// one CTA of 256 threads per SM) much slower (1.66 against 1.15 ms), so those keep 256-byte rows.
inline bool wide_var(int var) { return var == FWD_STORE || var == INV_STORE || var == FWD_PERM || var == INV_PERM; }

template <typename R, typename CR, int N>
void launch_nc(Ctx &ctx, const Basis &b, const PassArgs<R> &a, Geom2 gg, int var, bool wide = false) {
  if constexpr (sizeof(R) == 4 && sizeof(CR) == 4) {
    // 512-byte rows (64 single-precision states) for the plain streaming passes
    if (wide) {
      switch (var) {
        case FWD_STORE: launch_kernel<R, CR, N, FWD_STORE, 1>(ctx, b, a, gg); return;
        case INV_STORE: launch_kernel<R, CR, N, INV_STORE, 1>(ctx, b, a, gg); return;
        case FWD_PERM: launch_kernel<R, CR, N, FWD_PERM, 1>(ctx, b, a, gg); return;
        case INV_PERM: launch_kernel<R, CR, N, INV_PERM, 1>(ctx, b, a, gg); return;
        default: break;
      }
    }
  }
  switch (var) {
    case FWD_STORE: launch_kernel<R, CR, N, FWD_STORE>(ctx, b, a, gg); break;
    case INV_STORE: launch_kernel<R, CR, N, INV_STORE>(ctx, b, a, gg); break;
    case MID_KIN: launch_kernel<R, CR, N, MID_KIN>(ctx, b, a, gg); break;
    case INV_FINAL: launch_kernel<R, CR, N, INV_FINAL>(ctx, b, a, gg); break;
    case FWD_VPSI: launch_kernel<R, CR, N, FWD_VPSI>(ctx, b, a, gg); break;
    case FWD_PERM:
    case INV_PERM:
    case INV_FINAL_PERM:
      // digit-reversed passes exist for equal storage and arithmetic types only
      if constexpr (sizeof(CR) == sizeof(R)) {
        if (var == FWD_PERM) launch_kernel<R, CR, N, FWD_PERM>(ctx, b, a, gg);
        else if (var == INV_PERM) launch_kernel<R, CR, N, INV_PERM>(ctx, b, a, gg);
        else launch_kernel<R, CR, N, INV_FINAL_PERM>(ctx, b, a, gg);
      } else {
        throw Error(INQB_ERR_UNSUPPORTED, "digit-reversed FFT passes need equal storage and arithmetic types");
      }
      break;
    default: launch_kernel<R, CR, N, FWD_LAPLADD>(ctx, b, a, gg); break;
  }
}

// Arithmetic of the passes over single-precision orbitals (context option mixed_compute):
//   0 single precision everywhere; 1 double precision everywhere;
//   2 double except the final (inverse, epilogue) pass of the real-space operator;
//   3 as 2 and the first forward pass (z) of every transform also single.
// whether a pass over single-precision orbitals runs single-precision arithmetic (context option mixed_compute)
template <typename R> bool single_arith(const Ctx &ctx, const PassArgs<R> &a, int var) {
  const int mode = ctx.mixed_compute;
  const int bv = base_var(var);
  return mode == 0 || (mode >= 2 && bv == INV_FINAL) || (mode == 3 && a.axis == 2 && (bv == FWD_STORE || var == FWD_VPSI));
}

// the z pass over whole lines (fftz_kernel)
template <typename R, int N, int VAR>
void launch_zlines(Ctx &ctx, const Basis &b, const PassArgs<R> &a, const ZLines &z) {
  using T = C2<R>;
  constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2;
  GeomZ gz;
  gz.lines = (long long)b.n[0] * b.n[1];
  gz.lpt = z.lpt;
  gz.stages = z.stages;
  const long long tiles = (gz.lines + z.lpt - 1) / z.lpt;
  INQB_REQUIRE(tiles < (1LL << 31), INQB_ERR_UNSUPPORTED, "FFT pass has more than 2^31 tiles");
  gz.ntiles = int(tiles);
  auto mag = [](uint64_t d) { return d == 1 ? 0u : uint32_t(((1ull << 32) + d - 1) / d); };
  gz.mag_s = mag(uint64_t(a.S));
  gz.mag_a = mag(uint64_t(N2) * a.S);
  gz.mag_b = mag(uint64_t(N1) * a.S);
  const size_t smem = zlines_smem(N, a.S, int(sizeof(T)), z.lpt, z.stages);
  auto kern = fftz_kernel<R, N, VAR>;
  ensure_smem_attr(reinterpret_cast<const void *>(kern), smem);
  const int ctas = int((ctx.max_smem_optin + 1024) / (smem + 1024));
  long long grid = (long long)(ctas < 1 ? 1 : (ctas > 8 ? 8 : ctas)) * ctx.num_sms;
  if (grid > tiles) grid = tiles;
  const T *tw = reinterpret_cast<const T *>(sizeof(R) == 8 ? b.tw64[2] : b.tw32[2]);
  // an early start whatever the set's size: beyond L2 it gains or costs less than 1 % of H (72^3 x 31 double 460 against
  // 466 us without, 96^3 x 62 1797 against 1806, 64^3 x 79 724 against 705; single 72^3 x 180 1205 against 1207)
  pdl_launch(true, kern, dim3(unsigned(grid)), z.threads + 32, smem, ctx.stream, a, gz, tw, ctx.d_err);
  ctx.launches++;
}

template <typename R, int N>
void launch_n(Ctx &ctx, const Basis &b, const PassArgs<R> &a, Geom2 gg, int var) {
  if (gg.axis == 2 && (sizeof(R) == 8 || single_arith(ctx, a, var))) {
    const ZLines z = zlines_of(ctx, b, a.S, int(sizeof(C2<R>)));
    const bool tiles = sizeof(R) == 4 && base_var(var) == INV_FINAL && final_tiles(b, N, a.S);
    if (z.lpt > 0 && !tiles) {
      switch (var) {
        case FWD_STORE: launch_zlines<R, N, FWD_STORE>(ctx, b, a, z); return;
        case INV_STORE: launch_zlines<R, N, INV_STORE>(ctx, b, a, z); return;
        case INV_FINAL: launch_zlines<R, N, INV_FINAL>(ctx, b, a, z); return;
        case FWD_VPSI: launch_zlines<R, N, FWD_VPSI>(ctx, b, a, z); return;
        case FWD_PERM: launch_zlines<R, N, FWD_PERM>(ctx, b, a, z); return;
        case INV_PERM: launch_zlines<R, N, INV_PERM>(ctx, b, a, z); return;
        case INV_FINAL_PERM: launch_zlines<R, N, INV_FINAL_PERM>(ctx, b, a, z); return;
        default: break;
      }
    }
  }
  if constexpr (sizeof(R) == 4) {
    const bool single = single_arith(ctx, a, var);
    if (single) {
      // 64-state tiles unless they would leave more of the last tile empty than 32-state tiles do
      // (85 states: 43 empty slots against 11)
      const int pad64 = (64 - a.S % 64) % 64, pad32 = (32 - a.S % 32) % 32;
      const bool wide = ctx.fft_wide && wide_var(var) && (gg.flat || (a.S >= 64 && pad64 <= pad32 + 8));
      launch_nc<R, float, N>(ctx, b, a, gg, var, wide);
      return;
    }
    if constexpr (has_wide_arith(N)) launch_nc<R, double, N>(ctx, b, a, gg, var);
    else throw Error(INQB_ERR_UNSUPPORTED, "no double-precision arithmetic for this line length");
  } else {
    launch_nc<R, double, N>(ctx, b, a, gg, var);
  }
}

// one length's kernels, each instantiated in one of the fft2_inst_*.cu files
#define INQB_X(N, A, B)                                                                                    \
  extern template void launch_n<float, N>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);      \
  extern template void launch_n<double, N>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
INQB_FFT2_LENGTHS(INQB_X)
#undef INQB_X

// Returns false (and does nothing) when the pass is not covered by a specialised kernel.
template <typename R> bool launch(Ctx &ctx, const Basis &b, const PassArgs<R> &a, int prologue, int epilogue) {
  using T = C2<R>;
  if (ctx.fft_impl == 1) return false;
  const int n = b.n[a.axis];
  if (split_n2(n) == 0) return false;
  int var;
  if (a.mid_kinetic) var = MID_KIN;
  else if (prologue == PRO_VPSI) var = FWD_VPSI;
  else if (epilogue == EPI_FINAL_REAL) var = INV_FINAL;
  else if (epilogue == EPI_LAPL_ADD) var = FWD_LAPLADD;
  else var = a.dir > 0 ? FWD_STORE : INV_STORE;
  if ((var == INV_FINAL && a.dir > 0) || ((var == FWD_VPSI || var == FWD_LAPLADD) && a.dir < 0)) return false;
  const bool same_type = sizeof(R) == 8 || single_arith(ctx, a, var);
  if (!same_type && !has_wide_arith(n)) return false;
  // y and x passes over flattened columns (their second input, the Laplacian term's, lies alike)
  const bool flat = flat_ok(ctx, b, a.S, int(sizeof(T)), a.axis) &&
                    (var == FWD_STORE || var == INV_STORE || var == MID_KIN || var == FWD_LAPLADD);
  const bool zl = a.axis == 2 && same_type && zlines_of(ctx, b, a.S, int(sizeof(T))).lpt > 0;
  if (!flat && !zl) {
    if (a.S < 256 / int(sizeof(T))) return false;  // fewer states than one 256-byte row: generic kernel
    // rows that are not 16-byte multiples (an odd number of single-precision states): only the kernels with
    // a producer warp (single-precision arithmetic) move them, with 8-byte copies; otherwise the generic kernel
    if ((size_t(a.S) * sizeof(T)) % 16 != 0 && !(sizeof(R) == 4 && same_type)) return false;
  }
  if (a.perm) {
    INQB_REQUIRE(var == FWD_STORE || var == INV_STORE || var == INV_FINAL, INQB_ERR_UNSUPPORTED,
                 "digit-reversed frequency order is only kept by the plain forward and inverse passes");
    var = var == FWD_STORE ? FWD_PERM : (var == INV_STORE ? INV_PERM : INV_FINAL_PERM);
  }

  constexpr int W = 256 / int(sizeof(T));
  Geom2 gg;
  for (int i = 0; i < 3; i++) gg.g.n[i] = b.n[i];
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) gg.g.rlat[i][j] = b.rlat[i][j];
  const long long ny = b.n[1], nz = b.n[2];
  if (a.axis == 2) { gg.g.nb = int(ny); gg.g.sa = ny * nz; gg.g.sb = nz; gg.g.sp = 1; }
  else if (a.axis == 1) { gg.g.nb = int(nz); gg.g.sa = ny * nz; gg.g.sb = 1; gg.g.sp = nz; }
  else { gg.g.nb = int(nz); gg.g.sa = nz; gg.g.sb = 1; gg.g.sp = ny * nz; }
  gg.axis = a.axis;
  gg.flat = flat ? 1 : 0;
  gg.ncols = a.axis == 1 ? nz * a.S : ny * nz * a.S;
  gg.nsb = (a.S + W - 1) / W;
  gg.ntiles = (b.npoints / n) * gg.nsb;
  gg.cwords = int(sizeof(T) / 4);
  gg.stages = 2;
  switch (n) {
#define INQB_X(N, A, B) case N: launch_n<R, N>(ctx, b, a, gg, var); break;
    INQB_FFT2_LENGTHS(INQB_X)
#undef INQB_X
  }
  return true;
}

}  // namespace v2
}  // namespace inqb
