// Nonlocal projector kernels and the orbital-set kernels around the FFT passes.
//
// Every reduction here has a fixed order (warp shuffles in a fixed tree, per-block
// partials summed in index order by a second kernel), so results are bitwise
// reproducible run to run; no floating-point atomics are used anywhere.

#include "inqb_internal.h"
#include "ptx.cuh"

#include <algorithm>
#include <mutex>

namespace inqb {

static inline unsigned grid_for(long long n, int threads, long long cap = 148LL * 64) {
  long long g = (n + threads - 1) / threads;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return unsigned(g);
}

#define LAUNCHED(ctx)                   \
  do {                                  \
    INQB_CUDA(cudaGetLastError());      \
    (ctx).launches++;                   \
  } while (0)

// ------------------------------------------------------------------ nonlocal tables
// gcoef[p][i][l] = dV * e^{+i kA.pos} * M[p][l][i]   (gather side, projector_all.hpp:120-128,156)
// hcoef[h][l]    = e^{-i kA.pos} * M[p][l][i]        (apply side, projector_all.hpp:281-287)
__global__ void nl_tables_kernel(int nproj, int maxsph, const int *__restrict__ pt, const float *__restrict__ pos,
                                 const double *__restrict__ mat, double dv, double k0, double k1, double k2,
                                 double2 *gcoef, float2 *gcoef32) {
  const long long total = (long long)nproj * maxsph;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int p = int(idx / maxsph), i = int(idx % maxsph);
    double2 ph = make_double2(0.0, 0.0);
    if (pt[idx] >= 0) {
      // dot(kpoint, pos) of the reference: covariant double times float contravariant
      double arg = k0 * double(pos[idx * 3 + 0]) + k1 * double(pos[idx * 3 + 1]) + k2 * double(pos[idx * 3 + 2]);
      double sn, cs;
      sincos(arg, &sn, &cs);
      ph = make_double2(cs, sn);
    }
    for (int l = 0; l < 4; l++) {
      double m = mat[((long long)p * 4 + l) * maxsph + i];
      double2 g = make_double2(dv * m * ph.x, dv * m * ph.y);
      gcoef[idx * 4 + l] = g;
      gcoef32[idx * 4 + l] = make_float2(float(g.x), float(g.y));
    }
  }
}

__global__ void nl_hit_kernel(long long total, const int *__restrict__ hit, int maxsph, const float *__restrict__ pos,
                              const double *__restrict__ mat, double k0, double k1, double k2, double2 *hcoef,
                              float2 *hcoef32) {
  for (long long h = blockIdx.x * (long long)blockDim.x + threadIdx.x; h < total;
       h += (long long)gridDim.x * blockDim.x) {
    const long long idx = hit[h];
    const int p = int(idx / maxsph), i = int(idx % maxsph);
    double arg = k0 * double(pos[idx * 3 + 0]) + k1 * double(pos[idx * 3 + 1]) + k2 * double(pos[idx * 3 + 2]);
    double sn, cs;
    sincos(arg, &sn, &cs);
    for (int l = 0; l < 4; l++) {
      double m = mat[((long long)p * 4 + l) * maxsph + i];
      double2 c = make_double2(m * cs, -m * sn);
      hcoef[h * 4 + l] = c;
      hcoef32[h * 4 + l] = make_float2(float(c.x), float(c.y));
    }
  }
}

void launch_nl_tables(Ctx &ctx, const Basis &b, Hamiltonian &h, const double kA[3]) {
  Projectors &P = h.proj;
  if (P.nproj == 0 || P.maxsph == 0) return;
  const double dv = b.volume / double(b.npoints);
  const long long total = (long long)P.nproj * P.maxsph;
  nl_tables_kernel<<<grid_for(total, 256), 256, 0, ctx.stream>>>(P.nproj, P.maxsph, P.d_pt, P.d_pos, P.d_mat, dv,
                                                                 kA[0], kA[1], kA[2], P.d_gcoef, P.d_gcoef32);
  LAUNCHED(ctx);
  if (P.total > 0) {
    nl_hit_kernel<<<grid_for(P.total, 256), 256, 0, ctx.stream>>>(P.total, P.d_hit, P.maxsph, P.d_pos, P.d_mat, kA[0],
                                                                  kA[1], kA[2], P.d_hcoef, P.d_hcoef32);
    LAUNCHED(ctx);
  }
  for (int i = 0; i < 3; i++) P.kA[i] = kA[i];
}

// ------------------------------------------------------------------ bulk-copy kernels: shared pieces
// acc + a * b as four fused multiply-adds (one rounding per product term)
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
template <typename T> __device__ __forceinline__ T cmac(T acc, T a, T b) {
  acc.x = fma_rn(a.x, b.x, acc.x);
  acc.x = fma_rn(-a.y, b.y, acc.x);
  acc.y = fma_rn(a.x, b.y, acc.y);
  acc.y = fma_rn(a.y, b.x, acc.y);
  return acc;
}

// The bulk-copy forms of the projection and the apply run NLA_NT compute threads beside one producer
// warp that moves whole rows of states (contiguous in the state-fastest layout) with bulk
// asynchronous copies.  The projection's compute threads synchronise among
// themselves on named barrier 1.
constexpr int NLA_NT = 128;

// that barrier, returning whether any compute thread passed a nonzero value (uniform result)
__device__ __forceinline__ bool nla_sync_or(int v) {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
               : "=r"(r)
               : "r"(v), "n"(NLA_NT)
               : "memory");
  return r != 0;
}
// bounded wait on an mbarrier phase (2 s); false, with the CTA's abort flag and the error flag raised,
// on expiry, and false as soon as another thread of the CTA has raised the abort flag
__device__ __forceinline__ bool nla_wait(uint64_t *b, uint32_t parity, volatile int *abort_flag, int *err) {
  const uint64_t t0 = ptx::global_ns();
  while (!ptx::mbar_try_wait(b, parity)) {
    if (*abort_flag) return false;
    if (ptx::global_ns() - t0 > 2000000000ull) {
      *abort_flag = 1;
      atomicExch(err, 1);
      return false;
    }
  }
  return true;
}

// ------------------------------------------------------------------ nonlocal projection
// proj[p][l][s] = sum_i gcoef[p][i][l] * psi[pt_i][s]; projD = coeff[p] . proj
// (projector_all.hpp:113-211).  Stage 1: CTA = (projector p, range rg of its sphere points, chunk of
// K << sl states); each of its 8 warps takes a contiguous run of the range, reads 32 point indices with
// one coalesced load and hands them out by shuffles, and keeps NP points per lane group in flight.  A group
// of 2^sl lanes holds K states each, 2^sl apart; sets of at most 32 states use groups of as many lanes as
// they have states (a power of two), so that a warp takes several points at a time instead of idling its
// lanes.  Groups are summed by shuffles in a fixed tree, the warps in order into partial[p][rg][l][s].
// Stage 2 sums the ranges in order and applies the KB coefficients.  Latency-bound (a chain of index, row
// and coefficient loads per batch): what counts is few batches per warp.
constexpr int NLP_WARPS = 8, NLP_RANGES = 16;  // 16 ranges: the bulk projection 181 us against 218 with 8 (FP64, 96^3 x 256)
constexpr int NLP_MAX_RANGES = 32;

template <typename R, typename A, int K, int NP>
__global__ void __launch_bounds__(NLP_WARPS * 32) nl_project_kernel(const C2<R> *__restrict__ psi, int S, int sl,
                                                                    const int *__restrict__ pt,
                                                                    const C2<A> *__restrict__ gcoef,
                                                                    const int *__restrict__ npts, int maxsph,
                                                                    C2<A> *__restrict__ partial) {
  using T = C2<R>;
  using TA = C2<A>;
  __shared__ TA part[NLP_WARPS][4][32 * K];
  const int p = blockIdx.x, rg = blockIdx.y;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int SL = 1 << sl, G = 32 >> sl;        // lanes per group, groups per warp
  const int ls = lane & (SL - 1), g = lane >> sl;
  const int sbase = blockIdx.z * SL * K;
  ptx::grid_wait();
  ptx::grid_release();
  const int np = npts[p];
  const int nr = int(gridDim.y);  // ranges of a sphere
  const int rper = (np + nr - 1) / nr;
  const int r0 = rg * rper, r1 = min(np, r0 + rper);
  const int per = (max(r1 - r0, 0) + NLP_WARPS - 1) / NLP_WARPS;
  const int i0 = r0 + wp * per, i1 = min(r1, i0 + per);
  TA acc[K][4];
#pragma unroll
  for (int k = 0; k < K; k++)
#pragma unroll
    for (int l = 0; l < 4; l++) acc[k][l] = mk<TA>(A(0), A(0));
  const long long rowbase = (long long)p * maxsph;
  for (int base = i0; base < i1; base += 32) {
    const int cnt = min(32, i1 - base);
    const int qv = lane < cnt ? __ldg(&pt[rowbase + base + lane]) : 0;
    for (int j = 0; j < cnt; j += NP * G) {
      T x[NP][K];
#pragma unroll
      for (int u = 0; u < NP; u++) {
        const int i = j + u * G + g;
        const long long q = __shfl_sync(0xffffffffu, qv, i & 31);
#pragma unroll
        for (int k = 0; k < K; k++) {
          const int s = sbase + k * SL + ls;
          x[u][k] = (i < cnt && s < S) ? psi[q * S + s] : mk<T>(R(0), R(0));
        }
      }
#pragma unroll
      for (int u = 0; u < NP; u++) {
        const int i = j + u * G + g;
        if (i < cnt) {
          const TA *gc = gcoef + (rowbase + base + i) * 4;
          TA gl[4];
#pragma unroll
          for (int l = 0; l < 4; l++) gl[l] = gc[l];
#pragma unroll
          for (int k = 0; k < K; k++) {
            const TA v = mk<TA>(A(x[u][k].x), A(x[u][k].y));
#pragma unroll
            for (int l = 0; l < 4; l++) acc[k][l] = cadd(acc[k][l], cmul(gl[l], v));
          }
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < K; k++)
#pragma unroll
    for (int l = 0; l < 4; l++) {
      for (int o = 16; o >= SL; o >>= 1) {
        acc[k][l].x += __shfl_down_sync(0xffffffffu, acc[k][l].x, o);
        acc[k][l].y += __shfl_down_sync(0xffffffffu, acc[k][l].y, o);
      }
      if (g == 0) part[wp][l][k * SL + ls] = acc[k][l];
    }
  __syncthreads();
  for (int e = threadIdx.x; e < 4 * SL * K; e += blockDim.x) {
    const int l = e / (SL * K), c = e % (SL * K);
    const int s = sbase + c;
    TA t = part[0][l][c];
    for (int w = 1; w < NLP_WARPS; w++) t = cadd(t, part[w][l][c]);
    if (s < S) partial[(((long long)p * nr + rg) * 4 + l) * S + s] = t;
  }
}

// Bulk-copy form of the projection.  CTA = (projector p, range rg of its sphere points, chunk of up to
// NLA_NT * J states).  The producer warp copies the range's points in batches of KB -- each point's
// row of the chunk's states and the point's four gather coefficients -- into a ring of NLP_NS stages;
// each compute thread owns J states and sums over the range's points in order (a batch's points first,
// then the batch sums, so the chains stay as short as in nl_project_kernel).  No cross-warp reduction:
// the thread writes its states of partial[p][rg][l][s] directly.
constexpr int NLP_NS = 3;

template <typename R, typename A, int J>
__global__ void __launch_bounds__(NLA_NT + 32) nl_project_bulk_kernel(const C2<R> *psi, int S,
                                                                       const int *__restrict__ pt,
                                                                       const C2<A> *gcoef,
                                                                       const int *__restrict__ npts, int maxsph,
                                                                       int KB, C2<A> *__restrict__ partial, int *err) {
  using T = C2<R>;
  using TA = C2<A>;
  using namespace ptx;
  extern __shared__ __align__(128) unsigned char smem[];
  const int p = blockIdx.x, rg = blockIdx.y;
  const int s0 = blockIdx.z * NLA_NT * J;
  const int SCmax = min(NLA_NT * J, S);  // row stride of the stages
  const int SC = min(NLA_NT * J, S - s0);  // states of this chunk
  T *rows = reinterpret_cast<T *>(smem);                                     // [NS][KB][SCmax]
  TA *gs = reinterpret_cast<TA *>(rows + size_t(NLP_NS) * KB * SCmax);        // [NS][KB][4]
  uint64_t *full = reinterpret_cast<uint64_t *>(gs + size_t(NLP_NS) * KB * 4);  // stage loaded
  uint64_t *done = full + NLP_NS;                                            // stage consumed
  volatile int *abort_flag = reinterpret_cast<volatile int *>(done + NLP_NS);
  const long long rowbase = (long long)p * maxsph;
  const uint32_t row_bytes = uint32_t(SC) * uint32_t(sizeof(T));
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int st = 0; st < NLP_NS; st++) {
      mbar_init(&full[st], 1);
      mbar_init(&done[st], NLA_NT);
    }
    mbar_init_fence();
  }
  __syncthreads();
  grid_wait();
  grid_release();
  const int np = npts[p];
  const int nr = int(gridDim.y);  // ranges of a sphere
  const int rper = (np + nr - 1) / nr;
  const int r0 = rg * rper, r1 = min(np, r0 + rper);
  const int n = max(r1 - r0, 0);
  const int nbatch = (n + KB - 1) / KB;

  if (threadIdx.x >= NLA_NT) {
    // producer warp: lane q copies point q of a batch, lane 0 also the batch's coefficients
    const int lane = threadIdx.x - NLA_NT;
    auto issue = [&](int st, int b) {
      const int base = r0 + b * KB;
      const int nb = min(KB, r1 - base);
      const long long q = lane < nb ? (long long)pt[rowbase + base + lane] : 0;
      if (lane == 0) mbar_expect_tx(&full[st], uint32_t(nb) * (row_bytes + 4 * uint32_t(sizeof(TA))));
      __syncwarp();
      if (lane < nb) bulk_load(rows + (size_t(st) * KB + lane) * SCmax, psi + q * S + s0, row_bytes, &full[st]);
      if (lane == 0)
        bulk_load(gs + size_t(st) * KB * 4, gcoef + (rowbase + base) * 4, uint32_t(nb) * 4 * uint32_t(sizeof(TA)),
                  &full[st]);
    };
    int issued = 0;  // batches whose copies were issued
    for (int b = 0; b < NLP_NS && b < nbatch; b++) issue(b, b), issued++;
    for (int b = 0; b + NLP_NS < nbatch; b++) {
      const int st = b % NLP_NS;
      if (!nla_wait(&done[st], uint32_t(b / NLP_NS) & 1u, abort_flag, err)) break;
      issue(st, b + NLP_NS);
      issued++;
    }
    // after an abort the compute threads may leave early: wait (bounded) for every issued copy to land
    // before the CTA's shared memory is released (on the normal path these phases are already complete)
    for (int b = issued - NLP_NS < 0 ? 0 : issued - NLP_NS; b < issued; b++)
      mbar_wait_bounded(&full[b % NLP_NS], uint32_t(b / NLP_NS) & 1u, 2000000000ull);
    return;
  }

  const int tid = threadIdx.x;
  TA acc[J][4];
#pragma unroll
  for (int j = 0; j < J; j++)
#pragma unroll
    for (int l = 0; l < 4; l++) acc[j][l] = mk<TA>(A(0), A(0));
  for (int b = 0; b < nbatch; b++) {
    const int st = b % NLP_NS;
    const bool ok = nla_wait(&full[st], uint32_t(b / NLP_NS) & 1u, abort_flag, err);
    if (nla_sync_or(!ok || *abort_flag)) break;
    const int nb = min(KB, r1 - (r0 + b * KB));
    const T *rw = rows + size_t(st) * KB * SCmax;
    const TA *g = gs + size_t(st) * KB * 4;
    TA bacc[J][4];
#pragma unroll
    for (int j = 0; j < J; j++)
#pragma unroll
      for (int l = 0; l < 4; l++) bacc[j][l] = mk<TA>(A(0), A(0));
    for (int q = 0; q < nb; q++) {
      TA gl[4];
#pragma unroll
      for (int l = 0; l < 4; l++) gl[l] = g[q * 4 + l];
#pragma unroll
      for (int j = 0; j < J; j++) {
        const int sl = tid + j * NLA_NT;
        if (sl < SC) {
          const T x = rw[(size_t)q * SCmax + sl];
          const TA v = mk<TA>(A(x.x), A(x.y));
          // fused products in single precision (0.10 against 0.11 ms at 96^3 x 256); separate ones in
          // double (0.18 against 0.19 ms)
          if constexpr (sizeof(A) == 4) {
#pragma unroll
            for (int l = 0; l < 4; l++) bacc[j][l] = cmac(bacc[j][l], gl[l], v);
          } else {
#pragma unroll
            for (int l = 0; l < 4; l++) bacc[j][l] = cadd(bacc[j][l], cmul(gl[l], v));
          }
        }
      }
    }
#pragma unroll
    for (int j = 0; j < J; j++)
#pragma unroll
      for (int l = 0; l < 4; l++) acc[j][l] = cadd(acc[j][l], bacc[j][l]);
    mbar_arrive(&done[st]);  // the producer refills the stage
  }
#pragma unroll
  for (int j = 0; j < J; j++) {
    const int sl = tid + j * NLA_NT;
    if (sl < SC) {
#pragma unroll
      for (int l = 0; l < 4; l++) partial[(((long long)p * nr + rg) * 4 + l) * S + s0 + sl] = acc[j][l];
    }
  }
}

// Block = 32 states x 4 functions of one projector: a thread sums its function's ranges in order, eight
// loads in flight (one thread per projector and state, with a load at a time, took 10 us at any size).
constexpr int NLF_S = 32;

template <typename R, typename A>
__global__ void __launch_bounds__(NLF_S * 4) nl_project_finish_kernel(const C2<A> *__restrict__ partial, int nsb, int nr,
                                                                      int S, const A *__restrict__ coeff,
                                                                      C2<R> *projraw, C2<R> *projD) {
  using T = C2<R>;
  using TA = C2<A>;
  __shared__ TA pr[4][NLF_S];
  const int p = blockIdx.x / nsb, l = threadIdx.x / NLF_S, c = threadIdx.x % NLF_S;
  const int s = (blockIdx.x % nsb) * NLF_S + c;
  ptx::grid_wait();
  ptx::grid_release();
  if (s < S) {
    const TA *src = partial + ((long long)p * nr * 4 + l) * S + s;
    const long long step = 4LL * S;
    TA t = src[0];
    int rg = 1;
    for (; rg + 8 <= nr; rg += 8) {
      TA v[8];
#pragma unroll
      for (int u = 0; u < 8; u++) v[u] = src[(rg + u) * step];
#pragma unroll
      for (int u = 0; u < 8; u++) t = cadd(t, v[u]);
    }
    TA v[7];
#pragma unroll
    for (int u = 0; u < 7; u++) v[u] = rg + u < nr ? src[(rg + u) * step] : mk<TA>(A(0), A(0));
#pragma unroll
    for (int u = 0; u < 7; u++)
      if (rg + u < nr) t = cadd(t, v[u]);
    pr[l][c] = t;
    projraw[((long long)p * 4 + l) * S + s] = mk<T>(R(t.x), R(t.y));
  }
  __syncthreads();
  if (s < S) {
    TA t = mk<TA>(A(0), A(0));
#pragma unroll
    for (int j = 0; j < 4; j++) t = cadd(t, cscale(pr[j][c], coeff[(p * 4 + l) * 4 + j]));
    projD[((long long)p * 4 + l) * S + s] = mk<T>(R(t.x), R(t.y));
  }
}

template <typename R>
void launch_nl_project(Ctx &ctx, const Basis &b, const Hamiltonian &h, const C2<R> *psi, int S, C2<R> *projraw,
                       C2<R> *projD) {
  const Projectors &P = h.proj;
  if (P.nproj == 0) return;
  const bool dbl = sizeof(R) == 8 || ctx.mixed_compute != 0;  // double-precision coefficients and sums
  // ranges per sphere (option nl_project_ranges; the summation order follows it)
  int NR = ctx.nl_project_ranges > 0 ? ctx.nl_project_ranges : NLP_RANGES;
  // bulk form: rows of 16-byte multiples, and (automatic choice) more than 32 states and two CTAs per SM, with
  // the ranges the option asks for or, where it leaves them open, at most 32; the choice (and so the summation
  // order) follows the device's SM count, not the grid_sms option.  Fewer states leave most of the bulk form's threads idle: 8 states of 24 projectors
  // 29 us against 9 in the register form; 50 FP64 states of 12 projectors 19 against 28.
  constexpr int JB = 2;
  const size_t row_bytes = size_t(S) * sizeof(C2<R>);
  const int nchunks = (S + NLA_NT * JB - 1) / (NLA_NT * JB);
  const bool bulk_ok = row_bytes % 16 == 0 && reinterpret_cast<uintptr_t>(psi) % 16 == 0;
  const int most = ctx.nl_project_ranges > 0 ? NR : std::max(NR, NLP_MAX_RANGES);
  const bool bulk = bulk_ok && (ctx.nl_bulk > 0 || (ctx.nl_bulk == 0 && S > 32 &&
                                                    (long long)P.nproj * most * nchunks >= 2LL * ctx.device_sms));
  // register form: two states per lane, or one in lane groups of a power of two
  int sl = 5, K = 2;
  if (S <= 32) {
    K = 1;
    for (sl = 0; (1 << sl) < S; sl++) {
    }
  }
  const int rchunks = (S + (K << sl) - 1) / (K << sl);
  // few projectors: more, shorter ranges until the device has two CTAs per SM (8 projectors of 16 FP64 states:
  // projection and finish 10.7 us with 16 ranges, 9.4 with 32, 13.7 with 64)
  if (ctx.nl_project_ranges == 0)
    while (NR < NLP_MAX_RANGES && (long long)P.nproj * NR * (bulk ? nchunks : rchunks) < 2LL * ctx.device_sms) NR *= 2;
  void *partial = dev_alloc(ctx, size_t(P.nproj) * NR * 4 * S * (dbl ? sizeof(double2) : sizeof(float2)));
  auto go = [&](auto atype) {
    using A = decltype(atype);
    using TA = C2<A>;
    const TA *gcoef;
    const A *coeff;
    if constexpr (sizeof(A) == 8) gcoef = P.d_gcoef, coeff = P.d_coeff;
    else gcoef = P.d_gcoef32, coeff = P.d_coeff32;
    TA *part = static_cast<TA *>(partial);
    if (bulk) {
      const int SCmax = std::min(NLA_NT * JB, S);
      const size_t srow = size_t(SCmax) * sizeof(C2<R>);
      int KB = ctx.nl_project_points > 0 ? ctx.nl_project_points : int(16384 / srow);  // about 16 KB of rows per stage
      KB = KB < 1 ? 1 : (KB > 32 ? 32 : KB);
      auto smem_of = [&](int kb) {
        return size_t(NLP_NS) * kb * srow + size_t(NLP_NS) * kb * 4 * sizeof(TA) + 2 * NLP_NS * sizeof(uint64_t) + 16;
      };
      while (KB > 1 && smem_of(KB) > size_t(ctx.max_smem_optin)) KB--;  // an option asking for more than fits
      const size_t smem = smem_of(KB);
      auto kern = nl_project_bulk_kernel<R, A, JB>;
      ensure_smem_attr(reinterpret_cast<const void *>(kern), smem);
      pdl_launch(true, kern, dim3(P.nproj, NR, nchunks), NLA_NT + 32, smem, ctx.stream, psi, S, P.d_pt, gcoef, P.d_npts, P.maxsph,
                 KB, part, ctx.d_err);
    } else {
      const dim3 grid(P.nproj, NR, rchunks);
      // four points in flight at two states per lane (eight: 94 against 50 us at 72^3 x 99 single)
      if (K == 2)
        pdl_launch(true, nl_project_kernel<R, A, 2, 4>, grid, NLP_WARPS * 32, 0, ctx.stream, psi, S, sl, P.d_pt, gcoef, P.d_npts,
                   P.maxsph, part);
      else
        pdl_launch(true, nl_project_kernel<R, A, 1, 8>, grid, NLP_WARPS * 32, 0, ctx.stream, psi, S, sl, P.d_pt, gcoef, P.d_npts,
                   P.maxsph, part);
    }
    ctx.launches++;
    const int nsb = (S + NLF_S - 1) / NLF_S;
    pdl_launch(true, nl_project_finish_kernel<R, A>, dim3(unsigned(P.nproj) * nsb), NLF_S * 4, 0, ctx.stream, part, nsb, NR, S,
               coeff, projraw, projD);
    ctx.launches++;
  };
  if (dbl) go(double());
  else go(float());
  dev_free(ctx, partial);
}

// out[pt][s] = nonlocal term (ks_hamiltonian::non_local, ks_hamiltonian.hpp:106-120)
template <typename R>
__global__ void nl_scatter_kernel(long long npoints, int S, const int *__restrict__ offs, const int *__restrict__ hit,
                                  const C2<R> *__restrict__ hcoef, const C2<R> *__restrict__ projD, int maxsph,
                                  C2<R> *out) {
  using T = C2<R>;
  const long long total = npoints * S;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const long long pt = e / S;
    const int s = int(e % S);
    T acc = mk<T>(R(0), R(0));
    for (int hh = offs[pt]; hh < offs[pt + 1]; hh++) {
      const int p = hit[hh] / maxsph;
#pragma unroll
      for (int l = 0; l < 4; l++) acc = cadd(acc, cmul(hcoef[(long long)hh * 4 + l], projD[((long long)p * 4 + l) * S + s]));
    }
    out[e] = acc;
  }
}

template <typename R>
void launch_nl_scatter(Ctx &ctx, const Basis &b, const Hamiltonian &h, const C2<R> *projD, int S, C2<R> *out) {
  const Projectors &P = h.proj;
  const C2<R> *hc;
  if constexpr (sizeof(R) == 8) hc = P.d_hcoef;
  else hc = P.d_hcoef32;
  nl_scatter_kernel<R><<<grid_for(b.npoints * S, 256), 256, 0, ctx.stream>>>(b.npoints, S, P.d_offs, P.d_hit, hc,
                                                                             projD, P.maxsph, out);
  LAUNCHED(ctx);
}

// out[pt][s] += nonlocal term at the grid points that lie in a sphere (ks_hamiltonian.hpp:153,
// projector_all.hpp:276-288), hits of a point summed in projector order, no atomics; optionally scaled,
// out += scale * term (a Horner step of a Taylor exponential), or with the local potential,
// out = (V + vshift) out + term (the Fourier form, whose next pass multiplies the other points by it).
template <typename R> struct NlApply {
  const int4 *hrec;
  const int *hitp;
  const C2<R> *hcoef;
  const C2<R> *projD;
  C2<R> *out;
  int S;
  bool scaled;
  C2<R> scale;
  const R *V;  // null: out += term
  int nspin, spin;
  R vshift;
};
// the term's first hit is summed by the caller (fused products); the others follow
// VM: 0 without the local potential, 1 with it, 2 with it and V + vshift and its product in double (the passes'
// arithmetic is double then); a runtime choice cost 177 against 155 us at 96^3 x 256 single
template <typename R, int VM>
__device__ __forceinline__ C2<R> nl_value(const NlApply<R> &a, long long pt, int s, int h0, int nh, C2<R> o,
                                          const C2<R> (&hc)[4], const C2<R> (&pd)[4]) {
  using T = C2<R>;
  T accv = mk<T>(R(0), R(0));
#pragma unroll
  for (int l = 0; l < 4; l++) accv = cmac(accv, hc[l], pd[l]);
#pragma unroll 1  // few points lie in more than one sphere: no registers for them
  for (int k = 1; k < nh; k++) {
    const int h = h0 + k;
    const int p = a.hitp[h];
#pragma unroll
    for (int l = 0; l < 4; l++)
      accv = cadd(accv, cmul(a.hcoef[(long long)h * 4 + l], a.projD[((long long)p * 4 + l) * a.S + s]));
  }
  if constexpr (VM == 1) o = cscale(o, a.V[pt * a.nspin + a.spin] + a.vshift);
  if constexpr (VM == 2) {
    const double v = double(a.V[pt * a.nspin + a.spin]) + double(a.vshift);
    o = mk<T>(R(double(o.x) * v), R(double(o.y) * v));
  }
  return cadd(o, a.scaled ? cmul(a.scale, accv) : accv);
}

// Register form.  Owner computes: one group of 2^sl lanes per (grid point with sphere hits, chunk of
// U << sl states), lanes over states.  The point's record gives its first hit and projector in one load, so
// the coefficient, projection and output reads are all issued together (a two-level dependency instead of
// point -> CSR -> hit -> projection); splitting the states into chunks keeps the registers low and many
// warps resident.
template <typename R, int U, int VM>
__global__ void __launch_bounds__(128) nl_apply_kernel(NlApply<R> a, long long nitems, int nchunks, int sl) {
  using T = C2<R>;
  const int S = a.S, SL = 1 << sl;
  const int ls = threadIdx.x & (SL - 1);
  const long long group = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> sl;
  const long long ngroups = ((long long)gridDim.x * blockDim.x) >> sl;
  ptx::grid_wait();
  ptx::grid_release();
  // the record of the group's next item is requested while the current one is processed
  int4 next = group < nitems ? a.hrec[group / nchunks] : make_int4(0, 0, 0, 0);
  for (long long it = group; it < nitems; it += ngroups) {
    const int s0 = int(it % nchunks) * (SL * U);
    const int4 rec = next;
    if (it + ngroups < nitems) next = a.hrec[(it + ngroups) / nchunks];
    const long long pt = rec.x;
    const int h0 = rec.y, nh = rec.z, p0 = rec.w;
    T hc[4], o[U], pd[U][4];
#pragma unroll
    for (int l = 0; l < 4; l++) hc[l] = a.hcoef[(long long)h0 * 4 + l];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int s = s0 + u * SL + ls;
      if (s < S) {
        o[u] = a.out[pt * S + s];
#pragma unroll
        for (int l = 0; l < 4; l++) pd[u][l] = a.projD[((long long)p0 * 4 + l) * S + s];
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int s = s0 + u * SL + ls;
      if (s < S) a.out[pt * S + s] = nl_value<R, VM>(a, pt, s, h0, nh, o[u], hc, pd[u]);
    }
  }
}

// Bulk-copy form of the apply.  A CTA takes batches of KB consecutive hit points: a producer warp copies
// the points' output rows (S contiguous states each) into shared memory with bulk asynchronous copies, two
// batches ahead, so the copy engine keeps the bytes in flight that the register form cannot; the compute
// threads, in groups of 2^ts per row, add the nonlocal term and store the rows to global memory, or with BS
// to shared memory, from where bulk copies take them (rows of 2 KB single, where the stores are many: 151
// against 207 us at 96^3 x 256; no difference for shorter rows and double).  Rows that are not 16-byte
// multiples (odd single-precision counts) are copied with the 8 bytes before or after them, up to 16-byte
// boundaries; only their own states are stored.  The terms are summed in nl_apply_kernel's order.  Bound by
// HBM: 2 S elements per hit point; 120^3 x 64 FP64 328 -> 163 us, 32^3 x 16 FP64 23 -> 8.6 us against a
// thread per state and batches of 8 points.
constexpr int NLA_NS = 2;     // stages
constexpr int NLA_KMAX = 32;  // largest batch (one producer lane per row)

template <typename R, int J, bool BS, int VM>
__global__ void __launch_bounds__(NLA_NT + 32, sizeof(R) == 4 ? 6 : 3) nl_apply_bulk_kernel(NlApply<R> a, long long nrec,
                                                                                         int KB, int ts, int *err) {
  using T = C2<R>;
  using namespace ptx;
  extern __shared__ __align__(128) unsigned char smem[];
  const int S = a.S;
  const uint32_t row_bytes = uint32_t(S) * uint32_t(sizeof(T));
  const uint32_t slot = (row_bytes + 15) & ~15u;                         // bytes copied per row
  unsigned char *rows = smem;                                            // [NS][KB][slot]
  T *coefs = reinterpret_cast<T *>(rows + size_t(NLA_NS) * KB * slot);   // [NS][KB][4]
  int4 *recs = reinterpret_cast<int4 *>(coefs + NLA_NS * KB * 4);        // [NS][KB]
  uint64_t *full = reinterpret_cast<uint64_t *>(recs + NLA_NS * KB);     // rows, coefficients and records loaded
  uint64_t *done = full + NLA_NS;                                        // rows computed
  volatile int *abort_flag = reinterpret_cast<volatile int *>(done + NLA_NS);
  const long long nbatch = (nrec + KB - 1) / KB;
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int st = 0; st < NLA_NS; st++) {
      mbar_init(&full[st], 2);
      mbar_init(&done[st], NLA_NT);
    }
    mbar_init_fence();
  }
  __syncthreads();
  grid_wait();
  grid_release();
  auto wait_bar = [&](uint64_t *b, uint32_t parity) { return nla_wait(b, parity, abort_flag, err); };

  if (threadIdx.x >= NLA_NT) {
    // producer warp: lane q copies row q of a batch
    const int lane = threadIdx.x - NLA_NT;
    // the k-th batch's stage is computed: with BS its rows are copied out
    auto retire = [&](int k, long long b) -> bool {
      const int st = k % NLA_NS;
      if (!__all_sync(0xffffffffu, wait_bar(&done[st], uint32_t(k / NLA_NS) & 1u))) return false;
      if constexpr (BS) {
        const int nb = int(min((long long)KB, nrec - b * KB));
        if (lane < nb)
          bulk_store(a.out + (long long)recs[st * KB + lane].x * S, rows + (size_t(st) * KB + lane) * slot, row_bytes);
        bulk_commit();
        bulk_wait_read0();  // the stage may be refilled once its rows are read out
        __syncwarp();
      }
      return true;
    };
    int k = 0;
    long long b = blockIdx.x;
    bool live = true;
    for (; b < nbatch; b += gridDim.x, k++) {
      const int st = k % NLA_NS;
      const long long k0 = b * KB;
      const int nb = int(min((long long)KB, nrec - k0));
      int4 rec = make_int4(0, 0, 0, 0);
      if (lane < nb) rec = a.hrec[k0 + lane];
      if (k >= NLA_NS && !(live = retire(k - NLA_NS, b - (long long)NLA_NS * gridDim.x))) break;
      if (lane < nb) recs[st * KB + lane] = rec;
      if (lane == 0) mbar_expect_tx(&full[st], uint32_t(nb) * slot);
      __syncwarp();
      if (lane < nb) {
        const uintptr_t src = reinterpret_cast<uintptr_t>(a.out + (long long)rec.x * S) & ~uintptr_t(15);
        bulk_load(rows + (size_t(st) * KB + lane) * slot, reinterpret_cast<const void *>(src), slot, &full[st]);
        // the first hit's coefficients by plain loads (bulk copies of 32 bytes: 180 us against 151)
        const int4 *hc = reinterpret_cast<const int4 *>(a.hcoef + (long long)rec.y * 4);
        int4 v[4 * sizeof(T) / 16];
#pragma unroll
        for (int w = 0; w < int(4 * sizeof(T) / 16); w++) v[w] = __ldg(hc + w);
#pragma unroll
        for (int w = 0; w < int(4 * sizeof(T) / 16); w++) reinterpret_cast<int4 *>(coefs + (st * KB + lane) * 4)[w] = v[w];
      }
      __threadfence_block();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[st]);  // the barrier's second arrival: records and coefficients are there
    }
    if constexpr (BS) {
      for (int i = k - NLA_NS < 0 ? 0 : k - NLA_NS; live && i < k; i++)
        live = retire(i, blockIdx.x + (long long)i * gridDim.x);
      bulk_wait0();
    }
    // after an abort the compute threads may leave early: wait (bounded) for every issued load to land
    // before the CTA's shared memory is released (on the normal path these phases are already complete)
    for (int i = k - NLA_NS < 0 ? 0 : k - NLA_NS; i < k; i++)
      mbar_wait_bounded(&full[i % NLA_NS], uint32_t(i / NLA_NS) & 1u, 2000000000ull);
    return;
  }

  const int TS = 1 << ts, G = NLA_NT >> ts;
  const int t = threadIdx.x & (TS - 1), g = threadIdx.x >> ts;
  T pd[J][4];
  int pprev = -1, i = 0;
  for (long long b = blockIdx.x; b < nbatch; b += gridDim.x, i++) {
    const int st = i % NLA_NS;
    if (!wait_bar(&full[st], uint32_t(i / NLA_NS) & 1u)) break;
    const int nb = int(min((long long)KB, nrec - b * KB));
    for (int q = g; q < nb; q += G) {
      const int4 rec = recs[st * KB + q];
      const long long pt = rec.x;
      const int h0 = rec.y, nh = rec.z, p0 = rec.w;
      if (p0 != pprev) {
#pragma unroll
        for (int j = 0; j < J; j++) {
          const int s = t + j * TS;
          if (s < S) {
#pragma unroll
            for (int l = 0; l < 4; l++) pd[j][l] = a.projD[((long long)p0 * 4 + l) * S + s];
          }
        }
        pprev = p0;
      }
      T hc[4];
#pragma unroll
      for (int l = 0; l < 4; l++) hc[l] = coefs[(st * KB + q) * 4 + l];
      T *o = a.out + pt * S;
      T *rw = reinterpret_cast<T *>(rows + (size_t(st) * KB + q) * slot + (reinterpret_cast<uintptr_t>(o) & 15));
#pragma unroll
      for (int j = 0; j < J; j++) {
        const int s = t + j * TS;
        if (s < S) (BS ? rw : o)[s] = nl_value<R, VM>(a, pt, s, h0, nh, rw[s], hc, pd[j]);
      }
    }
    fence_proxy_async();
    mbar_arrive(&done[st]);  // the producer refills the stage
  }
}

template <typename R>
void launch_nl_apply(Ctx &ctx, const Hamiltonian &h, const C2<R> *projD, int S, C2<R> *out, bool scaled, C2<R> scale,
                     const R *V, int nspin, int spin, R vshift) {
  const Projectors &P = h.proj;
  if (P.nhitpts == 0) return;
  NlApply<R> a;
  if constexpr (sizeof(R) == 8) a.hcoef = P.d_hcoef;
  else a.hcoef = P.d_hcoef32;
  a.hrec = P.d_hrec;
  a.hitp = P.d_hitp;
  a.projD = projD;
  a.out = out;
  a.S = S;
  a.scaled = scaled;
  a.scale = scale;
  a.V = V;
  a.nspin = nspin;
  a.spin = spin;
  a.vshift = vshift;
  // with the local potential: 1, or 2 when the forward pass that multiplies the other points computes in double
  const int vm = V == nullptr ? 0 : (sizeof(R) == 4 && (ctx.mixed_compute == 1 || ctx.mixed_compute == 2) ? 2 : 1);
  constexpr int VW = sizeof(R) == 4 ? 2 : 1;  // double sets have no second form
  // bulk form: up to 4 states per compute thread; rows of 16-byte multiples, or sets whose last row's copy
  // ends inside them
  const size_t row_bytes = size_t(S) * sizeof(C2<R>), slot = (row_bytes + 15) & ~size_t(15);
  const bool whole = row_bytes % 16 == 0 || (size_t(h.basis->npoints) * S) % 2 == 0;
  // (rows below 256 bytes leave the bulk form to option 1: 24^3 x 9 single 3.4 us against 2.9, 64^3 x 8 FP64 16 against 13)
  if (ctx.nl_bulk >= 0 && (ctx.nl_bulk > 0 || row_bytes >= 256) && whole && S <= 4 * NLA_NT && reinterpret_cast<uintptr_t>(out) % 16 == 0) {
    // 8 points per batch, 16 for rows of at most 1 KB when there are many (measured at 120^3 x 64 FP64, 440 k
    // points: 186 us with 8, 162 with 16, 164 with 32; 40^3 x 50 single, 14 k points: 6.5, -, 8.5)
    int KB = slot <= 1024 && P.nhitpts / 16 >= 32LL * ctx.device_sms ? 16 : 8;
    if (KB > int(49152 / slot)) KB = int(49152 / slot);
    if (KB < 1) KB = 1;
    if (ctx.nl_apply_points > 0) KB = ctx.nl_apply_points;
    const size_t smem = size_t(NLA_NS) * KB * (slot + 4 * sizeof(C2<R>) + sizeof(int4)) + 2 * NLA_NS * sizeof(uint64_t) + 16;
    if (smem <= size_t(ctx.max_smem_optin)) {
      const bool bs = row_bytes % 16 == 0 && row_bytes >= 1024;
      using Kern = void (*)(NlApply<R>, long long, int, int, int *);
      static const Kern kerns[18] = {
          nl_apply_bulk_kernel<R, 1, false, 0>,  nl_apply_bulk_kernel<R, 2, false, 0>,  nl_apply_bulk_kernel<R, 4, false, 0>,
          nl_apply_bulk_kernel<R, 1, true, 0>,   nl_apply_bulk_kernel<R, 2, true, 0>,   nl_apply_bulk_kernel<R, 4, true, 0>,
          nl_apply_bulk_kernel<R, 1, false, 1>,  nl_apply_bulk_kernel<R, 2, false, 1>,  nl_apply_bulk_kernel<R, 4, false, 1>,
          nl_apply_bulk_kernel<R, 1, true, 1>,   nl_apply_bulk_kernel<R, 2, true, 1>,   nl_apply_bulk_kernel<R, 4, true, 1>,
          nl_apply_bulk_kernel<R, 1, false, VW>, nl_apply_bulk_kernel<R, 2, false, VW>, nl_apply_bulk_kernel<R, 4, false, VW>,
          nl_apply_bulk_kernel<R, 1, true, VW>,  nl_apply_bulk_kernel<R, 2, true, VW>,  nl_apply_bulk_kernel<R, 4, true, VW>};
      // states per thread 1, 2 or 4; rows copied out or stored; the local potential
      const int ki = (S <= NLA_NT ? 0 : (S <= 2 * NLA_NT ? 1 : 2)) + (bs ? 3 : 0) + 6 * vm;
      const Kern kern = kerns[ki];
      int ts = 7;  // threads per row: a power of two from 8 to 128
      while (ts > 3 && (1 << (ts - 1)) >= S) ts--;
      ensure_smem_attr(reinterpret_cast<const void *>(kern), smem);
      // CTAs per SM for this kernel and shared-memory size, computed once under a lock
      static std::mutex mtx;
      static size_t occ_smem[18] = {};
      static int occ_per_sm[18] = {};
      int per_sm;
      {
        std::lock_guard<std::mutex> lock(mtx);
        if (occ_smem[ki] != smem) {
          INQB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_per_sm[ki], kern, NLA_NT + 32, smem));
          occ_smem[ki] = smem;
        }
        per_sm = occ_per_sm[ki];
      }
      const long long nbatch = (P.nhitpts + KB - 1) / KB;
      long long grid = (long long)(per_sm < 1 ? 1 : per_sm) * ctx.num_sms;
      if (grid > nbatch) grid = nbatch;
      pdl_launch(true, kern, dim3(unsigned(grid)), NLA_NT + 32, smem, ctx.stream, a, P.nhitpts, KB, ts, ctx.d_err);
      ctx.launches++;
      return;
    }
  }
  int sl = 5;
  while (sl > 2 && (1 << (sl - 1)) >= S) sl--;
  constexpr int U = 16 / int(sizeof(R));  // states per lane: 4 single, 2 double; 1 when a warp holds them all
  const int chunk = S <= 32 ? 1 << sl : U << sl;
  const int nchunks = (S + chunk - 1) / chunk;
  const long long nitems = P.nhitpts * nchunks;
  long long blocks = ((nitems << sl) + 127) / 128;
  if (blocks > 148LL * 48) blocks = 148LL * 48;
  using Kern = void (*)(NlApply<R>, long long, int, int);
  static const Kern few[3] = {nl_apply_kernel<R, 1, 0>, nl_apply_kernel<R, 1, 1>, nl_apply_kernel<R, 1, VW>};
  static const Kern many[3] = {nl_apply_kernel<R, U, 0>, nl_apply_kernel<R, U, 1>, nl_apply_kernel<R, U, VW>};
  const Kern kern = S <= 32 ? few[vm] : many[vm];
  pdl_launch(true, kern, dim3(unsigned(blocks)), 128, 0, ctx.stream, a, nitems, nchunks, sl);
  ctx.launches++;
}

// ------------------------------------------------------------------ bounded-wait self-test
// One thread waits on an mbarrier phase that nothing completes; the wait is bounded by `limit_ns` of
// %globaltimer, after which the context's error flag is raised exactly as by an expired wait of the
// FFT ring, the tensor-core overlap or the bulk-copy nonlocal kernels.
__global__ void wait_timeout_kernel(int *err, long long limit_ns) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    ptx::mbar_init(&bar, 1);
    ptx::mbar_init_fence();
  }
  __syncthreads();
  if (threadIdx.x == 0 && !ptx::mbar_wait_bounded(&bar, 0, uint64_t(limit_ns))) atomicExch(err, 1);
}

void launch_wait_timeout(Ctx &ctx, long long limit_ns) {
  wait_timeout_kernel<<<1, 32, 0, ctx.stream>>>(ctx.d_err, limit_ns);
  LAUNCHED(ctx);
}

// ------------------------------------------------------------------ elementwise
template <typename R> __global__ void fill_kernel(C2<R> *p, long long n, R re, R im) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    p[i] = mk<C2<R>>(re, im);
}
template <typename R> void launch_fill(Ctx &ctx, C2<R> *p, long long n, double re, double im) {
  fill_kernel<R><<<grid_for(n, 256), 256, 0, ctx.stream>>>(p, n, R(re), R(im));
  LAUNCHED(ctx);
}

template <typename R> __global__ void axpy_kernel(C2<R> *y, const C2<R> *x, long long n, R re, R im) {
  const C2<R> c = mk<C2<R>>(re, im);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = cadd(y[i], cmul(c, x[i]));
}
template <typename R> void launch_axpy(Ctx &ctx, C2<R> *y, const C2<R> *x, long long n, double re, double im) {
  axpy_kernel<R><<<grid_for(n, 256), 256, 0, ctx.stream>>>(y, x, n, R(re), R(im));
  LAUNCHED(ctx);
}

// y[pt][s] += scale * coef[s] * x[pt][s]   (operations::shift with a per-state factor, shift.hpp:19-31)
template <typename R>
__global__ void shift_vec_kernel(C2<R> *y, const C2<R> *x, int S, long long n, const double *coef, double scale) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const R c = R(scale * coef[i % S]);
    y[i] = cadd(y[i], cscale(x[i], c));
  }
}
template <typename R>
void launch_shift_vec(Ctx &ctx, C2<R> *y, const C2<R> *x, int S, long long npoints, const double *coef_dev,
                      double scale) {
  shift_vec_kernel<R><<<grid_for(npoints * S, 256), 256, 0, ctx.stream>>>(y, x, S, npoints * S, coef_dev, scale);
  LAUNCHED(ctx);
}

struct Metric {
  int n[3];
  double rlat[3][3];
  double lat[3][3];
};

__device__ __forceinline__ int symi(int i, int n) { return i >= (n + 1) / 2 ? i - n : i; }

__device__ __forceinline__ double lapl_at(const Metric &m, long long pt, double factor, const double *gc, double k2) {
  const int iz = int(pt % m.n[2]);
  const int iy = int((pt / m.n[2]) % m.n[1]);
  const int ix = int(pt / ((long long)m.n[2] * m.n[1]));
  const double tp = 6.283185307179586476925286766559;
  double G0 = tp * symi(ix, m.n[0]), G1 = tp * symi(iy, m.n[1]), G2 = tp * symi(iz, m.n[2]);
  double c0 = (m.rlat[0][0] * G0 + m.rlat[1][0] * G1) + m.rlat[2][0] * G2;
  double c1 = (m.rlat[0][1] * G0 + m.rlat[1][1] * G1) + m.rlat[2][1] * G2;
  double c2 = (m.rlat[0][2] * G0 + m.rlat[1][2] * G1) + m.rlat[2][2] * G2;
  double g2 = c0 * c0 + c1 * c1 + c2 * c2;
  return factor * (-g2 + (gc[0] * G0 + gc[1] * G1 + gc[2] * G2) + k2);
}

static Metric metric_of(const Basis &b) {
  Metric m;
  for (int i = 0; i < 3; i++) {
    m.n[i] = b.n[i];
    for (int j = 0; j < 3; j++) {
      m.rlat[i][j] = b.rlat[i][j];
      m.lat[i][j] = b.lat[i][j];
    }
  }
  return m;
}

struct Vec3 {
  double v[3];
};

template <typename R>
__global__ void laplacian_kernel(Metric m, const C2<R> *in, C2<R> *out, int S, long long n, double factor, Vec3 gc) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const R f = R(lapl_at(m, i / S, factor, gc.v, 0.0));
    out[i] = cscale(in[i], f);
  }
}
template <typename R>
void launch_laplacian(Ctx &ctx, const Basis &b, const C2<R> *in, C2<R> *out, int S, double factor, const double gc[3]) {
  Vec3 g{{gc[0], gc[1], gc[2]}};
  laplacian_kernel<R><<<grid_for(b.npoints * S, 256), 256, 0, ctx.stream>>>(metric_of(b), in, out, S, b.npoints * S,
                                                                            factor, g);
  LAUNCHED(ctx);
}

// ------------------------------------------------------------------ overlap (complex GEMM, K = npoints)
// S[i][j] = dv * sum_p conj(a[p][i]) b[p][j].  64x64 output tile per CTA, split-K over point chunks,
// 256 threads with a 4x4 register tile each, two CTAs per SM (128 registers: 24.5 ms against 31.6 ms with
// 130 registers and one CTA per SM, 96^3 x 256 with itself); partial tiles summed in chunk order.
template <typename R>
__global__ void __launch_bounds__(256, 2) overlap_kernel(const C2<R> *__restrict__ a, int Sa, const C2<R> *__restrict__ b,
                                                      int Sb, long long npoints, long long chunk, int sym,
                                                      double2 *partial) {
  constexpr int TB = 64, KT = 16;
  __shared__ double2 As[KT][TB];
  __shared__ double2 Bs[KT][TB];
  // sym: blockIdx.x enumerates the tiles on and above the diagonal, column by column
  int bi = blockIdx.x, bj = blockIdx.y;
  if (sym) {
    bj = 0;
    while ((bj + 1) * (bj + 2) / 2 <= bi) bj++;
    bi -= bj * (bj + 1) / 2;
  }
  const int ti = bi * TB, tj = bj * TB;
  const long long p0 = blockIdx.z * chunk;
  const long long p1 = min(npoints, p0 + chunk);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  double2 acc[4][4];
#pragma unroll
  for (int u = 0; u < 4; u++)
#pragma unroll
    for (int v = 0; v < 4; v++) acc[u][v] = make_double2(0.0, 0.0);
  for (long long k0 = p0; k0 < p1; k0 += KT) {
    for (int e = threadIdx.x; e < KT * TB; e += 256) {
      const int kk = e / TB, c = e % TB;
      const long long p = k0 + kk;
      double2 va = make_double2(0.0, 0.0), vb = make_double2(0.0, 0.0);
      if (p < p1) {
        if (ti + c < Sa) {
          C2<R> x = a[p * Sa + ti + c];
          va = make_double2(double(x.x), double(x.y));
        }
        if (tj + c < Sb) {
          C2<R> y = b[p * Sb + tj + c];
          vb = make_double2(double(y.x), double(y.y));
        }
      }
      As[kk][c] = va;
      Bs[kk][c] = vb;
    }
    __syncthreads();
#pragma unroll 4
    for (int kk = 0; kk < KT; kk++) {
      double2 av[4], bv[4];
#pragma unroll
      for (int u = 0; u < 4; u++) av[u] = As[kk][ty + 16 * u];
#pragma unroll
      for (int v = 0; v < 4; v++) bv[v] = Bs[kk][tx + 16 * v];
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int v = 0; v < 4; v++) {
          acc[u][v].x += av[u].x * bv[v].x + av[u].y * bv[v].y;
          acc[u][v].y += av[u].x * bv[v].y - av[u].y * bv[v].x;
        }
    }
    __syncthreads();
  }
  const long long base = (long long)blockIdx.z * Sa * Sb;
#pragma unroll
  for (int u = 0; u < 4; u++)
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const int i = ti + ty + 16 * u, j = tj + tx + 16 * v;
      if (i < Sa && j < Sb) partial[base + (long long)i * Sb + j] = acc[u][v];
    }
}

// With sym (a set against itself, S x S) only tiles with i/64 <= j/64 were computed: an element below
// them is the conjugate of its mirror, since <a_j|a_i> = conj(<a_i|a_j>).
// The FP64 form of overlap_kernel with its operand tiles double-buffered in shared memory: the next
// 16 points of a and b are copied with cp.async while the current ones are multiplied, so the global
// latency no longer stalls the tile.  Same tiles, order and arithmetic: bitwise the same result.
__global__ void __launch_bounds__(256, 2) overlap64_kernel(const double2 *__restrict__ a, int Sa,
                                                        const double2 *__restrict__ b, int Sb, long long npoints,
                                                        long long chunk, int sym, double2 *partial) {
  constexpr int TB = 64, KT = 16;
  extern __shared__ __align__(16) double2 osm[];  // [2 buffers][a, b][KT][TB]
  int bi = blockIdx.x, bj = blockIdx.y;
  if (sym) {
    bj = 0;
    while ((bj + 1) * (bj + 2) / 2 <= bi) bj++;
    bi -= bj * (bj + 1) / 2;
  }
  const int ti = bi * TB, tj = bj * TB;
  const long long p0 = blockIdx.z * chunk;
  const long long p1 = min(npoints, p0 + chunk);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  auto tile = [&](int buf, int ab) { return osm + (size_t(buf) * 2 + ab) * KT * TB; };
  auto issue = [&](int buf, long long k0) {
    double2 *As = tile(buf, 0), *Bs = tile(buf, 1);
    for (int e = threadIdx.x; e < KT * TB; e += 256) {
      const int kk = e / TB, c = e % TB;
      const long long p = k0 + kk;
      const bool va = p < p1 && ti + c < Sa, vb = p < p1 && tj + c < Sb;
      ptx::cp_async16(As + e, va ? a + p * Sa + ti + c : a, va ? 16u : 0u);
      ptx::cp_async16(Bs + e, vb ? b + p * Sb + tj + c : b, vb ? 16u : 0u);
    }
    ptx::cp_async_commit();
  };
  double2 acc[4][4];
#pragma unroll
  for (int u = 0; u < 4; u++)
#pragma unroll
    for (int v = 0; v < 4; v++) acc[u][v] = make_double2(0.0, 0.0);
  if (p0 < p1) issue(0, p0);
  int cur = 0;
  for (long long k0 = p0; k0 < p1; k0 += KT, cur ^= 1) {
    if (k0 + KT < p1) {
      issue(cur ^ 1, k0 + KT);  // the other buffer was released by the barrier closing the last step
      ptx::cp_async_wait<1>();
    } else {
      ptx::cp_async_wait<0>();
    }
    __syncthreads();
    const double2 *As = tile(cur, 0), *Bs = tile(cur, 1);
#pragma unroll 4
    for (int kk = 0; kk < KT; kk++) {
      double2 av[4], bv[4];
#pragma unroll
      for (int u = 0; u < 4; u++) av[u] = As[kk * TB + ty + 16 * u];
#pragma unroll
      for (int v = 0; v < 4; v++) bv[v] = Bs[kk * TB + tx + 16 * v];
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int v = 0; v < 4; v++) {
          acc[u][v].x += av[u].x * bv[v].x + av[u].y * bv[v].y;
          acc[u][v].y += av[u].x * bv[v].y - av[u].y * bv[v].x;
        }
    }
    __syncthreads();
  }
  const long long base = (long long)blockIdx.z * Sa * Sb;
#pragma unroll
  for (int u = 0; u < 4; u++)
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const int i = ti + ty + 16 * u, j = tj + tx + 16 * v;
      if (i < Sa && j < Sb) partial[base + (long long)i * Sb + j] = acc[u][v];
    }
}

// The same 64 x 64 tiles of a^H b on the FP64 tensor-core path: mma.sync m8n8k4 (DMMA), four per pair
// of complex operand fragments (re.re + im.im into the real part, re.im - im.re into the imaginary).
// 128 threads: each warp owns a 32 x 32 block of the tile, 4 x 4 fragments of 8 x 8, and steps through
// the point chunk four points at a time; operand tiles double-buffered by cp.async as above, rows padded
// to 66 complex numbers so that the fragment loads of a quarter-warp hit distinct banks.
__device__ __forceinline__ void dmma_8x8x4(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

__global__ void __launch_bounds__(128) overlap64_mma_kernel(const double2 *__restrict__ a, int Sa,
                                                            const double2 *__restrict__ b, int Sb, long long npoints,
                                                            long long chunk, int sym, double2 *partial) {
  constexpr int TB = 64, KT = 16, LD = TB + 2;
  extern __shared__ __align__(16) double2 osm[];  // [2 buffers][a, b][KT][LD]
  int bi = blockIdx.x, bj = blockIdx.y;
  if (sym) {
    bj = 0;
    while ((bj + 1) * (bj + 2) / 2 <= bi) bj++;
    bi -= bj * (bj + 1) / 2;
  }
  const int ti = bi * TB, tj = bj * TB;
  const long long p0 = blockIdx.z * chunk;
  const long long p1 = min(npoints, p0 + chunk);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;  // the warp's block of the tile
  auto tile = [&](int buf, int ab) { return osm + (size_t(buf) * 2 + ab) * KT * LD; };
  auto issue = [&](int buf, long long k0) {
    double2 *As = tile(buf, 0), *Bs = tile(buf, 1);
    for (int e = threadIdx.x; e < KT * TB; e += 128) {
      const int kk = e / TB, c = e % TB;
      const long long p = k0 + kk;
      const bool va = p < p1 && ti + c < Sa, vb = p < p1 && tj + c < Sb;
      ptx::cp_async16(As + kk * LD + c, va ? a + p * Sa + ti + c : a, va ? 16u : 0u);
      ptx::cp_async16(Bs + kk * LD + c, vb ? b + p * Sb + tj + c : b, vb ? 16u : 0u);
    }
    ptx::cp_async_commit();
  };
  double cre[4][4][2], cim[4][4][2];
#pragma unroll
  for (int u = 0; u < 4; u++)
#pragma unroll
    for (int v = 0; v < 4; v++) cre[u][v][0] = cre[u][v][1] = cim[u][v][0] = cim[u][v][1] = 0.0;
  if (p0 < p1) issue(0, p0);
  int cur = 0;
  // fragment coordinates: A (8 x 4, row-major) element (row lane / 4, col lane % 4), B (4 x 8,
  // col-major) element (row lane % 4, col lane / 4); here the row of A and the col of B are states and
  // the k index is the point
  const int fk = lane & 3, fs = lane >> 2;
  for (long long k0 = p0; k0 < p1; k0 += KT, cur ^= 1) {
    if (k0 + KT < p1) {
      issue(cur ^ 1, k0 + KT);
      ptx::cp_async_wait<1>();
    } else {
      ptx::cp_async_wait<0>();
    }
    __syncthreads();
    const double2 *As = tile(cur, 0), *Bs = tile(cur, 1);
#pragma unroll
    for (int ks = 0; ks < KT; ks += 4) {
      double2 af[4], bf[4];
#pragma unroll
      for (int u = 0; u < 4; u++) af[u] = As[(ks + fk) * LD + wm + 8 * u + fs];
#pragma unroll
      for (int v = 0; v < 4; v++) bf[v] = Bs[(ks + fk) * LD + wn + 8 * v + fs];
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int v = 0; v < 4; v++) {
          dmma_8x8x4(cre[u][v], af[u].x, bf[v].x);
          dmma_8x8x4(cre[u][v], af[u].y, bf[v].y);
          dmma_8x8x4(cim[u][v], af[u].x, bf[v].y);
          dmma_8x8x4(cim[u][v], -af[u].y, bf[v].x);
        }
    }
    __syncthreads();
  }
  // accumulator fragment: element (row lane / 4, col 2 (lane % 4) + {0, 1}) of each 8 x 8 block
  const long long base = (long long)blockIdx.z * Sa * Sb;
#pragma unroll
  for (int u = 0; u < 4; u++)
#pragma unroll
    for (int v = 0; v < 4; v++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int i = ti + wm + 8 * u + fs, j = tj + wn + 8 * v + 2 * fk + h;
        if (i < Sa && j < Sb) partial[base + (long long)i * Sb + j] = make_double2(cre[u][v][h], cim[u][v][h]);
      }
}

// out = scale * the chunks' tiles, summed in eight slices of the chunks (each in order, then the slices in
// order); block = 32 elements x 8 slices (one thread per element adding up to 256 chunks took 29 us)
__global__ void __launch_bounds__(256) sum_tiles_kernel(const double2 *partial, int nz, long long n, int S, int sym,
                                                        double scale, double2 *out) {
  __shared__ double2 red[8][32];
  const int c = threadIdx.x % 32, sl = threadIdx.x / 32;
  const long long e = blockIdx.x * 32LL + c;
  bool mirror = false;
  double re = 0.0, im = 0.0;
  if (e < n) {
    long long src = e;
    if (sym) {
      const int i = int(e / S), j = int(e % S);
      if (i / 64 > j / 64) {
        src = (long long)j * S + i;
        mirror = true;
      }
    }
    const int per = (nz + 7) / 8, z1 = min(nz, (sl + 1) * per);
#pragma unroll 8
    for (int z = sl * per; z < z1; z++) {
      const double2 v = partial[z * n + src];
      re += v.x;
      im += v.y;
    }
  }
  red[sl][c] = make_double2(re, im);
  __syncthreads();
  if (sl == 0 && e < n) {
    for (int q = 1; q < 8; q++) {
      re += red[q][c].x;
      im += red[q][c].y;
    }
    out[e] = make_double2(scale * re, mirror ? -scale * im : scale * im);
  }
}

template <typename R>
void launch_overlap(Ctx &ctx, const C2<R> *a, int Sa, const C2<R> *b, int Sb, long long npoints, double dv,
                    double2 *out) {
  const int gi = (Sa + 63) / 64, gj = (Sb + 63) / 64;
  const int sym = (a == b && Sa == Sb) ? 1 : 0;
  const int tiles = sym ? gi * (gi + 1) / 2 : gi * gj;
  // CTAs in flight: two per SM of the 256-thread SIMT kernel, four of the 128-thread tensor-core one
  const int per_sm = (sizeof(R) == 8 && ctx.fp64_mma) ? 4 : 2;
  int nz = int((long long)per_sm * ctx.device_sms + tiles - 1) / tiles;  // independent of grid_sms
  if (nz < 1) nz = 1;
  if (nz > 256) nz = 256;
  long long chunk = (npoints + nz - 1) / nz;
  chunk = ((chunk + 15) / 16) * 16;
  nz = int((npoints + chunk - 1) / chunk);
  double2 *partial = static_cast<double2 *>(dev_alloc(ctx, sizeof(double2) * (size_t)nz * Sa * Sb));
  const dim3 grid = sym ? dim3(tiles, 1, nz) : dim3(gi, gj, nz);
  if constexpr (sizeof(R) == 8) {
    if (ctx.fp64_mma) {
      const size_t smem = 2 * 2 * 16 * 66 * sizeof(double2);
      ensure_smem_attr(reinterpret_cast<const void *>(overlap64_mma_kernel), smem);
      overlap64_mma_kernel<<<grid, 128, smem, ctx.stream>>>(a, Sa, b, Sb, npoints, chunk, sym, partial);
    } else {
      const size_t smem = 2 * 2 * 16 * 64 * sizeof(double2);
      ensure_smem_attr(reinterpret_cast<const void *>(overlap64_kernel), smem);
      overlap64_kernel<<<grid, 256, smem, ctx.stream>>>(a, Sa, b, Sb, npoints, chunk, sym, partial);
    }
  } else {
    overlap_kernel<R><<<grid, 256, 0, ctx.stream>>>(a, Sa, b, Sb, npoints, chunk, sym, partial);
  }
  LAUNCHED(ctx);
  const long long n = (long long)Sa * Sb;
  sum_tiles_kernel<<<unsigned((n + 31) / 32), 256, 0, ctx.stream>>>(partial, nz, n, Sb, sym, dv, out);
  LAUNCHED(ctx);
  dev_free(ctx, partial);
}

// ------------------------------------------------------------------ rotate: out[p][:] <- alpha in[p][:] R + beta out[p][:]
template <typename R>
__global__ void __launch_bounds__(256) rotate_kernel(const C2<R> *in, int Sin, C2<R> *out, int Sout, long long npoints,
                                                     const double2 *__restrict__ Rm, double2 alpha, double2 beta,
                                                     int scaled, int use_beta) {
  constexpr int ROWS = 8;
  extern __shared__ __align__(16) unsigned char sm[];
  double2 *rows = reinterpret_cast<double2 *>(sm);  // [ROWS][Sin]
  for (long long p0 = (long long)blockIdx.x * ROWS; p0 < npoints; p0 += (long long)gridDim.x * ROWS) {
    const int nr = int(min((long long)ROWS, npoints - p0));
    for (int e = threadIdx.x; e < ROWS * Sin; e += blockDim.x) {
      const int r = e / Sin, k = e % Sin;
      double2 v = make_double2(0.0, 0.0);
      if (r < nr) {
        C2<R> x = in[(p0 + r) * Sin + k];
        v = make_double2(double(x.x), double(x.y));
      }
      rows[e] = v;
    }
    __syncthreads();  // in place (in == out): every row is staged before any is overwritten
    for (int j = threadIdx.x; j < Sout; j += blockDim.x) {
      double2 acc[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; r++) acc[r] = make_double2(0.0, 0.0);
      for (int k = 0; k < Sin; k++) {
        const double2 rk = Rm[(long long)k * Sout + j];
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
          const double2 x = rows[r * Sin + k];
          acc[r].x += x.x * rk.x - x.y * rk.y;
          acc[r].y += x.x * rk.y + x.y * rk.x;
        }
      }
#pragma unroll
      for (int r = 0; r < ROWS; r++) {  // constant trip count: acc stays in registers
        if (r >= nr) break;
        double2 v = acc[r];
        if (scaled) v = make_double2(alpha.x * v.x - alpha.y * v.y, alpha.x * v.y + alpha.y * v.x);
        C2<R> *o = out + (p0 + r) * Sout + j;
        if (use_beta) {
          const double2 y = make_double2(double(o->x), double(o->y));
          v.x += beta.x * y.x - beta.y * y.y;
          v.y += beta.x * y.y + beta.y * y.x;
        }
        *o = mk<C2<R>>(R(v.x), R(v.y));
      }
    }
    __syncthreads();
  }
}

// Tiled form of the rotation for distinct in and out: CTA = 64 points x 64 output states, 4 x 4 per
// thread, the states k in steps of 16 with both operand tiles (rows of in, rows of Rm) double-buffered
// in shared memory by cp.async.  Each CTA reads Rm's 64 columns once for 64 points (the row form reads
// all of Rm for every 8 points: 116 GB of cache traffic at 96^3 x 256).  Rows of in must be 16-byte
// multiples (an even state count in single precision).
template <typename R>
__global__ void __launch_bounds__(256, 2) rotate_tiled_kernel(const C2<R> *__restrict__ in, int Sin,
                                                           C2<R> *__restrict__ out, int Sout, long long npoints,
                                                           const double2 *__restrict__ Rm, double2 alpha,
                                                           double2 beta, int scaled, int use_beta) {
  using T = C2<R>;
  constexpr int TP = 64, TJ = 64, KT = 16;
  constexpr int EPC = 16 / int(sizeof(T));  // elements of in per 16-byte copy
  extern __shared__ __align__(16) unsigned char rsm[];
  T *Abuf = reinterpret_cast<T *>(rsm);                                   // [2][TP][KT]
  double2 *Bbuf = reinterpret_cast<double2 *>(Abuf + 2 * TP * KT);        // [2][KT][TJ]
  // blockIdx.x enumerates (point tile, output tile) with the output tiles fastest, so the CTAs that
  // read one tile of points run together
  const int njt = (Sout + TJ - 1) / TJ;
  const int j0 = int(blockIdx.x % njt) * TJ;
  const long long p0 = (long long)(blockIdx.x / njt) * TP;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  auto issue = [&](int buf, int k0) {
    T *As = Abuf + buf * TP * KT;
    double2 *Bs = Bbuf + buf * KT * TJ;
    for (int e = threadIdx.x; e < TP * KT / EPC; e += 256) {
      const int r = e / (KT / EPC), kk = (e % (KT / EPC)) * EPC;
      const long long p = p0 + r;
      const bool v = p < npoints && k0 + kk < Sin;
      ptx::cp_async16(As + r * KT + kk, v ? in + p * Sin + k0 + kk : in, v ? 16u : 0u);
    }
    for (int e = threadIdx.x; e < KT * TJ; e += 256) {
      const int kk = e / TJ, c = e % TJ;
      const bool v = k0 + kk < Sin && j0 + c < Sout;
      ptx::cp_async16(Bs + e, v ? Rm + (long long)(k0 + kk) * Sout + j0 + c : Rm, v ? 16u : 0u);
    }
    ptx::cp_async_commit();
  };
  double2 acc[4][4];
#pragma unroll
  for (int u = 0; u < 4; u++)
#pragma unroll
    for (int v = 0; v < 4; v++) acc[u][v] = make_double2(0.0, 0.0);
  issue(0, 0);
  int cur = 0;
  for (int k0 = 0; k0 < Sin; k0 += KT, cur ^= 1) {
    if (k0 + KT < Sin) {
      issue(cur ^ 1, k0 + KT);  // the other buffer was released by the barrier closing the last step
      ptx::cp_async_wait<1>();
    } else {
      ptx::cp_async_wait<0>();
    }
    __syncthreads();
    const T *As = Abuf + cur * TP * KT;
    const double2 *Bs = Bbuf + cur * KT * TJ;
#pragma unroll 4
    for (int kk = 0; kk < KT; kk++) {
      double2 av[4], bv[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const T x = As[(ty + 16 * u) * KT + kk];
        av[u] = make_double2(double(x.x), double(x.y));
      }
#pragma unroll
      for (int v = 0; v < 4; v++) bv[v] = Bs[kk * TJ + tx + 16 * v];
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int v = 0; v < 4; v++) {
          acc[u][v].x += av[u].x * bv[v].x - av[u].y * bv[v].y;
          acc[u][v].y += av[u].x * bv[v].y + av[u].y * bv[v].x;
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < 4; u++)
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const long long p = p0 + ty + 16 * u;
      const int j = j0 + tx + 16 * v;
      if (p < npoints && j < Sout) {
        double2 w = acc[u][v];
        if (scaled) w = make_double2(alpha.x * w.x - alpha.y * w.y, alpha.x * w.y + alpha.y * w.x);
        T *o = out + p * Sout + j;
        if (use_beta) {
          const double2 y = make_double2(double(o->x), double(o->y));
          w.x += beta.x * y.x - beta.y * y.y;
          w.y += beta.x * y.y + beta.y * y.x;
        }
        *o = mk<T>(R(w.x), R(w.y));
      }
    }
}

// The tiled rotation on the FP64 tensor-core path (mma.sync m8n8k4, four per pair of complex fragments:
// re.re - im.im into the real part, re.im + im.re into the imaginary): 64 points x 64 output states per
// CTA of 128 threads, each warp a 32 x 32 block of 8 x 8 fragments; operand tiles double-buffered by
// cp.async, rows padded (20 elements of in, 66 of R) so that the fragment loads hit distinct banks.
// One output tile of 64 points from p0 and 64 states from j0.  UPPER: Rm is upper triangular and Sin == Sout, so
// the tile needs the input states up to its own last one only.
template <typename R, bool UPPER>
__device__ __forceinline__ void rotate_tile(const C2<R> *in, int Sin, C2<R> *out, int Sout, long long npoints,
                                            const double2 *__restrict__ Rm, double2 alpha, double2 beta, int scaled,
                                            int use_beta, long long p0, int j0) {
  using T = C2<R>;
  constexpr int TP = 64, TJ = 64, KT = 16, LDA = 20, LDB = TJ + 2;
  constexpr int EPC = 16 / int(sizeof(T));  // elements of in per 16-byte copy
  extern __shared__ __align__(16) unsigned char rsm[];
  T *Abuf = reinterpret_cast<T *>(rsm);                                   // [2][TP][LDA]
  double2 *Bbuf = reinterpret_cast<double2 *>(Abuf + 2 * TP * LDA);       // [2][KT][LDB]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  const int fk = lane & 3, fs = lane >> 2;
  // rows of 16-byte multiples (the full form is only launched for them); else 8-byte copies
  const bool whole = (size_t(Sin) * sizeof(T)) % 16 == 0;
  const int kend = UPPER && j0 + TJ < Sin ? j0 + TJ : Sin;
  auto issue = [&](int buf, int k0) {
    T *As = Abuf + buf * TP * LDA;
    double2 *Bs = Bbuf + buf * KT * LDB;
    if (!UPPER || sizeof(T) == 16 || whole) {
      for (int e = threadIdx.x; e < TP * KT / EPC; e += 128) {
        const int r = e / (KT / EPC), kk = (e % (KT / EPC)) * EPC;
        const long long p = p0 + r;
        const bool v = p < npoints && k0 + kk < Sin;
        ptx::cp_async16(As + r * LDA + kk, v ? in + p * Sin + k0 + kk : in, v ? 16u : 0u);
      }
    } else {
      for (int e = threadIdx.x; e < TP * KT; e += 128) {
        const int r = e / KT, kk = e % KT;
        const long long p = p0 + r;
        if (p < npoints && k0 + kk < Sin) ptx::cp_async8(As + r * LDA + kk, in + p * Sin + k0 + kk);
        else As[r * LDA + kk] = mk<T>(R(0), R(0));
      }
    }
    for (int e = threadIdx.x; e < KT * TJ; e += 128) {
      const int kk = e / TJ, c = e % TJ;
      const bool v = k0 + kk < Sin && j0 + c < Sout;
      ptx::cp_async16(Bs + kk * LDB + c, v ? Rm + (long long)(k0 + kk) * Sout + j0 + c : Rm, v ? 16u : 0u);
    }
    ptx::cp_async_commit();
  };
  double cre[4][4][2], cim[4][4][2];
#pragma unroll
  for (int u = 0; u < 4; u++)
#pragma unroll
    for (int v = 0; v < 4; v++) cre[u][v][0] = cre[u][v][1] = cim[u][v][0] = cim[u][v][1] = 0.0;
  issue(0, 0);
  int cur = 0;
  for (int k0 = 0; k0 < kend; k0 += KT, cur ^= 1) {
    if (k0 + KT < kend) {
      issue(cur ^ 1, k0 + KT);
      ptx::cp_async_wait<1>();
    } else {
      ptx::cp_async_wait<0>();
    }
    __syncthreads();
    const T *As = Abuf + cur * TP * LDA;
    const double2 *Bs = Bbuf + cur * KT * LDB;
    if (!UPPER || k0 < j0 + wn + 32) {  // the warp's 32 columns end above row k0
#pragma unroll
    for (int ks = 0; ks < KT; ks += 4) {
      double2 af[4], bf[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const T x = As[(wm + 8 * u + fs) * LDA + ks + fk];  // A (8 x 4, row-major): (point, input state)
        af[u] = make_double2(double(x.x), double(x.y));
      }
#pragma unroll
      for (int v = 0; v < 4; v++) bf[v] = Bs[(ks + fk) * LDB + wn + 8 * v + fs];  // B (4 x 8): (input, output)
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int v = 0; v < 4; v++) {
          dmma_8x8x4(cre[u][v], af[u].x, bf[v].x);
          dmma_8x8x4(cre[u][v], -af[u].y, bf[v].y);
          dmma_8x8x4(cim[u][v], af[u].x, bf[v].y);
          dmma_8x8x4(cim[u][v], af[u].y, bf[v].x);
        }
    }
    }
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < 4; u++)
#pragma unroll
    for (int v = 0; v < 4; v++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const long long p = p0 + wm + 8 * u + fs;
        const int j = j0 + wn + 8 * v + 2 * fk + h;
        if (p < npoints && j < Sout) {
          double2 w = make_double2(cre[u][v][h], cim[u][v][h]);
          if (scaled) w = make_double2(alpha.x * w.x - alpha.y * w.y, alpha.x * w.y + alpha.y * w.x);
          T *o = out + p * Sout + j;
          if (use_beta) {
            const double2 y = make_double2(double(o->x), double(o->y));
            w.x += beta.x * y.x - beta.y * y.y;
            w.y += beta.x * y.y + beta.y * y.x;
          }
          *o = mk<T>(R(w.x), R(w.y));
        }
      }
}

// A CTA per tile.  The tile is a function of its own for this kernel's sake: inside the loop over tiles that the
// triangular form needs, the same code took 3 % longer (64^3 x 128 FP64 1633 against 1680 us, 40^3 x 300 1874 against 1932).
template <typename R>
__global__ void __launch_bounds__(128) rotate_mma_kernel(const C2<R> *__restrict__ in, int Sin, C2<R> *__restrict__ out,
                                                         int Sout, long long npoints, const double2 *__restrict__ Rm,
                                                         double2 alpha, double2 beta, int scaled, int use_beta) {
  const int njt = (Sout + 63) / 64;
  rotate_tile<R, false>(in, Sin, out, Sout, npoints, Rm, alpha, beta, scaled, use_beta, (long long)(blockIdx.x / njt) * 64,
                        int(blockIdx.x % njt) * 64);
}

// phi <- phi X, X upper triangular, in place: a CTA takes all output tiles of its 64 points, from the last to the
// first.  A tile skips the zeros below its columns (5/8 of the products are left at 256 states) and overwrites states
// that no later tile reads, so no scratch block and copy back are needed.  *skip != 0 (when given) leaves the set as it is.
template <typename R>
__global__ void __launch_bounds__(128) rotate_upper_kernel(C2<R> *phi, int S, long long npoints,
                                                           const double2 *__restrict__ X, const int *skip) {
  if (skip && *skip) return;
  for (int jt = (S + 63) / 64 - 1; jt >= 0; jt--)
    rotate_tile<R, true>(phi, S, phi, S, npoints, X, make_double2(1.0, 0.0), make_double2(0.0, 0.0), 0, 0,
                         (long long)blockIdx.x * 64, jt * 64);
}

// out <- alpha (in Rm) + beta out, Rm [Sin][Sout]; in == out (Sin == Sout) rotates in place
template <typename R>
void launch_rotate_to(Ctx &ctx, const C2<R> *in, int Sin, C2<R> *out, int Sout, long long npoints, const double2 *Rdev,
                      double2 alpha, double2 beta) {
  const int scaled = !(alpha.x == 1.0 && alpha.y == 0.0);
  const int use_beta = !(beta.x == 0.0 && beta.y == 0.0);
  const bool aligned = (size_t(Sin) * sizeof(C2<R>)) % 16 == 0 && reinterpret_cast<uintptr_t>(in) % 16 == 0 &&
                       reinterpret_cast<uintptr_t>(Rdev) % 16 == 0;
  if (aligned) {
    // tiled kernel, out of place; in place, chunks of 32768 points go through a scratch block and are
    // copied back (the kernel's CTAs for one tile of points read all of its states)
    const size_t tsmem = 2 * 64 * 16 * sizeof(C2<R>) + 2 * 16 * 64 * sizeof(double2);
    const size_t msmem = 2 * 64 * 20 * sizeof(C2<R>) + 2 * 16 * 66 * sizeof(double2);
    if (ctx.fp64_mma) ensure_smem_attr(reinterpret_cast<const void *>(rotate_mma_kernel<R>), msmem);
    else ensure_smem_attr(reinterpret_cast<const void *>(rotate_tiled_kernel<R>), tsmem);
    auto launch = [&](const C2<R> *src, C2<R> *dst, long long n) {
      const long long nblk = (long long)((Sout + 63) / 64) * ((n + 63) / 64);
      INQB_REQUIRE(nblk < (1LL << 31), INQB_ERR_UNSUPPORTED, "set too large for the rotation grid");
      if (ctx.fp64_mma)
        rotate_mma_kernel<R><<<unsigned(nblk), 128, msmem, ctx.stream>>>(src, Sin, dst, Sout, n, Rdev, alpha, beta,
                                                                         scaled, use_beta);
      else
        rotate_tiled_kernel<R><<<unsigned(nblk), 256, tsmem, ctx.stream>>>(src, Sin, dst, Sout, n, Rdev, alpha, beta,
                                                                          scaled, use_beta);
      LAUNCHED(ctx);
    };
    if (in != out) {
      launch(in, out, npoints);
      return;
    }
    INQB_REQUIRE(Sin == Sout && !use_beta, INQB_ERR_ARG, "an in-place rotation is square and has no beta term");
    constexpr long long CH = 32768;
    const long long ch = npoints < CH ? npoints : CH;
    C2<R> *scratch = static_cast<C2<R> *>(dev_alloc(ctx, sizeof(C2<R>) * size_t(ch) * Sout));
    for (long long c0 = 0; c0 < npoints; c0 += CH) {
      const long long n = npoints - c0 < CH ? npoints - c0 : CH;
      launch(in + c0 * Sin, scratch, n);
      INQB_CUDA(cudaMemcpyAsync(out + c0 * Sout, scratch, sizeof(C2<R>) * size_t(n) * Sout, cudaMemcpyDeviceToDevice,
                                ctx.stream));
    }
    dev_free(ctx, scratch);
    return;
  }
  const size_t smem = sizeof(double2) * 8 * Sin;
  INQB_REQUIRE(smem <= ctx.max_smem_optin, INQB_ERR_UNSUPPORTED, "too many states for rotate");
  ensure_smem_attr(reinterpret_cast<const void *>(rotate_kernel<R>), smem);
  rotate_kernel<R><<<grid_for(npoints, 8, 148LL * 16), 256, smem, ctx.stream>>>(in, Sin, out, Sout, npoints, Rdev, alpha,
                                                                              beta, scaled, use_beta);
  LAUNCHED(ctx);
}

// phi <- phi X in place with X upper triangular, unless skip_dev is given and *skip_dev is set
template <typename R>
void launch_rotate_upper(Ctx &ctx, C2<R> *phi, int S, long long npoints, const double2 *X, const int *skip_dev) {
  const size_t smem = 2 * 64 * 20 * sizeof(C2<R>) + 2 * 16 * 66 * sizeof(double2);
  ensure_smem_attr(reinterpret_cast<const void *>(rotate_upper_kernel<R>), smem);
  const long long nblk = (npoints + 63) / 64;
  INQB_REQUIRE(nblk < (1LL << 31), INQB_ERR_UNSUPPORTED, "set too large for the rotation grid");
  rotate_upper_kernel<R><<<unsigned(nblk), 128, smem, ctx.stream>>>(phi, S, npoints, X, skip_dev);
  LAUNCHED(ctx);
}

template <typename R> void launch_rotate(Ctx &ctx, C2<R> *phi, int S, long long npoints, const double2 *Rdev) {
  launch_rotate_to<R>(ctx, phi, S, phi, S, npoints, Rdev, make_double2(1.0, 0.0), make_double2(0.0, 0.0));
}

// ------------------------------------------------------------------ density n[p] (+)= sum_s occ_s |phi[p][s]|^2
// One group of SL lanes per point (a warp, or as many lanes as the states below 32), lanes stride over the states,
// fixed shuffle tree (density.hpp:24-36)
template <typename R, int SL>
__global__ void density_kernel(const C2<R> *__restrict__ phi, int S, long long npoints, const double *__restrict__ occ,
                               double *dens, int accumulate) {
  const int lane = threadIdx.x % SL;
  const long long group = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / SL;
  const long long ngroups = ((long long)gridDim.x * blockDim.x) / SL;
  // every lane of a warp runs the same number of rounds (the shuffles name the whole warp)
  for (long long p0 = 0; p0 < npoints; p0 += ngroups) {
    const long long p = p0 + group;
    double acc = 0.0;
    if (p < npoints) {
      for (int s = lane; s < S; s += SL) {
        C2<R> x = phi[p * S + s];
        acc += occ[s] * (double(x.x) * double(x.x) + double(x.y) * double(x.y));
      }
    }
#pragma unroll
    for (int o = SL / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0 && p < npoints) dens[p] = accumulate ? dens[p] + acc : acc;
  }
}
template <typename R>
void launch_density(Ctx &ctx, const C2<R> *phi, int S, long long npoints, const double *occ_dev, double *dens,
                    int accumulate) {
  auto go = [&](auto kern, int sl) {
    kern<<<grid_for(npoints * sl, 256), 256, 0, ctx.stream>>>(phi, S, npoints, occ_dev, dens, accumulate);
    LAUNCHED(ctx);
  };
  if (S > 16) go(density_kernel<R, 32>, 32);
  else if (S > 8) go(density_kernel<R, 16>, 16);
  else if (S > 4) go(density_kernel<R, 8>, 8);
  else go(density_kernel<R, 4>, 4);
}

// ------------------------------------------------------------------ kick: phi *= exp(i E_cov . r_contra)
template <typename R>
__global__ void kick_kernel(Metric m, C2<R> *phi, int S, long long npoints, Vec3 ecov) {
  const long long n = npoints * S;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const long long pt = e / S;
    const int iz = int(pt % m.n[2]);
    const int iy = int((pt / m.n[2]) % m.n[1]);
    const int ix = int(pt / ((long long)m.n[2] * m.n[1]));
    // rvector: symmetric index times contravariant spacing 1/n (real_space.hpp:127-130)
    const double r0 = symi(ix, m.n[0]) * (1.0 / m.n[0]);
    const double r1 = symi(iy, m.n[1]) * (1.0 / m.n[1]);
    const double r2 = symi(iz, m.n[2]) * (1.0 / m.n[2]);
    const double arg = ecov.v[0] * r0 + ecov.v[1] * r1 + ecov.v[2] * r2;
    double sn, cs;
    sincos(arg, &sn, &cs);
    C2<R> x = phi[e];
    double re = double(x.x) * cs - double(x.y) * sn;
    double im = double(x.x) * sn + double(x.y) * cs;
    phi[e] = mk<C2<R>>(R(re), R(im));
  }
}
template <typename R> void launch_kick(Ctx &ctx, const Basis &b, C2<R> *phi, int S, const double ecov[3]) {
  Vec3 e{{ecov[0], ecov[1], ecov[2]}};
  kick_kernel<R><<<grid_for(b.npoints * S, 256), 256, 0, ctx.stream>>>(metric_of(b), phi, S, b.npoints, e);
  LAUNCHED(ctx);
}

// ------------------------------------------------------------------ sums over a density
constexpr int RED_BLOCKS = 592;  // block partials: 256 threads, four blocks per SM
// out[c] = scale * sum of partial[b * nc + c] over the blocks b, nc <= 3 values, in a fixed order: one block,
// each thread its strided share, then a tree (one thread adding all partials took 13 to 20 us)
__global__ void __launch_bounds__(256) block_sums_kernel(const double *partial, int nb, int nc, double scale, double *out) {
  __shared__ double red[256];
  for (int c = 0; c < nc; c++) {
    double acc = 0.0;
    for (int b = threadIdx.x; b < nb; b += 256) acc += partial[b * nc + c];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
      if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
      __syncthreads();
    }
    if (threadIdx.x == 0) out[c] = scale * red[0];
    __syncthreads();
  }
}

// sum |a - b| (integral_sum_absdiff)
__global__ void absdiff_kernel(const double *a, const double *b, long long n, double *partial) {
  __shared__ double red[256];
  const long long chunk = (n + gridDim.x - 1) / gridDim.x;
  const long long p0 = blockIdx.x * chunk, p1 = min(n, p0 + chunk);
  double acc = 0.0;
  for (long long i = p0 + threadIdx.x; i < p1; i += blockDim.x) acc += fabs(a[i] - b[i]);
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}
void launch_absdiff_sum(Ctx &ctx, const double *a, const double *b, long long n, double *out_dev) {
  double *partial = static_cast<double *>(dev_alloc(ctx, sizeof(double) * RED_BLOCKS));
  absdiff_kernel<<<RED_BLOCKS, 256, 0, ctx.stream>>>(a, b, n, partial);
  LAUNCHED(ctx);
  block_sums_kernel<<<1, 256, 0, ctx.stream>>>(partial, RED_BLOCKS, 1, 1.0, out_dev);
  LAUNCHED(ctx);
  dev_free(ctx, partial);
}

// dipole = dV sum_r n(r) r (observables::dipole, dipole.hpp:24-60) of a device density: r from the
// symmetric grid index of each point (cell-centred coordinates), contravariant -> cartesian.  Block b
// sums a contiguous point range, threads strided, then a shared-memory tree; the partials are added in
// block order.
__global__ void dipole_kernel(const double *__restrict__ dens, int nx, int ny, int nz, long long n, Vec3 a0, Vec3 a1,
                              Vec3 a2, double *partial) {
  __shared__ double red[3][256];
  const long long chunk = (n + gridDim.x - 1) / gridDim.x;
  const long long p0 = blockIdx.x * chunk, p1 = min(n, p0 + chunk);
  double acc[3] = {0.0, 0.0, 0.0};
  for (long long p = p0 + threadIdx.x; p < p1; p += blockDim.x) {
    const int iz = int(p % nz), iy = int((p / nz) % ny), ix = int(p / ((long long)ny * nz));
    const double c0 = (ix >= (nx + 1) / 2 ? ix - nx : ix) * (1.0 / nx);
    const double c1 = (iy >= (ny + 1) / 2 ? iy - ny : iy) * (1.0 / ny);
    const double c2 = (iz >= (nz + 1) / 2 ? iz - nz : iz) * (1.0 / nz);
    const double d = dens[p];
#pragma unroll
    for (int j = 0; j < 3; j++) acc[j] += ((a0.v[j] * c0 + a1.v[j] * c1) + a2.v[j] * c2) * d;
  }
  for (int j = 0; j < 3; j++) red[j][threadIdx.x] = acc[j];
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o)
      for (int j = 0; j < 3; j++) red[j][threadIdx.x] += red[j][threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x < 3) partial[blockIdx.x * 3 + threadIdx.x] = red[threadIdx.x][0];
}
void launch_dipole(Ctx &ctx, const Basis &b, const double *dens, double *out3_dev) {
  double *partial = static_cast<double *>(dev_alloc(ctx, sizeof(double) * 3 * RED_BLOCKS));
  Vec3 a[3];
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) a[i].v[j] = b.lat[i][j];
  dipole_kernel<<<RED_BLOCKS, 256, 0, ctx.stream>>>(dens, b.n[0], b.n[1], b.n[2], b.npoints, a[0], a[1], a[2], partial);
  LAUNCHED(ctx);
  block_sums_kernel<<<1, 256, 0, ctx.stream>>>(partial, RED_BLOCKS, 3, b.volume / double(b.npoints), out3_dev);
  LAUNCHED(ctx);
  dev_free(ctx, partial);
}

// ------------------------------------------------------------------ eigensolver pieces
// y[pt][s] += scale * (coef[s] * x[pt][s]) with complex per-state factors (operations::shift, shift.hpp:19-31)
template <typename R>
__global__ void shift_cvec_kernel(C2<R> *__restrict__ y, const C2<R> *__restrict__ x, int S, long long n,
                                  const double2 *__restrict__ coef, double scale) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double2 c = coef[i % S];
    const C2<R> xv = x[i];
    const double tr = c.x * double(xv.x) - c.y * double(xv.y), ti = c.x * double(xv.y) + c.y * double(xv.x);
    y[i] = mk<C2<R>>(R(double(y[i].x) + scale * tr), R(double(y[i].y) + scale * ti));
  }
}
template <typename R>
void launch_shift_cvec(Ctx &ctx, C2<R> *y, const C2<R> *x, int S, long long npoints, const double2 *coef_dev,
                       double scale) {
  shift_cvec_kernel<R><<<grid_for(npoints * S, 256), 256, 0, ctx.stream>>>(y, x, S, npoints * S, coef_dev, scale);
  LAUNCHED(ctx);
}

// ------------------------------------------------------------------ restart files
// out[k][pt] = (complex<double>) in[pt][s0 + k], k < ns: states [s0, s0 + ns) as contiguous rows
template <typename R>
__global__ void extract_states_kernel(const C2<R> *__restrict__ in, int S, long long np, int s0, int ns,
                                      double2 *__restrict__ out) {
  const long long n = np * ns;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long k = i / np, pt = i % np;
    const C2<R> v = in[pt * S + s0 + k];
    out[i] = make_double2(double(v.x), double(v.y));
  }
}
// the reverse: out[pt][s0 + k] = in[k][pt]
template <typename R>
__global__ void insert_states_kernel(const double2 *__restrict__ in, int S, long long np, int s0, int ns,
                                     C2<R> *__restrict__ out) {
  const long long n = np * ns;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long k = i / np, pt = i % np;
    const double2 v = in[i];
    out[pt * S + s0 + k] = mk<C2<R>>(R(v.x), R(v.y));
  }
}
template <typename R>
void launch_extract_states(Ctx &ctx, const C2<R> *in, int S, long long np, int s0, int ns, double2 *out) {
  extract_states_kernel<R><<<grid_for(np * ns, 256), 256, 0, ctx.stream>>>(in, S, np, s0, ns, out);
  LAUNCHED(ctx);
}
template <typename R>
void launch_insert_states(Ctx &ctx, const double2 *in, int S, long long np, int s0, int ns, C2<R> *out) {
  insert_states_kernel<R><<<grid_for(np * ns, 256), 256, 0, ctx.stream>>>(in, S, np, s0, ns, out);
  LAUNCHED(ctx);
}

// ------------------------------------------------------------------ interacting potential
// (solvers/poisson.hpp, hamiltonian/xc_term.hpp, hamiltonian/self_consistency.hpp)

__global__ void real_to_complex_kernel(const double *__restrict__ in, double2 *__restrict__ out, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = make_double2(in[i], 0.0);
}

// poisson_apply_kernel with poisson_kernel_3d (poisson.hpp:29-35, 72-87): times scal * kern,
// scal = -4 pi / N, kern = -1/|G|^2 (cartesian), 0 for |G|^2 < 1e-6
__global__ void poisson_factor_kernel(Metric m, double2 *__restrict__ f, long long n, double scal) {
  const double zero[3] = {0.0, 0.0, 0.0};
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double g2 = lapl_at(m, i, -1.0, zero, 0.0);
    const double k = g2 < 1e-6 ? 0.0 : -1.0 / g2;
    const double c = scal * k;
    f[i] = make_double2(f[i].x * c, f[i].y * c);
  }
}

// Slater exchange and Perdew-Zunger 1981 correlation of an unpolarised density (the published
// parametrisation, libxc's XC_LDA_X and XC_LDA_C_PZ): energy per particle and potential.
__device__ __forceinline__ void lda_xc(double n, double &eps, double &v) {
  if (!(n > 1e-15)) {
    eps = 0.0;
    v = 0.0;
    return;
  }
  const double pi = 3.14159265358979323846;
  const double cx = -0.75 * cbrt(3.0 / pi);
  const double ex = cx * cbrt(n);
  const double rs = cbrt(3.0 / (4.0 * pi * n));
  double ec, vc;
  if (rs >= 1.0) {
    const double sq = sqrt(rs);
    const double den = 1.0 + 1.0529 * sq + 0.3334 * rs;
    ec = -0.1423 / den;
    vc = ec * (1.0 + 7.0 / 6.0 * 1.0529 * sq + 4.0 / 3.0 * 0.3334 * rs) / den;
  } else {
    const double lr = log(rs);
    ec = 0.0311 * lr - 0.048 + 0.0020 * rs * lr - 0.0116 * rs;
    vc = 0.0311 * lr + (-0.048 - 0.0311 / 3.0) + 2.0 / 3.0 * 0.0020 * rs * lr + (2.0 * -0.0116 - 0.0020) / 3.0 * rs;
  }
  eps = ex + ec;
  v = 4.0 / 3.0 * ex + vc;
}

// V = V_ion + Re V_H + V_xc (double and single copies) and the block sums, in a fixed order, of
// n V_ion, n V_H, n eps_xc, n v_xc
__global__ void ks_potential_kernel(const double *__restrict__ n, const double *__restrict__ vion,
                                    const double2 *__restrict__ vh, int xc, long long np, double *__restrict__ V,
                                    float *__restrict__ V32, double *__restrict__ partial) {
  __shared__ double red[4][256];
  const long long chunk = (np + gridDim.x - 1) / gridDim.x;
  const long long p0 = blockIdx.x * chunk, p1 = min(np, p0 + chunk);
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (long long i = p0 + threadIdx.x; i < p1; i += blockDim.x) {
    const double d = n[i];
    const double h = vh ? vh[i].x : 0.0;
    double eps = 0.0, vx = 0.0;
    if (xc) lda_xc(d, eps, vx);
    const double v = (vion[i] + h) + vx;
    V[i] = v;
    V32[i] = float(v);
    s[0] += d * vion[i];
    s[1] += d * h;
    s[2] += d * eps;
    s[3] += d * vx;
  }
  for (int k = 0; k < 4; k++) red[k][threadIdx.x] = s[k];
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o)
      for (int k = 0; k < 4; k++) red[k][threadIdx.x] += red[k][threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int k = 0; k < 4; k++) partial[blockIdx.x * 4 + k] = red[k][0];
}

void launch_real_to_complex(Ctx &ctx, const double *in, double2 *out, long long n) {
  real_to_complex_kernel<<<grid_for(n, 256), 256, 0, ctx.stream>>>(in, out, n);
  LAUNCHED(ctx);
}

void launch_poisson_factor(Ctx &ctx, const Basis &b, double2 *f) {
  poisson_factor_kernel<<<grid_for(b.npoints, 256), 256, 0, ctx.stream>>>(metric_of(b), f, b.npoints,
                                                                         -4.0 * 3.14159265358979323846 / double(b.npoints));
  LAUNCHED(ctx);
}

void launch_ks_potential(Ctx &ctx, const double *n, const double *vion, const double2 *vh, int xc, long long np,
                         double *V, float *V32, double *partial_dev) {
  ks_potential_kernel<<<KS_BLOCKS, 256, 0, ctx.stream>>>(n, vion, vh, xc, np, V, V32, partial_dev);
  LAUNCHED(ctx);
}

// ------------------------------------------------------------------ instantiations
// ------------------------------------------------------------------ Taylor terms combined

struct TaylorCoefs {
  double2 c1[8], c2[8];
};
struct TaylorTerms {
  const void *u[8];
};

// e1 = x + sum_n c1[n] u[n], e2 = x + sum_n c2[n] u[n], element-wise, terms added in order n = 0, 1, ...
// (the order in which exponential.hpp:56-69 adds them); complex products in double
// K: the number of terms when it is known (4, the propagator's order), so that an element's loads are in flight
// together instead of one after the other (72^3 x 128 single 503 -> 449 us, 40^3 x 33 double 50 -> 35 us);
// 0: nterms.  Bound by HBM, K + 3 transits.
template <typename R, int K>
__global__ void __launch_bounds__(256) taylor_combine_kernel(const C2<R> *__restrict__ x, TaylorTerms u, int nterms,
                                                             TaylorCoefs c, C2<R> *e1, C2<R> *e2, long long n) {
  using T = C2<R>;
  const int nt = K ? K : nterms;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const T xv = x[i];
    T tk[K ? K : 1];
    if constexpr (K > 0) {
#pragma unroll
      for (int k = 0; k < K; k++) tk[k] = static_cast<const T *>(u.u[k])[i];
    }
    double2 a1 = make_double2(double(xv.x), double(xv.y)), a2 = a1;
#pragma unroll
    for (int k = 0; k < nt; k++) {
      const T t = K ? tk[K ? k : 0] : static_cast<const T *>(u.u[k])[i];
      const double2 tv = make_double2(double(t.x), double(t.y));
      if (e1) a1 = cadd(a1, cmul(c.c1[k], tv));
      a2 = cadd(a2, cmul(c.c2[k], tv));
    }
    if (e1) e1[i] = mk<T>(R(a1.x), R(a1.y));
    e2[i] = mk<T>(R(a2.x), R(a2.y));
  }
}

template <typename R>
void launch_taylor_combine(Ctx &ctx, const C2<R> *x, const C2<R> *const *u, int nterms, const double2 *c1,
                           const double2 *c2, C2<R> *e1, C2<R> *e2, long long n) {
  INQB_REQUIRE(nterms >= 1 && nterms <= 8, INQB_ERR_UNSUPPORTED, "Taylor order must be 1..8");
  TaylorTerms t{};
  TaylorCoefs c{};
  for (int k = 0; k < nterms; k++) {
    t.u[k] = u[k];
    c.c1[k] = c1 ? c1[k] : make_double2(0.0, 0.0);
    c.c2[k] = c2[k];
  }
  long long blocks = (n + 255) / 256;
  if (blocks > 16LL * ctx.num_sms) blocks = 16LL * ctx.num_sms;
  if (nterms == 4) taylor_combine_kernel<R, 4><<<unsigned(blocks), 256, 0, ctx.stream>>>(x, t, nterms, c, e1, e2, n);
  else taylor_combine_kernel<R, 0><<<unsigned(blocks), 256, 0, ctx.stream>>>(x, t, nterms, c, e1, e2, n);
  LAUNCHED(ctx);
}

#define INST(R)                                                                                                   \
  template void launch_nl_project<R>(Ctx &, const Basis &, const Hamiltonian &, const C2<R> *, int, C2<R> *,       \
                                     C2<R> *);                                                                    \
  template void launch_nl_scatter<R>(Ctx &, const Basis &, const Hamiltonian &, const C2<R> *, int, C2<R> *);     \
  template void launch_nl_apply<R>(Ctx &, const Hamiltonian &, const C2<R> *, int, C2<R> *, bool, C2<R>, const R *, \
                                   int, int, R);                                                                  \
  template void launch_taylor_combine<R>(Ctx &, const C2<R> *, const C2<R> *const *, int, const double2 *,         \
                                         const double2 *, C2<R> *, C2<R> *, long long);                           \
  template void launch_fill<R>(Ctx &, C2<R> *, long long, double, double);                                         \
  template void launch_axpy<R>(Ctx &, C2<R> *, const C2<R> *, long long, double, double);                          \
  template void launch_shift_vec<R>(Ctx &, C2<R> *, const C2<R> *, int, long long, const double *, double);        \
  template void launch_shift_cvec<R>(Ctx &, C2<R> *, const C2<R> *, int, long long, const double2 *, double);      \
  template void launch_extract_states<R>(Ctx &, const C2<R> *, int, long long, int, int, double2 *);               \
  template void launch_insert_states<R>(Ctx &, const double2 *, int, long long, int, int, C2<R> *);                \
  template void launch_laplacian<R>(Ctx &, const Basis &, const C2<R> *, C2<R> *, int, double, const double *);    \
  template void launch_overlap<R>(Ctx &, const C2<R> *, int, const C2<R> *, int, long long, double, double2 *);   \
  template void launch_rotate<R>(Ctx &, C2<R> *, int, long long, const double2 *);                                 \
  template void launch_rotate_upper<R>(Ctx &, C2<R> *, int, long long, const double2 *, const int *);              \
  template void launch_rotate_to<R>(Ctx &, const C2<R> *, int, C2<R> *, int, long long, const double2 *, double2,     \
                                    double2);                                                                      \
  template void launch_density<R>(Ctx &, const C2<R> *, int, long long, const double *, double *, int);            \
  template void launch_kick<R>(Ctx &, const Basis &, C2<R> *, int, const double *);

INST(double)
INST(float)

}  // namespace inqb

namespace inqb {

// ------------------------------------------------------------------ synthetic orbitals
// SplitMix64 (Steele, Lea & Flood 2014) counter stream and the Box-Muller transform.
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long seed, unsigned long long counter) {
  unsigned long long z = seed + (counter + 1ULL) * 0x9E3779B97F4A7C15ULL;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}
__device__ __forceinline__ double u01(unsigned long long x) { return double(x >> 11) * (1.0 / 9007199254740992.0); }

template <typename R>
__global__ void randomize_gsphere_kernel(Metric m, C2<R> *phi, int S, long long npoints, unsigned long long seed,
                                         double ecut) {
  const long long n = npoints * S;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const long long pt = e / S;
    const int s = int(e % S);
    const double half_g2 = -0.5 * lapl_at(m, pt, 1.0, Vec3{{0, 0, 0}}.v, 0.0);
    C2<R> v = mk<C2<R>>(R(0), R(0));
    if (half_g2 < ecut) {
      const unsigned long long c = (unsigned long long)s * (unsigned long long)npoints + (unsigned long long)pt;
      const double a = u01(splitmix64(seed, 2 * c)), b = u01(splitmix64(seed, 2 * c + 1));
      const double r = sqrt(-2.0 * log(1.0 - a));
      double sn, cs;
      sincospi(2.0 * b, &sn, &cs);
      v = mk<C2<R>>(R(r * cs), R(r * sn));
    }
    phi[e] = v;
  }
}

template <typename R>
void launch_randomize_gsphere(Ctx &ctx, const Basis &b, C2<R> *phi, int S, unsigned long long seed, double ecut) {
  randomize_gsphere_kernel<R><<<grid_for(b.npoints * S, 256), 256, 0, ctx.stream>>>(metric_of(b), phi, S, b.npoints,
                                                                                     seed, ecut);
  LAUNCHED(ctx);
}

template <typename RI, typename RO> __global__ void convert_kernel(const C2<RI> *in, C2<RO> *out, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    C2<RI> x = in[i];
    out[i] = mk<C2<RO>>(RO(x.x), RO(x.y));
  }
}

void launch_convert(Ctx &ctx, const void *in, int in_prec, void *out, int out_prec, long long n) {
  if (in_prec == INQB_F64 && out_prec == INQB_F32)
    convert_kernel<double, float><<<grid_for(n, 256), 256, 0, ctx.stream>>>(static_cast<const double2 *>(in),
                                                                            static_cast<float2 *>(out), n);
  else if (in_prec == INQB_F32 && out_prec == INQB_F64)
    convert_kernel<float, double><<<grid_for(n, 256), 256, 0, ctx.stream>>>(static_cast<const float2 *>(in),
                                                                            static_cast<double2 *>(out), n);
  else
    throw Error(INQB_ERR_ARG, "conversion needs two different precisions");
  LAUNCHED(ctx);
}

template void launch_randomize_gsphere<double>(Ctx &, const Basis &, double2 *, int, unsigned long long, double);
template void launch_randomize_gsphere<float>(Ctx &, const Basis &, float2 *, int, unsigned long long, double);

}  // namespace inqb
