// Per-state sums over the points of orbital sets, and the steepest-descent step built from them.
//
// Every sum has a fixed order, so results are bitwise reproducible: block b takes a contiguous point range;
// its threads are G groups of 2^ts lanes over the states, group g sums the points g, g + G, ... of the range
// in U running sums (the points' loads are independent, U points of every operand in flight per thread); the
// running sums are added pairwise, the groups in order, and a second kernel adds the blocks' partials in 32
// slices, each in block order, and the slices in a fixed tree.
//
// Bound by HBM (each operand read once).  Sets with fewer than 256 states used to leave the other threads of
// a block idle, and one thread per state added all 592 partials (73 us at any size); measured at 50^3 x 64
// FP64: one complex sum 72 + 73 -> 51 + 10 us.  The steps of an eigensolver need several sums of the same
// sets, so a pass forms all of them (up to seven real sums) from one read.

#include "inqb_internal.h"

#include <type_traits>

namespace inqb {

#define LAUNCHED(ctx)                   \
  do {                                  \
    INQB_CUDA(cudaGetLastError());      \
    (ctx).launches++;                   \
  } while (0)

namespace {

constexpr int SUM_BLOCKS = 592;   // four 256-thread blocks per SM, resident at once
constexpr int SUM_THREADS = 256;
constexpr int FIN_S = 8, FIN_SLICES = 32;

struct GMetric {
  int n[3];
  double rlat[3][3];
};
GMetric gmetric_of(const Basis &b) {
  GMetric m;
  for (int i = 0; i < 3; i++) {
    m.n[i] = b.n[i];
    for (int j = 0; j < 3; j++) m.rlat[i][j] = b.rlat[i][j];
  }
  return m;
}
// factor * (-|G|^2 + gc.G + k2) of a Fourier-space point (fourier_space.hpp:77-125)
// I: the type of a point's index; grids of fewer than 2^31 points take the 32-bit form, whose divisions are the cheaper
// (kinetic sums of 96^3 x 128 FP64 469 against 617 us with a 64-bit index)
template <typename I>
__device__ __forceinline__ double lapl_of(const GMetric &m, I pt, double factor, const double *gc, double k2) {
  const int row = int(pt / m.n[2]), iz = int(pt - I(row) * m.n[2]), ix = row / m.n[1], iy = row - ix * m.n[1];
  auto sym = [](int i, int n) { return i >= (n + 1) / 2 ? i - n : i; };
  const double tp = 6.283185307179586476925286766559;
  const double G0 = tp * sym(ix, m.n[0]), G1 = tp * sym(iy, m.n[1]), G2 = tp * sym(iz, m.n[2]);
  const double c0 = (m.rlat[0][0] * G0 + m.rlat[1][0] * G1) + m.rlat[2][0] * G2;
  const double c1 = (m.rlat[0][1] * G0 + m.rlat[1][1] * G1) + m.rlat[2][1] * G2;
  const double c2 = (m.rlat[0][2] * G0 + m.rlat[1][2] * G1) + m.rlat[2][2] * G2;
  return factor * (-(c0 * c0 + c1 * c1 + c2 * c2) + (gc[0] * G0 + gc[1] * G1 + gc[2] * G2) + k2);
}

__device__ __forceinline__ double2 wide(double2 x) { return x; }
__device__ __forceinline__ double2 wide(float2 x) { return make_double2(double(x.x), double(x.y)); }
__device__ __forceinline__ double norm2(double2 x) { return x.x * x.x + x.y * x.y; }
__device__ __forceinline__ double2 dotc(double2 x, double2 y) {  // conj(x) y
  return make_double2(x.x * y.x + x.y * y.y, x.x * y.y - x.y * y.x);
}

// ---- what a pass sums: V values per state; state(s) reads the state's coefficients, term(p, s) adds a point

// <a|b>.  Eight points in flight in single precision, whose elements need twice as many loads for the same bytes (two
// sets of 96^3 x 256 single 917 -> 841 us; in double eight take 596 -> 845 at 96^3 x 128)
template <typename R> struct SumDot {
  static constexpr int V = 2, U = sizeof(R) == 4 ? 8 : 4;
  const C2<R> *a, *b;
  __device__ void state(int) {}
  __device__ void term(long long p, int s, int S, double (&v)[V]) const {
    const double2 d = dotc(wide(a[p * S + s]), wide(b[p * S + s]));
    v[0] += d.x;
    v[1] += d.y;
  }
};
// <a|a>: each element read once, eight points in flight (as <a|b> of a set with itself 96^3 x 256 single 785 -> 475 us,
// 64^3 x 600 FP64 739 -> 510; four in flight 755 and 617)
template <typename R> struct SumNorm {
  static constexpr int V = 1, U = 8;
  const C2<R> *a;
  __device__ void state(int) {}
  __device__ void term(long long p, int s, int S, double (&v)[V]) const { v[0] += norm2(wide(a[p * S + s])); }
};
// (|a|^2, Re <a|b>): the two sums of one eigenvalue
template <typename R> struct SumEigen {
  static constexpr int V = 2, U = 4;
  const C2<R> *a, *b;
  __device__ void state(int) {}
  __device__ void term(long long p, int s, int S, double (&v)[V]) const {
    const double2 x = wide(a[p * S + s]), y = wide(b[p * S + s]);
    v[0] += norm2(x);
    v[1] += x.x * y.x + x.y * y.y;
  }
};
// |b - e a|^2 with e = ne.y / ne.x: the residual norm of energy.hpp:86-89 without forming the residual
template <typename R> struct SumResidual {
  static constexpr int V = 1, U = 4;
  const C2<R> *a, *b;
  const double2 *ne;
  double e;
  __device__ void state(int s) { e = ne[s].y / ne[s].x; }
  __device__ void term(long long p, int s, int S, double (&v)[V]) const {
    const double2 x = wide(a[p * S + s]), y = wide(b[p * S + s]);
    v[0] += norm2(make_double2(y.x - e * x.x, y.y - e * x.y));
  }
};
// <a| lapl |a>
template <typename R, typename I> struct SumKinetic {
  static constexpr int V = 1, U = 4;
  const C2<R> *a;
  GMetric m;
  double factor, gc[3], k2;
  __device__ void state(int) {}
  __device__ void term(long long p, int s, int S, double (&v)[V]) const {
    v[0] += lapl_of<I>(m, I(p), factor, gc, k2) * norm2(wide(a[p * S + s]));
  }
};

// Steepest descent (steepest_descent.hpp:23-86), the five sweeps of one step; e = <hphi|phi> / <phi|phi>.
// The residual res = hphi - e phi, in the storage type as it would be stored
template <typename R> __device__ __forceinline__ C2<R> residual(C2<R> hphi, C2<R> phi, double2 e) {
  const double2 x = wide(phi), y = wide(hphi);
  return mk<C2<R>>(R(y.x - (e.x * x.x - e.y * x.y)), R(y.y - (e.x * x.y + e.y * x.x)));
}
// (Re, Im <hphi|phi>, <phi|phi>)
template <typename R> struct SumRayleigh {
  static constexpr int V = 3, U = 4;
  const C2<R> *phi, *hphi;
  __device__ void state(int) {}
  __device__ void term(long long p, int s, int S, double (&v)[V]) const {
    const double2 x = wide(phi[p * S + s]), d = dotc(wide(hphi[p * S + s]), x);
    v[0] += d.x;
    v[1] += d.y;
    v[2] += norm2(x);
  }
};
// (<res| -1/2 lapl |res>, <res|res>)
template <typename R, typename I> struct SumResidualKinetic {
  static constexpr int V = 2, U = 4;
  const C2<R> *phi, *hphi;
  const double2 *coef;
  GMetric m;
  double2 e;
  __device__ void state(int s) { e = coef[s]; }
  __device__ void term(long long p, int s, int S, double (&v)[V]) const {
    const double zero[3] = {0.0, 0.0, 0.0};
    const double n = norm2(wide(residual<R>(hphi[p * S + s], phi[p * S + s], e)));
    v[0] += lapl_of<I>(m, I(p), -0.5, zero, 0.0) * n;
    v[1] += n;
  }
};
// (<res|res>, <phi|res>, <res|hres>, <phi|hres>)
template <typename R> struct SumLine {
  static constexpr int V = 7, U = 2;
  const C2<R> *phi, *res, *hres;
  __device__ void state(int) {}
  __device__ void term(long long p, int s, int S, double (&v)[V]) const {
    const double2 f = wide(phi[p * S + s]), r = wide(res[p * S + s]), h = wide(hres[p * S + s]);
    const double2 d1 = dotc(f, r), d2 = dotc(r, h), d3 = dotc(f, h);
    v[0] += norm2(r);
    v[1] += d1.x;
    v[2] += d1.y;
    v[3] += d2.x;
    v[4] += d2.y;
    v[5] += d3.x;
    v[6] += d3.y;
  }
};
// phi += c res, hphi += c hres, and the next step's Rayleigh sums of the new sets
template <typename R> struct SumUpdate {
  static constexpr int V = 3, U = 2;
  C2<R> *phi, *hphi;
  const C2<R> *res, *hres;
  const double2 *coef;
  double2 c;
  __device__ void state(int s) { c = coef[s]; }
  __device__ void term(long long p, int s, int S, double (&v)[V]) const {
    const long long i = p * S + s;
    const double2 r = wide(res[i]), h = wide(hres[i]), f = wide(phi[i]), g = wide(hphi[i]);
    const C2<R> nf = mk<C2<R>>(R(f.x + (c.x * r.x - c.y * r.y)), R(f.y + (c.x * r.y + c.y * r.x)));
    const C2<R> ng = mk<C2<R>>(R(g.x + (c.x * h.x - c.y * h.y)), R(g.y + (c.x * h.y + c.y * h.x)));
    phi[i] = nf;
    hphi[i] = ng;
    const double2 x = wide(nf), d = dotc(wide(ng), x);
    v[0] += d.x;
    v[1] += d.y;
    v[2] += norm2(x);
  }
};

// partial[block][value][state]
template <typename F>
__global__ void __launch_bounds__(SUM_THREADS) state_sums_kernel(F f, int S, int ts, long long npoints,
                                                                 double *__restrict__ partial) {
  constexpr int V = F::V, U = F::U;
  __shared__ double red[V][SUM_THREADS];
  const int TS = 1 << ts, G = SUM_THREADS >> ts;
  const int lane = threadIdx.x & (TS - 1), g = threadIdx.x >> ts;
  const long long chunk = (npoints + gridDim.x - 1) / gridDim.x;
  const long long p0 = blockIdx.x * chunk, p1 = min(npoints, p0 + chunk);
  for (int s0 = 0; s0 < S; s0 += TS) {
    const int s = s0 + lane;
    double acc[U][V];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int k = 0; k < V; k++) acc[u][k] = 0.0;
    if (s < S) {
      f.state(s);
      long long p = p0 + g;
      for (; p + (U - 1) * G < p1; p += U * G) {
#pragma unroll
        for (int u = 0; u < U; u++) f.term(p + u * G, s, S, acc[u]);
      }
#pragma unroll
      for (int u = 0; u < U - 1; u++)
        if (p + u * G < p1) f.term(p + u * G, s, S, acc[u]);
#pragma unroll
      for (int w = U / 2; w >= 1; w /= 2)
#pragma unroll
        for (int u = 0; u < w; u++)
#pragma unroll
          for (int k = 0; k < V; k++) acc[u][k] += acc[u + w][k];
    }
    if (G > 1) {
#pragma unroll
      for (int k = 0; k < V; k++) red[k][threadIdx.x] = acc[0][k];
      __syncthreads();
      if (g == 0) {
#pragma unroll
        for (int k = 0; k < V; k++)
          for (int q = 1; q < G; q++) acc[0][k] += red[k][q * TS + lane];
      }
      __syncthreads();
    }
    if (g == 0 && s < S) {
#pragma unroll
      for (int k = 0; k < V; k++) partial[((long long)blockIdx.x * V + k) * S + s] = acc[0][k];
    }
  }
}

// ---- what is done with a state's sums

// out[s] = scale * (v0, v1)
struct PutPair {
  double2 *out;
  double scale;
  __device__ void operator()(int s, const double (&v)[2]) const { out[s] = make_double2(scale * v[0], scale * v[1]); }
};
struct PutReal2 {  // out[s] = (scale * v0, 0)
  double2 *out;
  double scale;
  __device__ void operator()(int s, const double (&v)[1]) const { out[s] = make_double2(scale * v[0], 0.0); }
};
struct PutReal {
  double *out;
  double scale;
  __device__ void operator()(int s, const double (&v)[1]) const { out[s] = scale * v[0]; }
};
// e = <hphi|phi> / <phi|phi>, and the two (with the volume element) for the line minimisation
struct PutRayleigh {
  double2 *coef;  // [S]
  double2 *ray;   // [2][S]: <hphi|phi>, (<phi|phi>, 0)
  int S;
  double dv;
  __device__ void operator()(int s, const double (&v)[3]) const {
    const double er = dv * v[0], ei = dv * v[1], n = dv * v[2];
    ray[s] = make_double2(er, ei);
    ray[S + s] = make_double2(n, 0.0);
    coef[s] = make_double2(er / n, ei / n);
  }
};
struct PutRatio {
  double *out;
  double dv;
  __device__ void operator()(int s, const double (&v)[2]) const { out[s] = (dv * v[0]) / (dv * v[1]); }
};
// the step length of the line minimisation (steepest_descent.hpp:60-76)
struct PutStep {
  double2 *coef;
  const double2 *ray;
  int S;
  double dv;
  __device__ void operator()(int s, const double (&v)[7]) const {
    const double2 ev = ray[s];
    const double nrm = ray[S + s].x;
    const double m0 = dv * v[0], m1r = dv * v[1], m1i = dv * v[2], m2r = dv * v[3], m2i = dv * v[4], m3r = dv * v[5];
    const double ca = m0 * m3r - (m2r * m1r - m2i * m1i);
    const double cb = nrm * m2r - ev.x * m0;
    const double cc = (ev.x * m1r - ev.y * m1i) - m3r * nrm;
    const double den = cb + sqrt(cb * cb - 4.0 * ca * cc);
    coef[s] = make_double2(fabs(den) < 1e-15 ? 0.0 : 2.0 * cc / den, 0.0);
  }
};

template <int V, typename P>
__global__ void __launch_bounds__(FIN_S *FIN_SLICES) state_finish_kernel(const double *__restrict__ partial, int nblk, int S,
                                                                        P put) {
  __shared__ double red[V][FIN_SLICES][FIN_S];
  const int c = threadIdx.x % FIN_S, sl = threadIdx.x / FIN_S, s = blockIdx.x * FIN_S + c;
  const int per = (nblk + FIN_SLICES - 1) / FIN_SLICES, b0 = sl * per, b1 = min(nblk, b0 + per);
  double v[V];
#pragma unroll
  for (int k = 0; k < V; k++) v[k] = 0.0;
  if (s < S) {
    for (int b = b0; b < b1; b += 4) {  // four blocks' values in flight
      double x[4][V];
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int k = 0; k < V; k++) x[u][k] = b + u < b1 ? partial[((long long)(b + u) * V + k) * S + s] : 0.0;
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int k = 0; k < V; k++) v[k] += x[u][k];
    }
  }
#pragma unroll
  for (int k = 0; k < V; k++) red[k][sl][c] = v[k];
  __syncthreads();
  for (int o = FIN_SLICES / 2; o > 0; o >>= 1) {
    if (sl < o) {
#pragma unroll
      for (int k = 0; k < V; k++) red[k][sl][c] += red[k][sl + o][c];
    }
    __syncthreads();
  }
  if (sl == 0 && s < S) {
#pragma unroll
    for (int k = 0; k < V; k++) v[k] = red[k][0][c];
    put(s, v);
  }
}

template <typename F, typename P>
void state_sums(Ctx &ctx, const F &f, int S, long long npoints, const P &put, double *partial) {
  int ts = 3;  // lanes per group: the power of two that holds the states, from 8 to the whole block
  while (ts < 8 && (1 << ts) < S) ts++;
  // enough points per block for every group to have a few
  const long long most = (npoints * (1LL << ts)) / (4LL * SUM_THREADS) + 1;
  const int blocks = int(most < SUM_BLOCKS ? most : SUM_BLOCKS);
  state_sums_kernel<F><<<blocks, SUM_THREADS, 0, ctx.stream>>>(f, S, ts, npoints, partial);
  LAUNCHED(ctx);
  state_finish_kernel<F::V, P><<<(S + FIN_S - 1) / FIN_S, FIN_S * FIN_SLICES, 0, ctx.stream>>>(partial, blocks, S, put);
  LAUNCHED(ctx);
}
double *sums_scratch(Ctx &ctx, int S, int values) {
  return static_cast<double *>(dev_alloc(ctx, sizeof(double) * SUM_BLOCKS * size_t(S) * values));
}

// res = K(1/2 |G|^2 / T_s) (hphi - e phi), the preconditioned residual (Teter, Payne, Allan; preconditioner.hpp:24-46)
template <typename R, typename I>
__global__ void precondition_kernel(GMetric m, const C2<R> *__restrict__ phi, const C2<R> *__restrict__ hphi,
                                    C2<R> *__restrict__ res, int S, long long npoints, const double2 *__restrict__ coef,
                                    const double *__restrict__ kin) {
  const double zero[3] = {0.0, 0.0, 0.0};
  const long long n = npoints * S;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long p = n < (1LL << 31) ? (long long)(uint32_t(i) / uint32_t(S)) : i / S;
    const int s = int(i - p * S);
    const double2 x = wide(residual<R>(hphi[i], phi[i], coef[s]));
    const double t = lapl_of<I>(m, I(p), -0.5, zero, 0.0) / kin[s];
    const double num = ((8.0 * t + 12.0) * t + 18.0) * t + 27.0;
    const double den = (((16.0 * t + 8.0) * t + 12.0) * t + 18.0) * t + 27.0;
    const double k = num / den;
    res[i] = mk<C2<R>>(R(x.x * k), R(x.y * k));
  }
}

}  // namespace

template <typename R>
void launch_overlap_diag(Ctx &ctx, const C2<R> *a, const C2<R> *b, int S, long long npoints, double dv, double2 *out) {
  double *partial = sums_scratch(ctx, S, 2);
  if (a == b) state_sums(ctx, SumNorm<R>{a}, S, npoints, PutReal2{out, dv}, partial);
  else state_sums(ctx, SumDot<R>{a, b}, S, npoints, PutPair{out, dv}, partial);
  dev_free(ctx, partial);
}

// Eigenvalues and residual norms of energy.hpp:80-89 in two passes over a and b = H a:
// ne[s] = dv (<a|a>, Re<a|b>); when res is given, res[s].x = dv sum_p |b - e_s a|^2 with e_s = ne[s].y / ne[s].x
template <typename R>
void launch_eigen_sums(Ctx &ctx, const C2<R> *a, const C2<R> *b, int S, long long npoints, double dv, double2 *ne,
                       double2 *res) {
  double *partial = sums_scratch(ctx, S, 2);
  state_sums(ctx, SumEigen<R>{a, b}, S, npoints, PutPair{ne, dv}, partial);
  if (res) state_sums(ctx, SumResidual<R>{a, b, ne, 0.0}, S, npoints, PutReal2{res, dv}, partial);
  dev_free(ctx, partial);
}

template <typename R>
void launch_kinetic_ev(Ctx &ctx, const Basis &b, const C2<R> *fphi, int S, double factor, const double gc[3], double k2,
                       double *out_dev) {
  double *partial = sums_scratch(ctx, S, 1);
  auto go = [&](auto index) {
    state_sums(ctx, SumKinetic<R, decltype(index)>{fphi, gmetric_of(b), factor, {gc[0], gc[1], gc[2]}, k2}, S, b.npoints,
               PutReal{out_dev, 1.0}, partial);
  };
  if (b.npoints < (1LL << 31)) go(int());
  else go(0LL);
  dev_free(ctx, partial);
}

// One pass each; `work` holds launch_sd_work_bytes(S) bytes: the block partials and the coefficients
size_t launch_sd_work_bytes(int S) { return sizeof(double) * size_t(S) * (size_t(SUM_BLOCKS) * 7 + 2 + 4 + 1); }
struct SdWork {
  double *partial;
  double2 *coef, *ray;
  double *kin;
  SdWork(void *work, int S) {
    partial = static_cast<double *>(work);
    coef = reinterpret_cast<double2 *>(partial + size_t(SUM_BLOCKS) * 7 * S);
    ray = coef + S;
    kin = reinterpret_cast<double *>(ray + 2 * S);
  }
};
template <typename R>
void launch_sd_rayleigh(Ctx &ctx, const C2<R> *phi, const C2<R> *hphi, int S, long long npoints, double dv, void *work) {
  SdWork w(work, S);
  state_sums(ctx, SumRayleigh<R>{phi, hphi}, S, npoints, PutRayleigh{w.coef, w.ray, S, dv}, w.partial);
}
template <typename R>
void launch_sd_residual(Ctx &ctx, const Basis &b, const C2<R> *phi, const C2<R> *hphi, C2<R> *res, int S, double dv,
                        void *work) {
  SdWork w(work, S);
  const GMetric m = gmetric_of(b);
  const long long n = b.npoints * S;
  long long blocks = (n + 255) / 256;
  if (blocks > 148LL * 64) blocks = 148LL * 64;
  auto go = [&](auto index) {
    using I = decltype(index);
    state_sums(ctx, SumResidualKinetic<R, I>{phi, hphi, w.coef, m, make_double2(0.0, 0.0)}, S, b.npoints,
               PutRatio{w.kin, dv}, w.partial);
    precondition_kernel<R, I><<<unsigned(blocks), 256, 0, ctx.stream>>>(m, phi, hphi, res, S, b.npoints, w.coef, w.kin);
    LAUNCHED(ctx);
  };
  if (b.npoints < (1LL << 31)) go(int());
  else go(0LL);
}
// phi += c res and, unless this was the last step, hphi += c hres with the next step's Rayleigh sums
template <typename R>
void launch_sd_update(Ctx &ctx, C2<R> *phi, C2<R> *hphi, const C2<R> *res, const C2<R> *hres, int S, long long npoints,
                      double dv, void *work, bool last) {
  SdWork w(work, S);
  state_sums(ctx, SumLine<R>{phi, res, hres}, S, npoints, PutStep{w.coef, w.ray, S, dv}, w.partial);
  if (last) launch_shift_cvec<R>(ctx, phi, res, S, npoints, w.coef, 1.0);
  else
    state_sums(ctx, SumUpdate<R>{phi, hphi, res, hres, w.coef, make_double2(0.0, 0.0)}, S, npoints,
               PutRayleigh{w.coef, w.ray, S, dv}, w.partial);
}

#define INQB_INST(R)                                                                                                  \
  template void launch_overlap_diag<R>(Ctx &, const C2<R> *, const C2<R> *, int, long long, double, double2 *);       \
  template void launch_eigen_sums<R>(Ctx &, const C2<R> *, const C2<R> *, int, long long, double, double2 *, double2 *); \
  template void launch_kinetic_ev<R>(Ctx &, const Basis &, const C2<R> *, int, double, const double *, double, double *); \
  template void launch_sd_rayleigh<R>(Ctx &, const C2<R> *, const C2<R> *, int, long long, double, void *);           \
  template void launch_sd_residual<R>(Ctx &, const Basis &, const C2<R> *, const C2<R> *, C2<R> *, int, double, void *); \
  template void launch_sd_update<R>(Ctx &, C2<R> *, C2<R> *, const C2<R> *, const C2<R> *, int, long long, double, void *, \
                                    bool);
INQB_INST(double)
INQB_INST(float)

}  // namespace inqb
