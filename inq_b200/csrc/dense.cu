// Dense Hermitian matrices of the subspace operations on the device: Cholesky factor and triangular inverse
// (orthogonalize), eigen-decomposition (subspace_diagonalization).  FP64 throughout.
//
// On the host these took longer than the kernels around them.  Measured: Cholesky and inverse of 128 states
// 0.9 -> 0.22 ms of the 3.6 ms orthogonalisation at 64^3; Jacobi rotations of 64 states 48 -> 3.0 ms of the
// 65 ms ground-state iteration at 50^3, of 256 states 31 ms (seconds on the host).

#include "inqb_internal.h"

#include <cooperative_groups.h>

namespace inqb {

#define LAUNCHED(ctx)                   \
  do {                                  \
    INQB_CUDA(cudaGetLastError());      \
    (ctx).launches++;                   \
  } while (0)

namespace {

// ------------------------------------------------------------------ Cholesky S = U^H U and X = U^-1
// (matrix/cholesky.hpp:28-89, invert_triangular.hpp:20-60).  Blocked, 32 x 32 tiles, rows of U from the top:
// launch k factors the diagonal tile k (every CTA for itself: a serial chain of 32 reciprocals that is
// shorter than a launch) and solves for one tile of U's row k per CTA, the next launch subtracts the row's
// products from the tiles below.  Then one CTA per tile column back-substitutes its column of X.
constexpr int CB = 32;            // tile
constexpr int CT = 256;           // threads: 8 rows of 32 columns at a time
constexpr int CLD = CB + 1;       // padded row of a tile in shared memory

// tile (ti, tj) of the n x n matrix, identity outside it
__device__ __forceinline__ void tile_load(double2 (*t)[CLD], const double2 *A, int n, int ti, int tj) {
  for (int e = threadIdx.x; e < CB * CB; e += CT) {
    const int r = e / CB, c = e % CB, i = ti * CB + r, j = tj * CB + c;
    t[r][c] = i < n && j < n ? A[(long long)i * n + j] : make_double2(i == j ? 1.0 : 0.0, 0.0);
  }
}
__device__ __forceinline__ double2 csubmul(double2 a, double2 x, double2 y) {  // a - x y
  return make_double2(a.x - (x.x * y.x - x.y * y.y), a.y - (x.x * y.y + x.y * y.x));
}
__device__ __forceinline__ double2 csubmulc(double2 a, double2 x, double2 y) {  // a - conj(x) y
  return make_double2(a.x - (x.x * y.x + x.y * y.y), a.y - (x.x * y.y - x.y * y.x));
}

// CTA j: the diagonal tile k of A factored, and tile (k, k + 1 + j) of U = U_kk^-H A.  CTA 0 writes the
// diagonal tile to D (A is read by the others meanwhile).  The elimination keeps its rows unscaled (row q times
// 1 / d_qq is subtracted), so the serial chain per row is one reciprocal and one barrier; the square roots of
// the pivots scale all rows at the end (with the scaling inside the chain a tile took 36 us).
// *before: an earlier row had a pivot that is not positive; *after: this one or an earlier one has.  Two flags,
// so that no launch writes what its other CTAs read; every CTA finds the same pivots, and CTA 0 writes.
__global__ void __launch_bounds__(CT) chol_row_kernel(double2 *A, double2 *D, int n, int k, const int *before, int *after) {
  __shared__ double2 d[CB][CLD], t[CB][CLD];
  const bool writer = blockIdx.x == 0 && threadIdx.x == 0;
  if (*before) {
    if (writer) *after = 1;
    return;
  }
  tile_load(d, A, n, k, k);
  const int tj = k + 1 + int(blockIdx.x);
  const bool panel = tj * CB < n;
  if (panel) tile_load(t, A, n, k, tj);
  __syncthreads();
  for (int q = 0; q < CB; q++) {
    const double p = d[q][q].x;  // the tile is Hermitian: the pivot's imaginary part is rounding
    if (!(p > 0.0)) {  // every thread read the same pivot
      if (writer) *after = 1;
      return;
    }
    const double inv = 1.0 / p;
    for (int e = threadIdx.x; e < CB * CB; e += CT) {
      const int r = e / CB, c = e % CB;
      if (r <= q) continue;
      const double2 m = make_double2(d[q][r].x * inv, d[q][r].y * inv);
      if (c >= r) d[r][c] = csubmulc(d[r][c], m, d[q][c]);
      if (panel) t[r][c] = csubmulc(t[r][c], m, t[q][c]);
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < CB * CB; e += CT) {
    const int r = e / CB, c = e % CB, i = k * CB + r, j = tj * CB + c;
    const double u = sqrt(d[r][r].x);
    if (blockIdx.x == 0) {
      double2 v = make_double2(0.0, 0.0);
      if (c == r) v.x = u;
      else if (c > r) v = make_double2(d[r][c].x / u, d[r][c].y / u);
      D[e] = v;
    }
    if (panel && i < n && j < n) A[(long long)i * n + j] = make_double2(t[r][c].x / u, t[r][c].y / u);
  }
}

// tile (i, j), k < i <= j: A_ij -= U_ki^H U_kj
__global__ void __launch_bounds__(CT) chol_update_kernel(double2 *A, int n, int k, const int *bad) {
  __shared__ double2 x[CB][CLD], y[CB][CLD];
  if (*bad) return;
  int bj = 0, bi = blockIdx.x;
  while ((bj + 1) * (bj + 2) / 2 <= bi) bj++;
  bi -= bj * (bj + 1) / 2;
  const int ti = k + 1 + bi, tj = k + 1 + bj;
  tile_load(x, A, n, k, ti);
  tile_load(y, A, n, k, tj);
  __syncthreads();
  for (int e = threadIdx.x; e < CB * CB; e += CT) {
    const int r = e / CB, c = e % CB, i = ti * CB + r, j = tj * CB + c;
    if (i >= n || j >= n) continue;
    double2 v = A[(long long)i * n + j];
#pragma unroll 8
    for (int q = 0; q < CB; q++) v = csubmulc(v, x[q][r], y[q][c]);
    A[(long long)i * n + j] = v;
  }
}

// CTA j: tile column j of X = U^-1 from the bottom; X_jj = U_jj^-1, X_ij = -U_ii^-1 sum_k U_ik X_kj.
// D holds the diagonal tiles of U, A the others; everything below the diagonal of X is zero.
__global__ void __launch_bounds__(CT) tri_inverse_kernel(const double2 *A, const double2 *D, double2 *X, int n,
                                                         const int *bad) {
  __shared__ double2 u[CB][CLD], x[CB][CLD];  // x: the tiles of X multiplied, then the tile being solved
  if (*bad) return;
  const int tj = blockIdx.x, nt = (n + CB - 1) / CB;
  for (int ti = nt - 1; ti >= 0; ti--) {
    if (ti > tj) {
      for (int e = threadIdx.x; e < CB * CB; e += CT) {
        const int i = ti * CB + e / CB, j = tj * CB + e % CB;
        if (i < n && j < n) X[(long long)i * n + j] = make_double2(0.0, 0.0);
      }
      continue;
    }
    double2 v[CB * CB / CT];
    for (int w = 0; w < CB * CB / CT; w++) {
      const int e = threadIdx.x + w * CT;
      v[w] = make_double2(ti == tj && e / CB == e % CB ? 1.0 : 0.0, 0.0);
    }
    for (int tk = ti + 1; tk <= tj; tk++) {
      __syncthreads();
      tile_load(u, A, n, ti, tk);
      tile_load(x, X, n, tk, tj);
      __syncthreads();
#pragma unroll
      for (int w = 0; w < CB * CB / CT; w++) {
        const int e = threadIdx.x + w * CT, r = e / CB, c = e % CB;
#pragma unroll 8
        for (int q = 0; q < CB; q++) v[w] = csubmul(v[w], u[r][q], x[q][c]);
      }
    }
    __syncthreads();
    // back substitution on unscaled rows: column q of U over u_qq times row q is subtracted, the rows are
    // divided by their diagonal elements at the end (one barrier per row, no division in the chain)
    const double2 *Dt = D + (long long)ti * CB * CB;
    for (int w = 0; w < CB * CB / CT; w++) {
      const int e = threadIdx.x + w * CT, r = e / CB, c = e % CB;
      x[r][c] = v[w];
      const double q = Dt[c * CB + c].x;
      u[r][c] = make_double2(Dt[e].x / q, Dt[e].y / q);
    }
    __syncthreads();
    for (int q = CB - 1; q > 0; q--) {
      for (int e = threadIdx.x; e < q * CB; e += CT)
        x[e / CB][e % CB] = csubmul(x[e / CB][e % CB], u[e / CB][q], x[q][e % CB]);
      __syncthreads();
    }
    for (int e = threadIdx.x; e < CB * CB; e += CT) {
      const int r = e / CB, c = e % CB, i = ti * CB + r, j = tj * CB + c;
      const double q = Dt[r * CB + r].x;
      if (i < n && j < n) X[(long long)i * n + j] = make_double2(x[r][c].x / q, x[r][c].y / q);
    }
  }
}

// ------------------------------------------------------------------ Hermitian eigen-decomposition
// Cyclic Jacobi rotations in the order of the host routine (hermitian_eigen in abi.cpp: (p, q) row by row),
// run as waves: rotation (p, q) needs the results of (p, q') q' < q and (p', q) p' < p only, so all pairs with
// p + q = t are independent and follow the pairs of t - 1.  The eigenvectors come out with the phases and
// order of the host routine, to rounding.  A wave replaces A by G^H A G and V by V G with G the direct sum of
// its 2 x 2 rotations; every 2 x 2 block of A between two pairs is transformed on its own, from one copy of A
// to the other, so a wave ends with one barrier.  One cluster does it all: its CTAs form every rotation of
// the wave for themselves (n / 2 threads), transform their share of the block rows and their rows of V.
// Latency-bound: a chain of 2 n - 3 waves per sweep, each two L2 round trips, one rotation and one cluster
// barrier.
struct Rot {
  double c, s;
  double2 ph;  // e^{i phi} of A[p][q]
  int on;      // 0: the pair is left alone
};
constexpr int EIG_THREADS = 512;

// (b_p, b_q) of a row times the pair's rotation, as the host's A <- A U and V <- V U
__device__ __forceinline__ void rot_cols(double2 &a, double2 &b, const Rot &g) {
  const double2 uqp = make_double2(-g.s * g.ph.x, g.s * g.ph.y), uqq = make_double2(g.c * g.ph.x, -g.c * g.ph.y);
  const double2 p = a, q = b;
  a = make_double2(p.x * g.c + (q.x * uqp.x - q.y * uqp.y), p.y * g.c + (q.x * uqp.y + q.y * uqp.x));
  b = make_double2(p.x * g.s + (q.x * uqq.x - q.y * uqq.y), p.y * g.s + (q.x * uqq.y + q.y * uqq.x));
}
// the rotation's adjoint on two rows, A <- U^H A
__device__ __forceinline__ void rot_rows(double2 &a, double2 &b, const Rot &g) {
  const double2 uqp = make_double2(-g.s * g.ph.x, -g.s * g.ph.y), uqq = make_double2(g.c * g.ph.x, g.c * g.ph.y);  // conj
  const double2 p = a, q = b;
  a = make_double2(g.c * p.x + (uqp.x * q.x - uqp.y * q.y), g.c * p.y + (uqp.x * q.y + uqp.y * q.x));
  b = make_double2(g.s * p.x + (uqq.x * q.x - uqq.y * q.y), g.s * p.y + (uqq.x * q.y + uqq.y * q.x));
}

// the host routine's rotation of [[a, b], [conj b, d]], with theta = atan2(2 |b|, d - a) / 2 in [0, pi / 2]:
// tan of the angle (or of its complement, when d < a) from tau = (d - a) / 2 |b|, a short chain of roots and
// reciprocals in place of the arc tangent, sine and cosine
__device__ __forceinline__ Rot rotation(double a, double d, double2 b) {
  Rot g;
  const double m = fmax(fabs(b.x), fabs(b.y));
  const double up = m < 1e-140 ? 0x1p500 : 1.0;  // keep the squares in range
  const double bx = b.x * up, by = b.y * up;
  const double r = sqrt(bx * bx + by * by);
  g.on = r >= 1e-300 * up && r > 0.0 ? 1 : 0;
  if (!g.on) {
    g.c = 1.0;
    g.s = 0.0;
    g.ph = make_double2(1.0, 0.0);
    return g;
  }
  // first-order corrections of the roundings of |ph|^2 = 1 and c^2 + s^2 = 1: they would add up over the
  // thousands of rotations of a column
  const double ri = 1.0 / r;
  g.ph = make_double2(bx * ri, by * ri);
  const double ep = 0.5 * fma(-g.ph.y, g.ph.y, fma(-g.ph.x, g.ph.x, 1.0));
  g.ph = make_double2(fma(ep, g.ph.x, g.ph.x), fma(ep, g.ph.y, g.ph.y));
  const double x = (d - a) * up, ax = fabs(x), y = 2.0 * r;
  // t = y / (|x| + sqrt(x^2 + y^2)); the larger of |x| and y in front keeps the squares in range
  const double big = fmax(ax, y), small = fmin(ax, y), q = small / big;
  const double tt = y / (ax + big * sqrt(1.0 + q * q));
  double ci = 1.0 / sqrt(1.0 + tt * tt);
  double si = tt * ci;
  const double es = 0.5 * fma(-si, si, fma(-ci, ci, 1.0));
  ci = fma(es, ci, ci);
  si = fma(es, si, si);
  g.c = x >= 0.0 ? ci : si;
  g.s = x >= 0.0 ? si : ci;
  return g;
}
// the 2 x 2 (2 x 1, 1 x 2, 1 x 1) block of rows p, q and columns k, l; units u (rows) and j (columns)
struct Block {
  int u, j, p, q, k, l;
  bool rp, cp;
  double2 a, b, c, d;
};

// A0 holds the matrix (upper triangle read), A1 and V are work and result; norms [2][cluster size]; the
// eigenvalues (unsorted) go to w, column i of V is the vector of w[i]
__global__ void __launch_bounds__(EIG_THREADS) jacobi_kernel(double2 *A0, double2 *A1, double2 *V, int n, double *norms,
                                                             double *w) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = int(cl.block_rank()), size = int(cl.num_blocks());
  extern __shared__ __align__(16) unsigned char sm[];
  // rotations of a wave, two sets: a thread may form the next wave's while another still rotates its V
  Rot *rots = reinterpret_cast<Rot *>(sm);  // [2][n / 2 + 1]
  __shared__ double red[EIG_THREADS];
  const int tid = threadIdx.x;
  double2 *A = A0, *B = A1;

  // the Hermitian matrix of the upper triangle, V = 1, |A|^2
  double tot = 0.0;
  for (int i = rank; i < n; i += size)
    for (int j = tid; j < n; j += EIG_THREADS) {
      double2 a = i <= j ? A0[(long long)i * n + j] : A0[(long long)j * n + i];
      if (i == j) a.y = 0.0;
      else if (i > j) a.y = -a.y;
      B[(long long)i * n + j] = a;
      V[(long long)i * n + j] = make_double2(i == j ? 1.0 : 0.0, 0.0);
      tot += a.x * a.x + a.y * a.y;
    }
  auto sum = [&](double v, double *slot) {  // block sum in a fixed tree, into this CTA's slot
    red[tid] = v;
    __syncthreads();
    for (int o = EIG_THREADS / 2; o > 0; o >>= 1) {
      if (tid < o) red[tid] += red[tid + o];
      __syncthreads();
    }
    if (tid == 0) slot[rank] = red[0];
  };
  auto all = [&](const double *slot) {  // the CTAs' sums in order: the same value everywhere
    double v = 0.0;
    for (int r = 0; r < size; r++) v += __ldcg(slot + r);
    return v;
  };
  sum(tot, norms);
  cl.sync();
  const double total = all(norms);
  A = A1;
  B = A0;

  for (int sweep = 0; sweep < 60; sweep++) {
    double off = 0.0;
    for (int i = rank; i < n; i += size)
      for (int j = i + 1 + tid; j < n; j += EIG_THREADS) {
        const double2 a = __ldcg(A + (long long)i * n + j);
        off += a.x * a.x + a.y * a.y;
      }
    sum(off, norms + size * (1 + (sweep & 1)));
    cl.sync();
    if (!(all(norms + size * (1 + (sweep & 1))) > 1e-30 * total)) break;
    for (int t = 1; t <= 2 * n - 3; t++) {
      // pairs (p, t - p), p = lo .. lo + np - 1; the other indices stand alone
      const int lo = t - n + 1 > 0 ? t - n + 1 : 0, np = (t - 1) / 2 - lo + 1;
      Rot *rot = rots + (t & 1) * (n / 2 + 1);
      // units: the pairs, then the single indices
      const int alone = n - 2 * np, units = np + alone;
      const int mid = (t & 1) == 0 && t / 2 < n ? t / 2 : -1;  // p = q, when it is an index
      auto single = [&](int k) {  // the k-th index without a partner
        if (t < n) return k == 0 && mid >= 0 ? mid : t + k + (mid >= 0 ? 0 : 1);
        return k < lo ? k : mid;
      };
      // this CTA's blocks: its row units (every size-th one) times all column units
      const int mine = units > rank ? (units - rank + size - 1) / size : 0, items = mine * units;
      auto fetch = [&](int e, Block &k) {
        const int ur = e / units;
        k.u = rank + ur * size;
        k.j = e - ur * units;
        k.rp = k.u < np;
        k.cp = k.j < np;
        k.p = k.rp ? lo + k.u : single(k.u - np);
        k.q = k.rp ? t - k.p : k.p;
        k.k = k.cp ? lo + k.j : single(k.j - np);
        k.l = k.cp ? t - k.k : k.k;
        const double2 *Ap = A + (long long)k.p * n, *Aq = A + (long long)k.q * n;
        k.a = __ldcg(Ap + k.k);
        if (k.cp) k.b = __ldcg(Ap + k.l);
        if (k.rp) k.c = __ldcg(Aq + k.k);
        if (k.rp && k.cp) k.d = __ldcg(Aq + k.l);
      };
      Block blk;
      if (tid < items) fetch(tid, blk);  // in flight while the rotations are formed
      for (int j = tid; j < np; j += EIG_THREADS) {
        const int p = lo + j, q = t - p;
        const double2 b = __ldcg(A + (long long)p * n + q);
        const double a = __ldcg(&A[(long long)p * n + p].x), d = __ldcg(&A[(long long)q * n + q].x);
        rot[j] = rotation(a, d, b);
      }
      __syncthreads();
      for (int e = tid; e < items; e += EIG_THREADS) {
        if (e != tid) fetch(e, blk);
        const Rot gc = blk.cp ? rot[blk.j] : Rot{}, gr = blk.rp ? rot[blk.u] : Rot{};
        if (blk.cp && gc.on) {
          rot_cols(blk.a, blk.b, gc);
          if (blk.rp) rot_cols(blk.c, blk.d, gc);
        }
        if (blk.rp && gr.on) {
          rot_rows(blk.a, blk.c, gr);
          if (blk.cp) rot_rows(blk.b, blk.d, gr);
          if (blk.cp && blk.j == blk.u) {  // the rotated pair itself
            blk.b = blk.c = make_double2(0.0, 0.0);
            blk.a.y = blk.d.y = 0.0;
          }
        }
        double2 *Bp = B + (long long)blk.p * n, *Bq = B + (long long)blk.q * n;
        Bp[blk.k] = blk.a;
        if (blk.cp) Bp[blk.l] = blk.b;
        if (blk.rp) Bq[blk.k] = blk.c;
        if (blk.rp && blk.cp) Bq[blk.l] = blk.d;
      }
      cl.barrier_arrive();
      // meanwhile this CTA's rows of V (no other CTA touches them)
      const int rows = n > rank ? (n - rank + size - 1) / size : 0;
      for (int e = tid; e < rows * np; e += EIG_THREADS) {
        const int r = e / np, j = e - r * np;
        if (!rot[j].on) continue;
        double2 *v = V + (long long)(rank + r * size) * n;
        const int p = lo + j, q = t - p;
        double2 a = v[p], b = v[q];
        rot_cols(a, b, rot[j]);
        v[p] = a;
        v[q] = b;
      }
      cl.barrier_wait();
      double2 *s = A;
      A = B;
      B = s;
    }
  }
  for (int i = rank * EIG_THREADS + tid; i < n; i += size * EIG_THREADS) w[i] = __ldcg(&A[(long long)i * n + i].x);
}

// out[i][k] = V[i][order[k]]
__global__ void permute_columns_kernel(const double2 *__restrict__ V, const int *__restrict__ order, int n,
                                       double2 *__restrict__ out) {
  const long long m = (long long)n * n;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < m; e += (long long)gridDim.x * blockDim.x) {
    const int i = int(e / n), k = int(e - (long long)i * n);
    out[e] = V[(long long)i * n + order[k]];
  }
}

}  // namespace

// S [n][n] -> X = U^-1 of S = U^H U (S is overwritten); *bad_dev becomes 1, and X is not written, when S is not
// positive definite
void launch_cholesky_inverse(Ctx &ctx, int n, double2 *S, double2 *X, int *bad_dev) {
  const int nt = (n + CB - 1) / CB;
  double2 *D = static_cast<double2 *>(dev_alloc(ctx, sizeof(double2) * size_t(nt) * CB * CB));
  int *flags = static_cast<int *>(dev_alloc(ctx, sizeof(int) * size_t(nt)));  // what the rows before k found
  INQB_CUDA(cudaMemsetAsync(flags, 0, sizeof(int) * size_t(nt), ctx.stream));
  INQB_CUDA(cudaMemsetAsync(bad_dev, 0, sizeof(int), ctx.stream));
  for (int k = 0; k < nt; k++) {
    const int left = nt - 1 - k;
    int *after = left > 0 ? flags + k + 1 : bad_dev;
    chol_row_kernel<<<left > 0 ? left : 1, CT, 0, ctx.stream>>>(S, D + size_t(k) * CB * CB, n, k, flags + k, after);
    LAUNCHED(ctx);
    if (left > 0) {
      chol_update_kernel<<<left * (left + 1) / 2, CT, 0, ctx.stream>>>(S, n, k, after);
      LAUNCHED(ctx);
    }
  }
  tri_inverse_kernel<<<nt, CT, 0, ctx.stream>>>(S, D, X, n, bad_dev);
  LAUNCHED(ctx);
  dev_free(ctx, flags);
  dev_free(ctx, D);
}

// A [n][n] (overwritten) -> eigenvalues w_dev [n], unsorted, and V with the vector of w[i] in column i
void launch_jacobi(Ctx &ctx, int n, double2 *A, double2 *V, double *w_dev) {
  double2 *B = static_cast<double2 *>(dev_alloc(ctx, sizeof(double2) * size_t(n) * n));
  double *norms = static_cast<double *>(dev_alloc(ctx, sizeof(double) * 3 * 16));
  const size_t smem = 2 * sizeof(Rot) * size_t(n / 2 + 1);
  INQB_REQUIRE(smem + sizeof(double) * EIG_THREADS <= ctx.max_smem_optin, INQB_ERR_UNSUPPORTED,
               "too many states for the eigen-decomposition");  // beside the kernel's sums in static shared memory
  ensure_smem_attr(reinterpret_cast<const void *>(jacobi_kernel), smem);
  INQB_CUDA(cudaFuncSetAttribute(jacobi_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  cfg.blockDim = dim3(EIG_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx.stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // 8 CTAs, 16 for larger matrices where the device can hold such a cluster
  int size = 8, fits = 0;
  for (size = n <= 96 ? 8 : 16; size > 1; size /= 2) {
    attr[0].val.clusterDim.x = unsigned(size);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(unsigned(size));
    if (cudaOccupancyMaxActiveClusters(&fits, jacobi_kernel, &cfg) == cudaSuccess && fits > 0) break;
    cudaGetLastError();
  }
  if (size <= 1) {
    attr[0].val.clusterDim.x = 1;
    cfg.gridDim = dim3(1);
  }
  INQB_CUDA(cudaLaunchKernelEx(&cfg, jacobi_kernel, A, B, V, n, norms, w_dev));
  LAUNCHED(ctx);
  dev_free(ctx, norms);
  dev_free(ctx, B);
}

void launch_permute_columns(Ctx &ctx, const double2 *V, const int *order_dev, int n, double2 *out) {
  const long long blocks = ((long long)n * n + 255) / 256;
  permute_columns_kernel<<<unsigned(blocks < 1184 ? blocks : 1184), 256, 0, ctx.stream>>>(V, order_dev, n, out);
  LAUNCHED(ctx);
}

}  // namespace inqb
