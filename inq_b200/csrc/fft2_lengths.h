// Line lengths of the specialised FFT passes (fft2.cuh) and the rules that say which decomposition of a
// set a pass uses.  Host code only: shared by the dispatch and by the operator, which keeps the z
// frequencies in digit-reversed order between passes only when specialised kernels run all of them.
#pragma once

#include "inqb_internal.h"

namespace inqb {
namespace v2 {

// X(N, N1, N2): every product of 2, 3, 5 and 7 from 16 to 128 (grids follow from a spacing as the next such
// product) with two factors N = N1 x N2 of at most 16 points each, what a thread's registers hold: all but
// 125 = 5 x 25.  Against the generic kernel, which moves one tile per CTA without a pipeline (about 1.6 TB/s),
// H at 54 x 60 x 45 x 50 double takes 382 us instead of 942.
#define INQB_FFT2_LENGTHS(X)                                                                             \
  X(16, 4, 4) X(18, 3, 6) X(20, 4, 5) X(21, 3, 7) X(24, 8, 3) X(25, 5, 5) X(27, 3, 9) X(28, 4, 7)        \
  X(30, 5, 6) X(32, 8, 4) X(35, 5, 7) X(36, 6, 6) X(40, 8, 5) X(42, 6, 7) X(45, 5, 9) X(48, 8, 6)        \
  X(49, 7, 7) X(50, 5, 10) X(54, 6, 9) X(56, 8, 7) X(60, 6, 10) X(63, 7, 9) X(64, 8, 8) X(70, 7, 10)     \
  X(72, 8, 9) X(75, 5, 15) X(80, 8, 10) X(81, 9, 9) X(84, 7, 12) X(90, 9, 10) X(96, 8, 12) X(98, 7, 14)  \
  X(100, 10, 10) X(105, 7, 15) X(108, 9, 12) X(112, 8, 14) X(120, 8, 15) X(126, 9, 14) X(128, 8, 16)

// A set small enough to stay in L2 from one pass to the next
inline bool stays_in_l2(const Basis &b, int S, int elem_bytes) {
  return size_t(b.npoints) * S * elem_bytes <= (size_t(128) << 20);
}

// N2 of a specialised length, 0 for the others
inline int split_n2(int n) {
  switch (n) {
#define INQB_X(N, A, B) case N: return B;
    INQB_FFT2_LENGTHS(INQB_X)
#undef INQB_X
  }
  return 0;
}
// lengths that also have kernels with double arithmetic on single-precision orbitals (mixed_compute 1..3)
constexpr bool has_wide_arith(int n) {
  return n == 24 || n == 32 || n == 40 || n == 48 || n == 64 || n == 72 || n == 96 || n == 120 || n == 128;
}

// y and x passes over flattened columns (context option fft_flat): the rows of the flattened view are
// 16-byte multiples, its 32-bit words stay below 2^31 (a TMA coordinate), and the state rows are not whole
// 512-byte rows already (then the line tiles are the same tiles with cheaper index arithmetic).
inline bool flat_ok(const Ctx &ctx, const Basis &b, int S, int elem_bytes, int axis) {
  const long long words = (axis == 1 ? (long long)b.n[2] : (long long)b.n[1] * b.n[2]) * S * (elem_bytes / 4);
  return ctx.fft_flat && axis != 2 && (size_t(b.n[2]) * S * elem_bytes) % 16 == 0 && words < (1LL << 31) &&
         (size_t(S) * elem_bytes) % 512 != 0;
}

// z passes over whole lines: the chunk of `lpt` lines a CTA takes at a time is contiguous in memory.
struct ZLines {
  int lpt = 0;      // lines per chunk; 0: the lines do not fit, or their rows already are whole 256-byte tiles
  int stages = 2;
  int threads = 0;  // compute threads per CTA
};
inline size_t zlines_smem(int n, int S, int elem_bytes, int lpt, int stages) {
  const size_t tw = size_t(elem_bytes == 8 ? 2 : 1) * n * elem_bytes;
  const size_t bars = stages < 8 ? 128 : 160;  // two barriers per stage and a flag
  return size_t(stages) * lpt * n * S * elem_bytes + tw + ((size_t(lpt) * n * (elem_bytes / 2) + 15) & ~size_t(15)) + bars;
}
inline ZLines zlines_of(const Ctx &ctx, const Basis &b, int S, int elem_bytes) {
  ZLines z;
  const int n = b.n[2], n2 = split_n2(n);
  if (!ctx.fft_flat || n2 == 0 || (size_t(S) * elem_bytes) % 256 == 0) return z;
  const long long lines = (long long)b.n[0] * b.n[1];
  const size_t line = size_t(n) * S * elem_bytes;
  // chunks start and end on 16-byte boundaries: pairs of lines when one line is an odd number of 8-byte elements
  const int step = line % 16 ? 2 : 1;
  if (lines % step) return z;
  // about 16 KB per chunk, but at least two chunks per SM while there are lines for them
  long long lpt = (long long)(16384 / line);
  if (lpt > lines / (2LL * ctx.device_sms)) lpt = lines / (2LL * ctx.device_sms);
  lpt = lpt < step ? step : lpt / step * step;
  const size_t top = ctx.max_smem_optin;
  if (zlines_smem(n, S, elem_bytes, int(lpt), 2) > top) return z;
  z.stages = zlines_smem(n, S, elem_bytes, int(lpt), 3) <= top / 2 ? 3 : 2;
  if (ctx.fft_stages > 0) {  // the depth asked for, as far as it fits (two stages do)
    z.stages = ctx.fft_stages < 2 ? 2 : ctx.fft_stages;
    while (z.stages > 2 && zlines_smem(n, S, elem_bytes, int(lpt), z.stages) > top) z.stages--;
  }
  const size_t smem = zlines_smem(n, S, elem_bytes, int(lpt), z.stages) + 1024;
  const int ctas = int((top + 1024) / smem);
  // 10 to 18 warps per SM, by the CTAs that shared memory would hold; registers allow fewer in most final passes in double
  const int most = elem_bytes == 16 ? 320 : 480;
  z.threads = ctas <= 1 ? most : (ctas == 2 ? 256 : (ctas == 3 ? 192 : 128));
  const long long items = lpt * S * (n2 > n / n2 ? n2 : n / n2);
  if (items < z.threads) z.threads = int((items + 31) / 32 * 32);
  z.lpt = int(lpt);
  return z;
}

// Final passes of single-precision sets beyond L2 that keep the line tiles although their other z passes take whole
// lines: three transits, whose second input a tile brings in by TMA, and the whole-line kernel reads it with its
// registers' loads.  H single, whole lines against tiles in the final pass: 96^3 x 44 815 -> 730 us, x 62 1024 -> 957,
// 72^3 x 62 462 -> 438, x 180 1245 -> 1180, 64^3 x 190 872 -> 833, 48^3 x 180 403 -> 374; the same at 96^3 x 110 and more.
// Not at 80 or 90 points (80^3 x 40 446 -> 478 us, 90^3 x 34 598 -> 645) nor at 120 (x 34 1318 -> 1433: its second
// tiles have a single buffer), not in L2 (48^3 x 80 176 -> 197), and not in double (96^3 x 62 1797 -> 1880).
inline bool final_tiles(const Basis &b, int n, int S) {
  return has_wide_arith(n) && n <= 96 && S >= 32 && S % 2 == 0 && !stays_in_l2(b, S, 8);
}

// whether a specialised pass moves this set along `axis`, given that it computes in the storage type
inline bool covers(const Ctx &ctx, const Basis &b, int S, int elem_bytes, int axis) {
  if (ctx.fft_impl == 1 || split_n2(b.n[axis]) == 0) return false;
  if (flat_ok(ctx, b, S, elem_bytes, axis)) return true;
  if (axis == 2 && zlines_of(ctx, b, S, elem_bytes).lpt > 0) return true;
  if (S < 256 / elem_bytes) return false;  // fewer states than one 256-byte row: generic kernel
  // rows that are not 16-byte multiples: single-precision orbitals only (the compute threads copy them)
  return (size_t(S) * elem_bytes) % 16 == 0 || elem_bytes == 8;
}

}  // namespace v2
}  // namespace inqb
