// The rule of the whole-line z passes (zlines_of) over every line length it knows, state counts from one to its
// limit, grids with few, odd and many lines, both precisions and every ring depth an option may ask for: what the
// kernel takes for granted about alignment, shared memory, threads and its reciprocal divisions.
#include <cstdio>
#include <cstdlib>

#include "fft2_lengths.h"

using namespace inqb;

#define CHECK(c)                                                                                           \
  do {                                                                                                     \
    if (!(c)) {                                                                                            \
      std::printf("%s: %d x %d x %d, %d states, %d bytes, depth %d\n", #c, b.n[0], b.n[1], n, S, es, depth); \
      return 1;                                                                                            \
    }                                                                                                      \
  } while (0)

// the kernel's division by a reciprocal (div_by in fft2.cuh; launch_zlines makes the reciprocals)
static int div_by(long long i, long long d) {
  const unsigned m = d == 1 ? 0u : unsigned(((1ull << 32) + d - 1) / d);
  return m ? int((unsigned long long)(unsigned(i)) * m >> 32) : int(i);
}

int main() {
  const int lengths[] = {
#define INQB_X(N, A, B) N,
      INQB_FFT2_LENGTHS(INQB_X)
#undef INQB_X
  };
  const int grids[][2] = {{1, 1}, {1, 2}, {2, 3}, {3, 5}, {16, 18}, {21, 25}, {48, 48}, {120, 128}, {2048, 1}};
  Ctx ctx;
  ctx.device_sms = ctx.num_sms = 148;
  ctx.max_smem_optin = 232448;
  long long used = 0;
  for (int n : lengths)
    for (const auto &g : grids)
      for (int es : {8, 16})
        for (int depth : {0, 1, 2, 3, 4, 8})
          for (int S = 1; S <= 1024; S += S < 70 ? 1 : 13) {
            Basis b;
            b.n[0] = g[0];
            b.n[1] = g[1];
            b.n[2] = n;
            b.npoints = (long long)g[0] * g[1] * n;
            ctx.fft_stages = depth;
            const v2::ZLines z = v2::zlines_of(ctx, b, S, es);
            if (z.lpt == 0) continue;
            used++;
            const long long lines = (long long)g[0] * g[1], line = (long long)n * S, chunk = line * z.lpt;
            const long long last = lines % z.lpt ? lines % z.lpt : z.lpt;
            CHECK((chunk * es) % 16 == 0 && (last * line * es) % 16 == 0);  // every bulk copy
            CHECK(chunk * es < (1 << 20));                                  // a barrier's transaction count
            const size_t top = ctx.max_smem_optin, smem = v2::zlines_smem(n, S, es, z.lpt, z.stages);
            CHECK(smem <= top);
            // ring, twiddles, factors of the chunk's points, two barriers per stage, flag
            size_t at = size_t(z.stages) * chunk * es + size_t(es == 8 ? 2 : 1) * n * es + size_t(z.lpt) * n * (es / 2);
            at = (at + 15) & ~size_t(15);
            CHECK(at + 16 * size_t(z.stages) + 4 <= smem);
            CHECK(z.stages >= 2 && z.stages <= 8);
            if (depth > 0) {  // the depth asked for, or the deepest that fits
              const int want = depth < 2 ? 2 : depth;
              CHECK(z.stages == want || (z.stages < want && v2::zlines_smem(n, S, es, z.lpt, z.stages + 1) > top));
            }
            CHECK(z.threads >= 32 && z.threads <= (es == 16 ? 320 : 480) && z.threads % 32 == 0);
            if (depth > 0) continue;
            const int n2 = v2::split_n2(n), n1 = n / n2;
            for (long long d : {(long long)S, (long long)n2 * S, (long long)n1 * S})
              for (long long q = 0; q * d <= chunk; q++)  // both sides of every step of the quotient
                for (long long i = q * d; i >= q * d - 1 && i >= 0; i--) CHECK(div_by(i, d) == i / d);
          }
  std::printf("%lld forms\n", used);
  return used > 10000 ? 0 : 1;
}
