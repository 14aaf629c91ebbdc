// The bit forms of the double <-> double-single conversions against the plain
// ones, on the host: random significands over every exponent, ties, powers of
// two and their neighbours, zeros, denormals, infinities.
#include "fft_reg.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

using namespace fame;

static int bad = 0;
static long long covered = 0;
static void check(double d) {
  uint64_t u;
  std::memcpy(&u, &d, 8);
  ff v;
  if (ff_split_bits((uint32_t)(u >> 32), (uint32_t)u, v)) {
    const ff w(d);
    ++covered;
    if ((f32_bits(v.hi) != f32_bits(w.hi) || v.lo != w.lo) && bad++ < 10)
      std::printf("split %a: %a %a, want %a %a\n", d, v.hi, v.lo, w.hi, w.lo);
  }
  const ff w(d);
  for (float f : {w.hi, w.lo}) {
    uint32_t h, l;
    if (f32_widen_bits(f, h, l)) {
      const uint64_t x = ((uint64_t)h << 32) | l;
      double g;
      std::memcpy(&g, &x, 8);
      const double want = f;
      if (std::memcmp(&g, &want, 8) != 0 && bad++ < 10) std::printf("widen %a: %a\n", f, g);
    } else if (f != 0.0f && std::isnormal(f) && bad++ < 10) {
      std::printf("widen refuses %a\n", f);
    }
  }
}

int main() {
  std::mt19937_64 g(1);
  for (int e = -1074; e <= 1024; ++e)
    for (int k = 0; k < 500; ++k) {
      uint64_t m = g() >> 12;
      if (k < 64) m = (m & ~0x1fffffffull) | 0x10000000ull;                // ties
      else if (k < 96) m = (m & ~0x1fffffffull) | (0x10000000ull + k - 80);  // and their neighbours
      else if (k < 100) m = k == 96 ? 0 : k == 97 ? 1 : k == 98 ? 0xfffffffffffffull : 0xfffffe0000000ull;
      const uint64_t b = e < -1022 ? m >> (-1022 - e) : ((uint64_t)(e + 1023) << 52) | m;
      for (uint64_t s : {0ull, 1ull << 63}) {
        const uint64_t u = b | s;
        double d;
        std::memcpy(&d, &u, 8);
        if (!std::isnan(d)) check(d);
      }
    }
  check(0.0);
  check(-0.0);
  check(INFINITY);
  if (covered < 2ll * 500 * 201) {
    std::printf("only %lld values in range\n", covered);
    return 1;
  }
  std::printf("%lld splits, %d wrong\n", covered, bad);
  return bad != 0;
}
