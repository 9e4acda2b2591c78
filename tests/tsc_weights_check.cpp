// Compares the 9-point deposit weights and their products (fx::tsc_weights_q58,
// fx::mul_floor in fixmap.cuh) with the separate squares and the exact 128-bit
// products they stand for, bit for bit, over random and edge fractions; prints
// the number that differ.
#include "py-orbit_gb300/csrc/fixmap.cuh"

#include <cstdio>
#include <cstdlib>
#include <random>

using namespace orbit;
typedef __int128 i128;

static int64_t sq_q58(int64_t g) {  // g in Q56
  const i128 a = (i128)(g < 0 ? -g : g) << 5;
  return (int64_t)((a * a) >> 64);
}

int main(int, char** argv) {
  std::mt19937_64 g(std::atoi(argv[2]));
  const long n = std::atol(argv[1]);
  const int64_t lim = 5ll << 54;  // 1.25 in Q56
  long bad = 0;
  for (long i = 0; i < n; ++i) {
    int64_t f[2];
    for (int c = 0; c < 2; ++c) {
      const int kind = g() % 8;
      f[c] = (int64_t)(g() % (uint64_t)(2 * lim + 1)) - lim;
      if (kind < 5) f[c] = (int64_t)(g() % (1ull << 56)) - (1ll << 55);  // inside the cell
      if (kind == 5) f[c] = (int64_t)(g() % 5) - 2 + ((int64_t)(g() % 11) - 5) * (1ll << 54);
      if (kind == 6) f[c] &= ~0xffffffffll;
    }
    fx::V a[3], b[3];
    int64_t w[2][3];
    for (int c = 0; c < 2; ++c) {
      w[c][0] = sq_q58(f[c] - (1ll << 55)) >> 1;
      w[c][1] = (3ll << 56) - sq_q58(f[c]);
      w[c][2] = sq_q58(f[c] + (1ll << 55)) >> 1;
    }
    fx::tsc_weights_q58(f[0] << 5, 4, a);
    fx::tsc_weights_q58(f[1] << 5, 1, b);
    const int K = 29 + g() % 27, sh = 57 - K;
    for (int j = 0; j < 3; ++j)
      for (int k = 0; k < 3; ++k) {
        const int64_t p = (int64_t)(((i128)(w[0][j] << 4) * (w[1][k] << 4)) >> 64);  // Q60
        const int64_t want = (p + (1ll << (59 - K))) >> (60 - K);
        if (fx::mul_floor_r(a[j], b[k], 1 << (sh - 1)) >> sh != want ||
            fx::mul_floor(a[j], b[k], 1ll << (sh - 1)) >> sh != want) ++bad;
      }
  }
  std::printf("%ld\n", bad);
  return 0;
}
