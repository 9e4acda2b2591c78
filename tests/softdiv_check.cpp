// Compares sf::div (softf64.cuh) with the host's IEEE division, bit for bit:
// argv[1] random pairs of seed argv[2]; prints the number that differ.
#include "softf64.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

int main(int, char** argv) {
  std::mt19937_64 g(std::atoi(argv[2]));
  const long n = std::atol(argv[1]);
  const uint64_t sign = 1ull << 63, frac = (1ull << 52) - 1, expo = 0x7ffull << 52;
  long bad = 0;
  for (long i = 0; i < n; ++i) {
    uint64_t a = g(), b = g();
    const int kind = i % 7;
    if (kind < 4) {  // quotients well inside the normal range
      a = (a & (sign | frac)) | ((uint64_t)(993 + g() % 60) << 52);
      b = (b & (sign | frac)) | ((uint64_t)(993 + g() % 60) << 52);
    }
    if (kind == 1) b &= ~(0xfffffull << 32);             // short divisors
    if (kind == 2) a &= ~0xfffffull, b &= ~0xffffffffull;
    if (kind == 3) b = (b & (sign | expo)) | (frac - g() % 16);  // just below a power of two
    if (kind == 4) {                                     // exact quotients
      const double q = (double)(g() % 4096 + 1), d = (double)(g() % 100000 + 1), p = q * d;
      std::memcpy(&a, &p, 8);
      std::memcpy(&b, &d, 8);
    }
    if (kind == 5) b = (b & sign) | ((uint64_t)(1000 + g() % 40) << 52) | (g() % 8);  // just above one
    double x, y;
    std::memcpy(&x, &a, 8);
    std::memcpy(&y, &b, 8);
    const double h = x / y, s = orbit::sf::div(x, y);
    if (std::memcmp(&h, &s, 8) != 0 && !(std::isnan(h) && std::isnan(s))) ++bad;
  }
  std::printf("%ld\n", bad);
  return 0;
}
