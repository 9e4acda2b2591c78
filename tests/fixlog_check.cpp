// log_q55 (fixlog.cuh) against long double over argv[1] random arguments of seed
// argv[2]; prints its largest error and that of std::log(double), both in units
// of 2^-53 max(1, |log|).
#include "py-orbit_gb300/csrc/fixlog.cuh"

#include <cstdio>
#include <cstdlib>
#include <random>

int main(int, char** argv) {
  std::mt19937_64 g(std::atoi(argv[2]));
  const long n = std::atol(argv[1]);
  orbit::LogTab t;
  orbit::make_log_tab(&t);
  double worst = 0.0, lib = 0.0;
  for (long i = 0; i < n; ++i) {
    uint64_t u = g() & ((1ull << 52) - 1);
    const int kind = i % 4;
    if (kind == 1) u = (u & ~(((1ull << 7) - 1) << 45) & ~((1ull << 45) - 1)) | ((g() & 127) << 45) | (g() % 3);  // at a table edge
    if (kind == 2) u = (g() & 1) ? g() % 1000 : ((1ull << 52) - 1 - g() % 1000);                                  // next to a power of two
    const int e = kind == 3 ? (int)(g() % 512) - 256 : (int)(g() % 40) - 30;
    const double v = orbit::sf::from_bits(u | ((uint64_t)(1023 + e) << 52));
    int64_t q;
    if (!orbit::log_q55(&t, v, &q)) {
      std::printf("refused %a\n", v);
      return 1;
    }
    const long double l = std::log((long double)v), s = std::fabs(l) > 1.0L ? std::fabs(l) : 1.0L;
    const double a = (double)(std::fabs((long double)q * 0.25L - l * 9007199254740992.0L) / s);
    const double b = (double)(std::fabs((long double)std::log(v) - l) * 9007199254740992.0L / s);
    worst = a > worst ? a : worst;
    lib = b > lib ? b : lib;
  }
  for (double v : {0.0, -1.0, 1e300, 1e-300, 1e-310, (double)INFINITY, (double)NAN}) {
    int64_t q;
    if (orbit::log_q55(&t, v, &q)) {
      std::printf("accepted %a\n", v);
      return 1;
    }
  }
  std::printf("%.3f %.3f\n", worst, lib);
  return 0;
}
