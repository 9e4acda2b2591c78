// The natural logarithm in 64-bit fixed point, by table lookup and a short
// series (P. T. P. Tang, "Table-driven implementation of the logarithm function
// in IEEE floating-point arithmetic", ACM TOMS 16, 1990): with v = 2^e m and c
// near 1/m from the top seven bits of m's fraction,
//   log v = e log 2 + log(1/c) + log(1 + t),   t = m c - 1,   |t| <= 2^-8.
// About a hundred integer instructions, where the logarithm of the math library
// keeps the FP64 pipe for some forty instructions of 64 clocks a warp.
#pragma once

#include "fixmap.cuh"

namespace orbit {

struct LogTab {
  struct {
    uint32_t c;   // 2^32 / (1 + (i + 1/2) / 128)
    int64_t l;    // log(2^32 / c) in Q55
  } at[128];
  int64_t ln2;    // log 2 in Q55, rounded down
  uint32_t ln2x;  // the rest in Q87
};

inline void make_log_tab(LogTab* t) {
  for (int i = 0; i < 128; ++i) {
    t->at[i].c = (uint32_t)std::floor(4294967296.0L / (1.0L + (i + 0.5L) / 128.0L) + 0.5L);
    t->at[i].l = (int64_t)std::floor(-std::log((long double)t->at[i].c / 4294967296.0L) * 36028797018963968.0L + 0.5L);
  }
  const long double l2 = std::log(2.0L) * 36028797018963968.0L;
  t->ln2 = (int64_t)std::floor(l2);
  t->ln2x = (uint32_t)((l2 - std::floor(l2)) * 4294967296.0L);
}

// log(v) in Q55 to about 2^-54; false for v beyond 2^+-256 (among them zero,
// negative and non-finite ones).
FX_HD bool log_q55(const LogTab* t, double v, int64_t* out) {
  const uint64_t u = sf::bits(v);
  const int e = (int)(u >> 52) - 1023;
  if ((unsigned)(e + 256) > 512u) return false;
  const uint64_t m = (u << 11) | (1ull << 63);  // Q63
  const int i = (int)(u >> 45) & 127;
  const uint64_t c = t->at[i].c;
  // m c in Q95; less 1 in Q70
  const uint64_t hi = (m >> 32) * c, lo = (m & 0xffffffffull) * c;
  const int64_t t70 = (int64_t)((hi << 7) + (lo >> 25));
  const fx::V T = fx::sp(t70);
  // log(1 + t) = t (1 + t (-1/2 + t (1/3 + t (-1/4 + t (1/5 + t (-1/6 + t / 7)))))),
  // the sums in Q62
  const int64_t one = 1ll << 62;
  int64_t p = one / 7;
  p = -one / 6 + (fx::mul(T, fx::sp(p)) >> 6);
  p = one / 5 + (fx::mul(T, fx::sp(p)) >> 6);
  p = -one / 4 + (fx::mul(T, fx::sp(p)) >> 6);
  p = one / 3 + (fx::mul(T, fx::sp(p)) >> 6);
  p = -one / 2 + (fx::mul(T, fx::sp(p)) >> 6);
  const int64_t s = fx::mul(T, fx::sp(p)) >> 6;          // log(1 + t) / t - 1
  const int64_t q68 = (t70 >> 2) + fx::mul(T, fx::sp(s));  // Q68
  *out = t->at[i].l + ((q68 + (1ll << 12)) >> 13) + e * t->ln2 + (int64_t)(((int64_t)e * t->ln2x) >> 32);
  return true;
}

}  // namespace orbit
