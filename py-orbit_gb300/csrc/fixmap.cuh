// The TEAPOT maps in 64-bit fixed point, for the fused lattice pass.
//
// GB300 issues one binary64 instruction per sub-partition every 64 clocks and
// an integer multiply every other clock, so the FP64 maps (even with their
// multiplies emulated on the integer pipes, ~45 instructions each) bound the
// pass.  Between two kicks every particle goes through the same short list of
// maps and the beam's extents are known, so the coordinates can be held as
// 64-bit integers with one scale for the whole bunch: x, y in units of
// 2^-Sx, xp, yp in units of 2^-Sp, the sum of the changes of z in units of
// 2^-Sd, and dp_p, 1/(1+dp_p) - 1 as fractions.  A product is four
// instructions (three 32 x 32 + 64-bit multiply-adds and a shift) and a sum
// of products about three more per term, with one rounding at the end.
//
// Accuracy.  The scales put the bunch's bound at 2^61 units at most: a rounding
// is 2^-61 of the bound where binary64 rounds by 2^-53 of the value.  One scale
// serves both planes and every particle, so it has to suit the smaller of x and
// y (xp and yp) at its typical size, the geometric mean of a sample followed
// through the maps: the pass runs in fixed point only where each keeps the 2^53
// units of a double (fx::fine_enough).  Round beams have 2^55 to 2^58, which is
// the room for planes apart.  Gaussian beams through random drifts, quadrupoles
// with fringes, sextupoles and bends, planes up to a factor of 1e5 apart: rms
// error of a coordinate over binary64's on the same particles, by its typical
// size in units: 2^55 0.45, 2^54 0.47 (at most 1.03), 2^53 0.57 (1.13), 2^52 0.68
// (1.3), 2^50 1.7 (3.6), 2^48 6.0.
//
// The bound is the extent or 24 times the typical size, whichever is less, so a
// few far particles cannot coarsen the others' units; a particle beyond it, one
// whose kick exceeds a quarter of the momentum bound, and one with |dp_p| >= 1/8
// take the FP64 routines, and so does the whole pass where the maps' constants do
// not fit the scales (prep_pass).
//
// The functions are __host__ __device__: a host build checks them against
// extended-precision maps.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#include "softf64.cuh"
#include "../../include/orbit_gb300.h"

#ifdef __CUDACC__
#define FX_HD __host__ __device__ __forceinline__
#else
#define FX_HD inline
#endif

namespace orbit {

// A compiled map: its constants for the FP64 routines (teapot.cuh) and, from
// fx::compile_fixed, for the fixed-point form: f bounds the map's effect on
// the coordinates, v are the constants fx::consts_op scales.
struct DevOp {
  int code, i0, i1, i2;
  double c[12];
  float f[8];
  double v[10];
};

namespace fx {

// A 64-bit integer h 2^32 + l with l signed.
struct V {
  int h, l;
};

FX_HD V sp(int64_t v) {
  V r;
  r.l = (int)(uint32_t)v;
  r.h = (int)(v >> 32) + (int)((uint32_t)r.l >> 31);
  return r;
}

FX_HD int64_t join(V a) { return (int64_t)a.h * 4294967296ll + a.l; }

static const int64_t kRnd = 0x80000000ll;

// c + a b: one instruction (left to itself the compiler widens some of the
// operands first and multiplies in 64 bits: 1468 instructions a particle for
// a drift segment, 566 of them multiplies, against 1119).
FX_HD int64_t mad(int a, int b, int64_t c) {
#ifdef __CUDA_ARCH__
  int64_t r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return (int64_t)a * b + c;
#endif
}

// The sum of the products' middle words, and its high word joined to a base.
FX_HD int64_t mid(V a, V b, int64_t t) { return mad(a.l, b.h, mad(a.h, b.l, t)); }
FX_HD int64_t mids(V a, V b, int64_t t) { return mad(a.l, -b.h, mad(-a.h, b.l, t)); }  // less a b
FX_HD int64_t top(int64_t t, int64_t base) { return base + (t >> 32); }

// base + (a b) / 2^64, and sums of two and three such products with one
// rounding.  The low words' products (below 2^-2 of a unit, signed) are left
// out.  One constant of a sum may reach 2^63, the others 2^61 (2^62 in a sum
// of two); the values stay below 2^61: the middle words' sum stays below 2^63.
FX_HD int64_t mul(V a, V b, int64_t base = 0) { return mad(a.h, b.h, top(mid(a, b, kRnd), base)); }
FX_HD int64_t mul2(V a, V b, V c, V d, int64_t base = 0) {
  return mad(c.h, d.h, mad(a.h, b.h, top(mid(c, d, mid(a, b, kRnd)), base)));
}
FX_HD int64_t mul3(V a, V b, V c, V d, V e, V f, int64_t base = 0) {
  return mad(e.h, f.h, mad(c.h, d.h, mad(a.h, b.h, top(mid(e, f, mid(c, d, mid(a, b, kRnd))), base))));
}
// base + (a b - c d) / 2^64; the high words carry the sign (a low word of
// -2^31 has no negative).
FX_HD int64_t mul2s(V a, V b, V c, V d, int64_t base = 0) {
  return mad(-c.h, d.h, mad(a.h, b.h, top(mids(c, d, mid(a, b, kRnd)), base)));
}

// base + floor(a b / 2^64), exactly: the sums floor at 2^32 and at 2^64 nest.
// |a| < 1.6 2^62 and |b| <= 2^61, or both up to 2^62.
FX_HD int64_t mul_floor(V a, V b, int64_t base = 0) {
  return mad(a.h, b.h, top(mad(a.l, b.h, mad(a.h, b.l, mad(a.l, b.l, 0) >> 32)), base));
}

// The same for 0 <= base < 2^28 and products below 2^123: added at 2^32, a
// carry less.
FX_HD int64_t mul_floor_r(V a, V b, int base) {
  const int64_t ll = mad(a.l, b.l, 0);
  const int64_t t = (int64_t)(((uint64_t)(uint32_t)((int)(ll >> 63) + base) << 32) | (uint32_t)(ll >> 32));
  return mad(a.h, b.h, mad(a.l, b.h, mad(a.h, b.l, t)) >> 32);
}

// The 9-point weights of f (Q61, a multiple of 32: Q56 shifted), as
// floor((f - 1/2)^2 / 2) etc. in Q58 times 2^k, k >= 1.  One square: (f -+ 1/2)^2
// = f^2 -+ f + 1/4, whose last two terms are whole units, so the floors are the
// separate squares'.
FX_HD void tsc_weights_q58(int64_t f61, int k, V w[3]) {
  const V f = sp(f61);
  const int64_t q = mad(f.h, f.h, mad(f.h + f.h, f.l, mad(f.l, f.l, 0) >> 32) >> 32);  // f^2
  const int64_t t = q + (1ll << 56), u = f61 >> 3;
  w[0] = sp((int64_t)((uint64_t)((t - u) & ~1ll) << (k - 1)));
  w[1] = sp((int64_t)((uint64_t)((3ll << 56) - q) << k));
  w[2] = sp((int64_t)((uint64_t)((t + u) & ~1ll) << (k - 1)));
}

// base + k v for a small integer k.
FX_HD int64_t kmad(int k, V v, int64_t base) {
  const int64_t r = mad(v.l, k, base);
  return r + (int64_t)((uint64_t)((uint32_t)v.h * (uint32_t)k) << 32);
}

// |hi word| <= lim, as the check of a magnitude below lim 2^32.
FX_HD bool within(int64_t v, int lim) {
  const int h = (int)(v >> 32);
  return (h <= lim) & (h >= -lim);
}

// floor(log2 |v|) of a normal number, -100000 of zero or a subnormal.
FX_HD int exp_of(double v) {
  const int e = (int)(sf::bits(v) >> 52) & 0x7FF;
  return e == 0 ? -100000 : e - 1023;
}

// v 2^F rounded to the nearest integer; false when it reaches 2^62.
FX_HD bool fixc(double v, int F, int64_t* out) {
  const uint64_t u = sf::bits(v);
  const int e = (int)(u >> 52) & 0x7FF;
  *out = 0;
  if (e == 0) return true;
  const int sh = e - 1075 + F;
  if (sh > 10) return false;  // also infinities and NaN for any F >= -900
  uint64_t m = (u & ((1ull << 52) - 1)) | (1ull << 52);
  if (sh >= 0)
    m <<= sh;
  else
    m = sh < -60 ? 0 : (m + (1ull << (-sh - 1))) >> -sh;
  *out = (u >> 63) ? -(int64_t)m : (int64_t)m;
  return m < (1ull << 62);
}

FX_HD bool fixv(double v, int F, V* out) {
  int64_t t;
  const bool ok = fixc(v, F, &t);
  *out = sp(t);
  return ok;
}

// x 2^S to the nearest integer and back, by the conversion instructions (the
// power of two joins the exponent): the FP64 pipe is otherwise idle in the
// fixed-point pass.
FX_HD int64_t cvt_to(double x, int S) {
#ifdef __CUDA_ARCH__
  return __double2ll_rn(__hiloint2double(__double2hiint(x) + (S << 20), __double2loint(x)));
#else
  return (int64_t)std::llrint(sf::from_bits(sf::bits(x) + ((uint64_t)(int64_t)S << 52)));
#endif
}
FX_HD double cvt_from(int64_t v, int S) {
#ifdef __CUDA_ARCH__
  const double d = __ll2double_rn(v);
  const int h = __double2hiint(d);
  return __hiloint2double(h == 0 ? 0 : h - (S << 20), __double2loint(d));
#else
  const uint64_t u = sf::bits((double)v);
  return sf::from_bits(u == 0 ? 0 : u - ((uint64_t)(int64_t)S << 52));
#endif
}

// x 2^S truncated, for |x| 2^S < 2^62 (false otherwise); of the host check.
FX_HD bool to_fix(double x, int S, int64_t* out) {
  const uint64_t u = sf::bits(x);
  int r = 1085 - S - ((int)(u >> 52) & 0x7FF);
  const bool ok = r >= 1;
  r = r < 1 ? 1 : (r > 63 ? 63 : r);
  const uint64_t m = ((u & ((1ull << 52) - 1)) | (1ull << 52)) << 10;
  const int64_t t = (int64_t)(m >> r), s = (int64_t)u >> 63;
  *out = (t ^ s) - s;
  return ok;
}

// v 2^-S rounded to the nearest double (half away from zero).
FX_HD double from_fix(int64_t v, int S) {
  const uint64_t s = (uint64_t)v & 0x8000000000000000ull;
  const uint64_t a = v < 0 ? 0ull - (uint64_t)v : (uint64_t)v;
  if (a == 0) return 0.0;
  const int lz = sf::clz64(a);
  const uint64_t n = a << lz;
  const uint64_t m = (n >> 11) + ((n >> 10) & 1ull);
  return sf::from_bits((((uint64_t)(1085 - lz - S)) << 52) + m + s);
}

// knl = 1/(1+dp_p) in [3/4, 3/2): (knl - 1) 2^64, exact.
FX_HD int64_t kappa_of(double knl) {
  const uint64_t u = sf::bits(knl);
  const uint64_t m = (u & ((1ull << 52) - 1)) | (1ull << 52);
  return (int64_t)(m << (((int)(u >> 52) & 0x7FF) - 1011));
}

// ---------------------------------------------------------------------
// scales of one pass
// ---------------------------------------------------------------------
struct Scales {
  int x, p, d, k;  // Sx, Sp, Sd; dp_p in units of 2^-k (k >= 64)
};

static const int kMaxOps = 32;
static const int kNC = 10;
// The changes of z that hang on dp_p alone (terms of dp_p, e and q below) add
// up over the maps from the start, or from a wrap, to the next wrap: their
// constants are kZ0.. of a start's entry and of a wrap's.
static const int kZ0 = 2;

// A map's constants.  The coefficients x <- p and p <- x may exceed 1 in the
// units' ratio: k holds their nearest integers, c the rest.
struct alignas(16) Op {
  int code, i0, i1, bad;
  int k[4];
  V c[kNC];
};

// Bounds of |x|, |y| and |xp|, |yp| along the segment, and what its maps ask
// of the scales.
struct Bounds {
  float x, p;       // current bounds
  float dp;         // bound of |dp_p|
  float xp, px;     // largest coefficients x <- p and p <- x
  int bad;
};

// Typical magnitudes of |x|, |xp|, |y|, |yp|, each by itself: the larger of a
// map's terms, from below.
struct Typical {
  float x, p, y, r;
};

FX_HD float fmaxf_(float a, float b) { return a > b ? a : b; }

// Whether the map has a fixed-point form.
FX_HD bool supported(const DevOp& o) {
  switch (o.code) {
    case ORBIT_OP_DRIFT: case ORBIT_OP_QUAD1: case ORBIT_OP_QUAD2: case ORBIT_OP_BEND2: case ORBIT_OP_QFRIN:
    case ORBIT_OP_QFROUT: case ORBIT_OP_BEND1: case ORBIT_OP_BEND3: case ORBIT_OP_BEND4: case ORBIT_OP_BFRIN:
    case ORBIT_OP_BFROUT: case ORBIT_OP_WRAP:
      return true;
    case ORBIT_OP_MULTP:
      return o.i0 >= 0 && o.i0 <= 3;
    case ORBIT_OP_MPFRIN: case ORBIT_OP_MPFROUT:
      return o.i0 >= 1 && o.i0 <= 3;
    case ORBIT_OP_KICK:
      return o.c[2] == 0.;
    default:
      return false;
  }
}

// The map changes x or y.
FX_HD bool moves_x(const DevOp& o) {
  return o.code != ORBIT_OP_MULTP && o.code != ORBIT_OP_KICK && o.code != ORBIT_OP_WRAP;
}

// The start's entry of a segment's maps.
static const int kStart = -1;

// The constants of dp_p, e and q in the map's change of z.
inline void z_terms(const DevOp& o, double g2, double v[3]) {
  if (o.code == ORBIT_OP_QUAD1) v[0] += o.c[8];
  if (o.code == ORBIT_OP_BEND1) v[0] += o.c[8];
  if (o.code == ORBIT_OP_DRIFT) v[1] -= o.c[0] * g2;
  if (o.code == ORBIT_OP_QUAD2 || o.code == ORBIT_OP_BEND2) v[2] -= o.c[0] * g2;
}

// The map's bounds and scaled constants (host, once per compiled program);
// g2 = 1/gamma^2.
inline void compile_fixed(DevOp& o, double g2) {
  auto up = [](double a) { return (float)(std::fabs(a) * 1.0001); };
  auto ups = [](double a) { return (float)(a * 1.0001); };
  const double* c = o.c;
  std::memset(o.f, 0, sizeof(o.f));
  std::memset(o.v, 0, sizeof(o.v));
  float* f = o.f;
  double* v = o.v;
  switch (o.code) {
    case ORBIT_OP_DRIFT: case ORBIT_OP_QUAD2: case ORBIT_OP_BEND2:
      f[0] = up(c[0]);
      v[0] = c[0];
      v[1] = 0.5 * c[0];
      break;
    case ORBIT_OP_QUAD1:
      for (int i = 0; i < 8; i += 4) {  // the planes
        f[i] = ups(c[i] - 1.0);
        f[i + 1] = up(c[i + 1]);
        f[i + 2] = up(c[i + 2]);
        f[i + 3] = ups(c[i + 3] - 1.0);
      }
      for (int i = 0; i < 8; ++i) v[i] = c[i];
      v[0] -= 1.0;
      v[3] -= 1.0;
      v[4] -= 1.0;
      v[7] -= 1.0;
      break;
    case ORBIT_OP_QFRIN: case ORBIT_OP_QFROUT:
      f[0] = up(c[0]);
      v[0] = c[0];
      v[1] = c[1];
      v[2] = 1.0;
      break;
    case ORBIT_OP_BEND1:
      f[0] = ups(c[0] - 1.0);
      f[1] = up(c[1]);
      f[2] = up(c[2]);
      f[3] = up(c[3]);
      f[4] = ups(c[4] - 1.0);
      f[5] = up(c[5]);
      f[6] = up(c[9]);
      for (int i = 0; i < 6; ++i) v[i] = c[i];
      v[0] -= 1.0;
      v[4] -= 1.0;
      v[6] = c[9];
      for (int i = 6; i < 8; ++i) v[i + 1] = c[i];
      break;
    case ORBIT_OP_BEND3:
      f[0] = up(c[0]);
      v[0] = v[3] = 0.5 * c[0];
      v[1] = 0.5 * c[0] * g2;
      v[2] = c[0];
      v[4] = c[0] * g2;
      break;
    case ORBIT_OP_BEND4:
      f[0] = up(c[0]);
      v[0] = v[1] = 0.5 * c[0];
      break;
    case ORBIT_OP_BFRIN: case ORBIT_OP_BFROUT:
      f[0] = up(c[0]);
      f[1] = up(c[1]);
      v[0] = v[2] = c[0];
      v[1] = c[1];
      break;
    case ORBIT_OP_MULTP:
      f[0] = up(c[0]);
      f[1] = o.i1 ? 1.f : 0.f;
      v[0] = c[0];
      break;
    case ORBIT_OP_MPFRIN: case ORBIT_OP_MPFROUT:
      f[0] = up(c[0]) + up(c[1]);
      f[1] = (float)c[5];
      v[0] = c[0] != 0.0 ? c[0] : c[1];  // the kterm is real or imaginary
      v[2] = 1.0;
      o.i2 = c[0] != 0.0 ? 0 : 1;
      break;
    case ORBIT_OP_KICK:
      f[0] = up(c[0]);
      f[1] = up(c[1]);
      v[0] = c[0];
      v[1] = c[1];
      break;
    case ORBIT_OP_WRAP:
      v[0] = c[0];
      v[1] = c[1];
      break;
    default:
      break;
  }
}

// A segment's maps ops[1..n]: fills the start's entry ops[0] and the wraps'
// z sums.
inline void compile_segment(DevOp* ops, int n, double g2) {
  std::memset(&ops[0], 0, sizeof(DevOp));
  ops[0].code = kStart;
  for (int k = 1; k <= n; ++k) compile_fixed(ops[k], g2);
  double v[3] = {0.0, 0.0, 0.0};
  for (int k = n; k >= 0; --k) {
    z_terms(ops[k], g2, v);
    if (k == 0 || ops[k].code == ORBIT_OP_WRAP)
      for (int i = 0; i < 3; ++i) {
        ops[k].v[kZ0 + i] = v[i];
        v[i] = 0.0;
      }
  }
}

// Passes the bounds through one map of code `code`, pole i0 and f.
FX_HD void bound_op(int code, int i0, const float* f, Bounds& b) {
  const float kb = 1.0f + 1.2f * b.dp;  // |1/(1+dp_p)|
  const float x = b.x, p = b.p;
  switch (code) {
    case ORBIT_OP_DRIFT:
      b.x = x + kb * f[0] * p;
      b.xp = fmaxf_(b.xp, f[0]);
      break;
    case ORBIT_OP_QUAD1: {
      const float xp = fmaxf_(f[1], f[5]), px = fmaxf_(f[2], f[6]);
      b.x = x * (1.0f + fmaxf_(fabsf(f[0]), fabsf(f[4]))) + xp * p;
      b.p = p * (1.0f + fmaxf_(fabsf(f[3]), fabsf(f[7]))) + px * x;
      b.xp = fmaxf_(b.xp, xp);
      b.px = fmaxf_(b.px, px);
      break;
    }
    case ORBIT_OP_QUAD2:
    case ORBIT_OP_BEND2:
      b.x = x + kb * b.dp * f[0] * p;
      b.xp = fmaxf_(b.xp, f[0]);
      break;
    case ORBIT_OP_QFRIN:
    case ORBIT_OP_QFROUT:
      if (!(f[0] * kb * 2.0f * x * x <= 0x1p-7f)) b.bad = 1;
      b.x = x * 1.01f;
      b.p = p * 1.02f;
      break;
    case ORBIT_OP_BEND1:
      b.x = fmaxf_(x * (1.0f + fabsf(f[0])) + f[1] * p + f[2] * b.dp, x + f[6] * p);
      b.p = p * (1.0f + fabsf(f[4])) + f[3] * x + f[5] * b.dp;
      b.xp = fmaxf_(b.xp, fmaxf_(f[1], f[6]));
      b.px = fmaxf_(b.px, f[3]);
      break;
    case ORBIT_OP_BEND3:
      b.p = p + f[0] * (kb * p * p + b.dp * b.dp);
      b.x = x * (1.0f + f[0] * kb * p);
      break;
    case ORBIT_OP_BEND4:
      if (!(f[0] * kb * p <= 0x1p-8f)) b.bad = 1;
      b.x = x * 1.01f;
      b.p = p * 1.01f;
      break;
    case ORBIT_OP_BFRIN:
    case ORBIT_OP_BFROUT:
      b.x = x * (1.0f + f[0] * kb * x);
      b.p = p * (1.0f + f[1] * kb * x);
      break;
    case ORBIT_OP_MULTP: {
      float z = 1.0f;
      for (int q = 0; q < i0; ++q) z *= 1.4143f * x;
      b.p = p + f[0] * z;
      if (i0 == 1) b.px = fmaxf_(b.px, f[0]);
      break;
    }
    case ORBIT_OP_MPFRIN:
    case ORBIT_OP_MPFROUT: {
      float z = 1.4143f * x;
      for (int q = 0; q < i0; ++q) z *= 1.4143f * x;
      if (!(f[0] * kb * 2.0f * f[1] * z <= 0x1p-7f)) b.bad = 1;
      b.x = x * 1.01f;
      b.p = p * 1.02f;
      break;
    }
    case ORBIT_OP_KICK:
      b.p = p + fmaxf_(f[0], f[1]);
      break;
    default:
      break;
  }
}

// The same for the typical magnitudes.
FX_HD void typical_op(int code, int i0, const float* f, Typical& t) {
  const Typical o = t;
  switch (code) {
    case ORBIT_OP_DRIFT:
      t.x = fmaxf_(o.x, f[0] * o.p);
      t.y = fmaxf_(o.y, f[0] * o.r);
      break;
    case ORBIT_OP_QUAD1:
      t.x = fmaxf_(o.x * fabsf(1.0f + f[0]), f[1] * o.p);
      t.p = fmaxf_(o.p * fabsf(1.0f + f[3]), f[2] * o.x);
      t.y = fmaxf_(o.y * fabsf(1.0f + f[4]), f[5] * o.r);
      t.r = fmaxf_(o.r * fabsf(1.0f + f[7]), f[6] * o.y);
      break;
    case ORBIT_OP_BEND1:
      t.x = fmaxf_(o.x * fabsf(1.0f + f[0]), f[1] * o.p);
      t.p = fmaxf_(o.p * fabsf(1.0f + f[4]), f[3] * o.x);
      t.y = fmaxf_(o.y, f[6] * o.r);
      break;
    case ORBIT_OP_MULTP: {
      float a = 1.0f, b = 0.0f;  // |z^n|'s parts
      if (i0 == 1) a = o.x, b = o.y;
      if (i0 == 2) a = fmaxf_(o.x * o.x, o.y * o.y), b = 2.0f * o.x * o.y;
      if (i0 == 3) a = o.x * fmaxf_(o.x * o.x, 3.0f * o.y * o.y), b = o.y * fmaxf_(o.y * o.y, 3.0f * o.x * o.x);
      t.p = fmaxf_(o.p, f[0] * (f[1] != 0.0f ? b : a));
      t.r = fmaxf_(o.r, f[0] * (f[1] != 0.0f ? a : b));
      break;
    }
    case ORBIT_OP_KICK:
      t.p = fmaxf_(o.p, f[0]);
      t.r = fmaxf_(o.r, f[1]);
      break;
    default:
      break;
  }
}

// An integer above log2 f of a positive float.
FX_HD int exp_above(float f) {
  if (!(f > 0.0f)) return -200;
  if (!(f < 1e30f)) return 200;
  return (int)(sf::fbits(f) >> 23) - 126;
}

// v 2^(F - 64) as an integer and a fraction in [-1/2, 1/2) (units 2^-64);
// false when the integer exceeds 8.
FX_HD bool fixk(double v, int F, V* out, int* k) {
  const uint64_t u = sf::bits(v);
  const int e = (int)(u >> 52) & 0x7FF;
  *k = 0;
  out->h = out->l = 0;
  if (e == 0) return true;
  if (e + F - 64 >= 1023 + 3) return false;
  if (e + F - 64 < 1) return true;
  const double c = sf::from_bits(u + ((uint64_t)(int64_t)(F - 64) << 52));
  *k = (int)floor(c + 0.5);
  // the fraction is exact: to units of 2^-64 through its halves
  int64_t t;
  const bool ok = fixc(c - (double)*k, 62, &t);
  *out = sp((int64_t)((uint64_t)t << 2));
  if (e + F - 64 < 1023 - 8) {  // small: all of its bits
    const bool small = fixc(v, F, &t);
    *out = sp(t);
    return small;
  }
  return ok;
}

// Sx, Sp and k from the bounds after the last map: the finest units, or coarser
// ones of the coordinate whose coefficients would not fit beside the other's;
// false when the maps mix x and p too strongly for any.
FX_HD bool choose_scales(const Bounds& b, Scales& s) {
  if (b.bad || !(b.x > 0.0f) || !(b.p > 0.0f) || !(b.x < 1e6f) || !(b.p < 1e3f) || !(b.dp < 0.15f)) return false;
  s.x = 61 - exp_above(b.x);
  s.p = 61 - exp_above(b.p);
  const int xp = exp_above(b.xp), px = exp_above(b.px);
  if (px + s.p - s.x > 3) s.p = 3 + s.x - px;
  if (xp + s.x - s.p > 3) s.x = 3 + s.p - xp;
  const int k = 61 - exp_above(b.dp * 1.2f);
  s.k = k < 64 ? 64 : (k > 80 ? 80 : k);
  return s.x <= 100 && s.p <= 100 && xp + s.x - s.p <= 3 && px + s.p - s.x <= 3;
}

// The scales suit the typical magnitudes after the last map.
FX_HD bool fine_enough(const Typical& t, const Scales& s) {
  const float x = t.x < t.y ? t.x : t.y, p = t.p < t.r ? t.p : t.r;
  return exp_above(x) + s.x > 53 && exp_above(p) + s.p > 53;
}

// Left shift of z^n before the multipole kick's product.
FX_HD int zshift(int n) { return n < 2 ? 0 : 2 * (n - 1); }

// The constants of one map.  With pick_d: returns the largest Sd at which the
// map's z constants stay below 2^58 (so that the sum of up to 32 maps'
// changes stays below 2^61); otherwise fills out.c and out.bad.
FX_HD int consts_op(const DevOp& o, const Scales& s, Op& out, bool pick_d) {
  int md = 80;  // largest Sd
  out.code = o.code;
  out.i0 = o.i0;
  out.i1 = o.i1;
  out.bad = 0;
  auto put = [&](int i, int F) {
    if (!pick_d && !fixv(o.v[i], F, &out.c[i])) out.bad = 1;
  };
  auto putk = [&](int i, int q, int F) {
    if (!pick_d && !fixk(o.v[i], F, &out.c[i], &out.k[q])) out.bad = 1;
  };
  auto putz = [&](int i, int F) {  // in units of 2^-Sd
    if (pick_d) {
      const int e = 57 - exp_of(o.v[i]) - F;
      if (e < md) md = e;
    } else if (!fixv(o.v[i], s.d + F, &out.c[i])) {
      out.bad = 1;
    }
  };
  const int xp = s.x - s.p + 64, px = s.p - s.x + 64;
  switch (o.code) {
    case ORBIT_OP_DRIFT:
    case ORBIT_OP_QUAD2:
    case ORBIT_OP_BEND2:
      putk(0, 0, xp);
      putz(1, 128 - 2 * s.p);
      break;
    case ORBIT_OP_QUAD1:
      put(0, 64);
      putk(1, 0, xp);
      putk(2, 1, px);
      put(3, 64);
      put(4, 64);
      putk(5, 2, xp);
      putk(6, 3, px);
      put(7, 64);
      break;
    case ORBIT_OP_QFRIN:
    case ORBIT_OP_QFROUT:
      put(0, 190 - 2 * s.x);
      put(1, 190 - 2 * s.x);
      putz(2, 128 - s.p - s.x);
      break;
    case ORBIT_OP_BEND1:
      put(0, 64);
      putk(1, 0, xp);
      put(2, s.x - s.k + 64);
      putk(3, 1, px);
      put(4, 64);
      put(5, s.p - s.k + 64);
      putk(6, 2, xp);
      putz(7, 64 - s.x);
      putz(8, 64 - s.p);
      break;
    case ORBIT_OP_BEND3:
      put(0, 128 - s.p);
      put(1, s.p - s.k + 64);
      put(2, 128 - s.p);
      putz(3, 192 - 2 * s.p - s.x);
      putz(4, 128 - s.k - s.x);
      break;
    case ORBIT_OP_BEND4:
      put(0, 128 - s.p);
      putz(1, 192 - 2 * s.p - s.x);
      break;
    case ORBIT_OP_BFRIN:
    case ORBIT_OP_BFROUT:
      put(0, 128 - s.x);
      put(1, 128 - s.x);
      putz(2, 192 - s.p - 2 * s.x);
      break;
    case ORBIT_OP_MULTP:
      if (o.i0 == 1) putk(0, 0, px);
      else put(0, o.i0 == 0 ? s.p : s.p + 64 - (o.i0 * s.x - 64 * (o.i0 - 1)) - zshift(o.i0));
      break;
    case ORBIT_OP_MPFRIN:
    case ORBIT_OP_MPFROUT:
      put(0, 128 - ((o.i0 + 1) * s.x - 64 * o.i0));
      out.i1 = o.i2;
      putz(2, 128 - s.p - s.x);
      break;
    case ORBIT_OP_KICK:
      put(0, s.p);
      put(1, s.p);
      break;
    case ORBIT_OP_WRAP:
    case kStart:
      for (int i = kZ0; i < kZ0 + 3; ++i) putz(i, 64 - s.k);
      // a wrap's L and L/2 as the doubles' bits
      for (int i = 0; i < 2; ++i) {
        const uint64_t u = sf::bits(o.v[i]);
        out.c[i].h = (int)(u >> 32);
        out.c[i].l = (int)(uint32_t)u;
      }
      break;
    default:
      break;
  }
  return md;
}

// ---------------------------------------------------------------------
// one particle
// ---------------------------------------------------------------------
struct Part {
  int64_t x, p, y, r;  // x, xp, y, yp
  int64_t d;           // change of z since the start or the last wrap
  V kap;               // 1/(1+dp_p) - 1, units 2^-64
  V dp, e, q;          // dp_p, kap + kap^2/2 and kap^2/2 - kap dp_p, units 2^-k
  double z;
};

// kap, dp_p and the two combinations the z terms of drift and quad2 share;
// dpf = dp_p in units of 2^-k.
FX_HD void part_init(Part& t, int64_t kap, int64_t dpf, int k) {
  t.kap = sp(kap);
  t.dp = sp(dpf);
  const int64_t ks = kap << (k - 64);
  const int64_t h = mul(t.kap, sp(ks)) >> 1;
  t.e = sp(ks + h);
  t.q = sp(h - mul(t.kap, t.dp));
}

// (x + i y)^n for n = 1..3, in units of 2^-(n Sx - 64 (n - 1)).
FX_HD void zpow(int n, V x, V y, int64_t xr, int64_t yr, int64_t* zr, int64_t* zi) {
  *zr = xr;
  *zi = yr;
  for (int q = 1; q < n; ++q) {
    const V a = sp(*zr), b = sp(*zi);
    *zr = mul2s(a, x, b, y);
    *zi = mul2(a, y, b, x);
  }
}

// Starts the sum of the changes of z.
FX_HD void start_z(Part& t, const Op& o) { t.d = mul3(o.c[kZ0], t.dp, o.c[kZ0 + 1], t.e, o.c[kZ0 + 2], t.q); }

// ops[0] is the start's entry, the n maps follow.
FX_HD void apply(Part& t, const Op* ops, int n, const Scales& s) {
  start_z(t, ops[0]);
  for (int k = 1; k <= n; ++k) {
    const Op& o = ops[k];
    const V* c = o.c;
    switch (o.code) {
      case ORBIT_OP_DRIFT: {
        const V p = sp(t.p), r = sp(t.r);
        const V p1 = sp(mul(t.kap, p, t.p)), r1 = sp(mul(t.kap, r, t.r));
        t.x = mul(c[0], p1, kmad(o.k[0], p1, t.x));
        t.y = mul(c[0], r1, kmad(o.k[0], r1, t.y));
        const V q = sp(mul2(p1, p1, r1, r1));
        t.d -= mul(c[1], q);
        break;
      }
      case ORBIT_OP_QUAD1: {
        const V x = sp(t.x), p = sp(t.p), y = sp(t.y), r = sp(t.r);
        t.x = mul2(c[0], x, c[1], p, kmad(o.k[0], p, t.x));
        t.p = mul2(c[2], x, c[3], p, kmad(o.k[1], x, t.p));
        t.y = mul2(c[4], y, c[5], r, kmad(o.k[2], r, t.y));
        t.r = mul2(c[6], y, c[7], r, kmad(o.k[3], y, t.r));
        break;
      }
      case ORBIT_OP_QUAD2:
      case ORBIT_OP_BEND2: {
        const int64_t u = mul(t.kap, sp(t.p)), w = mul(t.kap, sp(t.r));
        const V p1 = sp(t.p + u), r1 = sp(t.r + w);
        const V uv = sp(u), wv = sp(w);
        t.x = mul(c[0], uv, kmad(o.k[0], uv, t.x));
        t.y = mul(c[0], wv, kmad(o.k[0], wv, t.y));
        const V q = sp(mul2(p1, p1, r1, r1));
        t.d -= mul(c[1], q);
        break;
      }
      case ORBIT_OP_QFRIN:
      case ORBIT_OP_QFROUT: {
        const V x = sp(t.x), p = sp(t.p), y = sp(t.y), r = sp(t.r);
        const int64_t x2 = mul(x, x) << 2, y2 = mul(y, y) << 2, xy = mul(x, y) << 2;
        const V k4 = sp(mul(t.kap, c[0], join(c[0]))), k12 = sp(mul(t.kap, c[1], join(c[1])));
        const V kr = sp(mul(k4, sp(x2 + y2))), kxy = sp(2 * mul(k4, sp(xy)));
        const V tt = sp(mul(k4, sp(x2 - y2)));
        const int64_t u = mul(tt, tt);  // 1/(1-u) = (1 + u)(1 + u^2), u < 2^-16
        const V uu = sp(u);
        const int64_t u2 = mul(uu, uu);
        const V w = sp(mul(uu, sp(u2), u + u2));
        const int64_t np = mul2s(kxy, r, kr, p, t.p), nr = mul2s(kr, r, kxy, p, t.r);
        const int64_t dx = mul(sp(mul(k12, sp(x2 + 3 * y2))), x), dy = mul(sp(mul(k12, sp(y2 + 3 * x2))), y);
        int64_t q = mul2s(p, sp(dx), r, sp(dy));
        q = mul(t.kap, sp(q), q);
        t.d = mul(c[2], sp(q), t.d);
        t.p = mul(w, sp(np), np);
        t.r = mul(w, sp(nr), nr);
        t.x += dx;
        t.y -= dy;
        break;
      }
      case ORBIT_OP_BEND1: {
        const V x = sp(t.x), p = sp(t.p), r = sp(t.r);
        t.d = mul2(c[7], x, c[8], p, t.d);
        t.x = mul2(c[0], x, c[1], p, mul(c[2], t.dp, kmad(o.k[0], p, t.x)));
        t.p = mul2(c[3], x, c[4], p, mul(c[5], t.dp, kmad(o.k[1], x, t.p)));
        t.y = mul(c[6], r, kmad(o.k[2], r, t.y));
        break;
      }
      case ORBIT_OP_BEND3: {
        const V r = sp(t.r), x = sp(t.x);
        const V r1 = sp(mul(t.kap, r, t.r));
        const V kd = sp(mul(t.kap, t.dp));
        t.p = mul2s(c[1], kd, c[0], sp(mul(r1, r)), t.p);
        t.y = mul(c[2], sp(mul(r1, x)), t.y);
        t.d -= mul2(c[3], sp(mul(sp(mul(r1, r1)), x)), c[4], sp(mul(t.e, x)));
        break;
      }
      case ORBIT_OP_BEND4: {
        const V p = sp(t.p);
        const V p1 = sp(mul(t.kap, p, t.p));
        const V al = sp(mul(c[0], p1));  // 1 + al = 1 + KNL xp theta / 2, |al| < 2^-9
        const int64_t a0 = join(al);
        const int64_t x1 = mul(al, sp(t.x), t.x);
        t.x = mul(al, sp(x1), x1);
        int64_t w = a0;  // al / (1 + al) by w <- al - al w
#pragma unroll
        for (int q = 0; q < 5; ++q) w = a0 - mul(al, sp(w));
        t.p -= mul(sp(w), p);
        t.d -= mul(c[1], sp(mul(sp(mul(p1, p1)), sp(t.x))));
        break;
      }
      case ORBIT_OP_BFRIN:
      case ORBIT_OP_BFROUT: {
        const V y = sp(t.y), p = sp(t.p);
        const int64_t y2 = mul(y, y);
        const V k2 = sp(mul(t.kap, sp(y2), y2)), p1 = sp(mul(t.kap, p, t.p));
        t.x = mul(c[0], k2, t.x);
        t.r -= mul(c[1], sp(mul(p1, y)));
        t.d = mul(c[2], sp(mul(p1, k2)), t.d);
        break;
      }
      case ORBIT_OP_MULTP: {
        if (o.i0 == 0) {  // z^0 = 1
          if (o.i1) t.r += join(c[0]);
          else t.p -= join(c[0]);
          break;
        }
        int64_t zr, zi;
        zpow(o.i0, sp(t.x), sp(t.y), t.x, t.y, &zr, &zi);
        const int za = zshift(o.i0), q = o.i0 == 1 ? o.k[0] : 0;
        const int64_t a = mul(c[0], sp(zr << za), kmad(q, sp(zr), 0)), b = mul(c[0], sp(zi << za), kmad(q, sp(zi), 0));
        t.p = o.i1 ? t.p + b : t.p - a;
        t.r = o.i1 ? t.r + a : t.r + b;
        break;
      }
      case ORBIT_OP_MPFRIN:
      case ORBIT_OP_MPFROUT: {
        // as multpfringe_body: kt (A + i B) = kterm z^(l-1), l = i0 + 1; an
        // imaginary kterm turns z^(l-1) by a right angle
        const int l = o.i0 + 1;
        const V x = sp(t.x), p = sp(t.p), y = sp(t.y), r = sp(t.r);
        int64_t zr, zi;
        zpow(o.i0, x, y, t.x, t.y, &zr, &zi);
        const V A = sp(o.i1 ? -zi : zr), B = sp(o.i1 ? zr : zi);
        const int64_t C = mul2s(A, x, B, y), D = mul2(A, y, B, x);
        const V lC = sp(l * C), lD = sp((l + 2) * D);
        const V kt = sp(mul(t.kap, c[0], join(c[0])));
        const V fx = sp(mul2(lC, x, lD, y)), fy = sp(mul2s(lC, y, lD, x));
        const int64_t Ay = mul(A, y), Bx = mul(B, x);
        const V u = sp(mul(kt, sp((int64_t)(l * (l + 1)) * mul2(A, x, B, y))));
        const V m21 = sp(mul(kt, sp((int64_t)((l + 1) * (l - 2)) * Bx - (int64_t)((l + 1) * (l + 2)) * Ay)));
        const V m12 = sp(mul(kt, sp((int64_t)((l + 1) * (l + 2)) * Bx - (int64_t)((l + 1) * (l - 2)) * Ay)));
        const int64_t e = mul2(u, u, m12, m21);
        const V w = sp(e + mul(sp(e), sp(e)));  // 1/(1-e) = 1 + e + e^2
        const int64_t np = mul2s(u, p, m12, r, t.p), nr = t.r - mul2(u, r, m21, p);
        t.p = mul(w, sp(np), np);
        t.r = mul(w, sp(nr), nr);
        const int64_t dx = mul(kt, fx), dy = mul(kt, fy);
        t.x -= dx;
        t.y -= dy;
        int64_t q = mul2(sp(t.p), sp(dx), sp(t.r), sp(dy));
        q = mul(t.kap, sp(q), q);
        t.d -= mul(c[2], sp(q));
        break;
      }
      case ORBIT_OP_KICK:
        t.p += join(c[0]);
        t.r += join(c[1]);
        break;
      case ORBIT_OP_WRAP: {
        t.z += from_fix(t.d, s.d);
        const double L = sf::from_bits(((uint64_t)(uint32_t)c[0].h << 32) | (uint32_t)c[0].l);
        const double h = sf::from_bits(((uint64_t)(uint32_t)c[1].h << 32) | (uint32_t)c[1].l);
        if (t.z < -h) t.z += L;
        if (t.z > h) t.z -= L;
        start_z(t, o);
        break;
      }
      default:
        break;
    }
  }
}

}  // namespace fx
}  // namespace orbit
