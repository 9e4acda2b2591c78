// Host check of the fixed-point maps (csrc/fixmap.cuh) against long double
// maps: random segments of maps over random beams.  Prints the numbers of
// segments and of those with a fixed-point form, then for the fixed-point
// maps and for the same maps in binary64 the largest and the rms error of x
// and of p in units of the segment's bound, and of z in metres.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "../py-orbit_gb300/csrc/fixmap.cuh"

using namespace orbit;
typedef long double L;

template <class T>
struct P {
  T x, p, y, r, z, dp;
};

// One map in type T.
template <class T>
static void map(P<T>& t, const DevOp& o, T g2) {
  const T k = T(1) / (T(1) + t.dp), x = t.x, p = t.p, y = t.y, r = t.r, d = t.dp;
  const double* c = o.c;
  switch (o.code) {
    case ORBIT_OP_DRIFT: {
      t.x += k * c[0] * p; t.y += k * c[0] * r;
      T f = (p * p + r * r + d * d * g2) / 2;
      t.z -= c[0] * (f * k - d * g2) * k;
      break;
    }
    case ORBIT_OP_QUAD1:
      t.x = c[0] * x + c[1] * p; t.p = c[2] * x + c[3] * p; t.y = c[4] * y + c[5] * r; t.r = c[6] * y + c[7] * r;
      t.z += d * c[8];
      break;
    case ORBIT_OP_QUAD2: case ORBIT_OP_BEND2: {
      t.x -= k * c[0] * d * p; t.y -= k * c[0] * d * r;
      T f = (p * p + r * r + d * d * g2) / 2;
      t.z -= c[0] * (f * k + d * d * g2) * k;
      break;
    }
    case ORBIT_OP_QFRIN: case ORBIT_OP_QFROUT: {
      T k4 = c[0] * k, k12 = c[1] * k, u = k4 * (x * x - y * y);
      u = 1 - u * u;
      t.p = (p - k4 * (x * x + y * y) * p + 2 * k4 * x * y * r) / u;
      t.r = (r + k4 * (x * x + y * y) * r - 2 * k4 * x * y * p) / u;
      T X = k12 * x * (x * x + 3 * y * y), Y = k12 * y * (y * y + 3 * x * x);
      t.x += X; t.y -= Y; t.z += k * (p * X - r * Y);
      break;
    }
    case ORBIT_OP_BEND1:
      t.x = c[0] * x + c[1] * p + c[2] * d; t.p = c[3] * x + c[4] * p + c[5] * d; t.y += c[9] * r;
      t.z += c[6] * x + c[7] * p + c[8] * d;
      break;
    case ORBIT_OP_BEND3: {
      T f = (r * r + d * d * g2) / 2;
      t.p -= f * k * c[0]; t.y += k * r * x * c[0];
      t.z -= c[0] * (f * k - d * g2) * k * x;
      break;
    }
    case ORBIT_OP_BEND4: {
      T a = 1 + k * p * c[0] / 2;
      t.x = x * a * a; t.p = p / a; t.z -= c[0] * (k * p) * (k * p) / 2 * t.x;
      break;
    }
    case ORBIT_OP_BFRIN: case ORBIT_OP_BFROUT:
      t.x += k * y * y * c[0]; t.r -= k * p * y * c[1]; t.z += k * k * p * y * y * c[0];
      break;
    case ORBIT_OP_MULTP: {
      T zr = 1, zi = 0;
      for (int q = 0; q < o.i0; ++q) { T s = zr * x - zi * y; zi = zr * y + zi * x; zr = s; }
      if (o.i1) { t.p += c[0] * zi; t.r += c[0] * zr; } else { t.p -= c[0] * zr; t.r += c[0] * zi; }
      break;
    }
    case ORBIT_OP_MPFRIN: case ORBIT_OP_MPFROUT: {
      T zr = 1, zi = 0, l = o.i0 + 1;
      for (int q = 0; q < o.i0; ++q) { T s = zr * x - zi * y; zi = zr * y + zi * x; zr = s; }
      T A = c[0] * zr - c[1] * zi, B = c[0] * zi + c[1] * zr, C = A * x - B * y, D = A * y + B * x;
      T fx = l * C * x + (l + 2) * D * y, fy = l * C * y - (l + 2) * D * x;
      T a = l * (l + 1) * (A * x + B * y) * k, b = ((l + 1) * (l + 2) * A * y - (l + 1) * (l - 2) * B * x) * k;
      T e = ((l + 1) * (l - 2) * A * y - (l + 1) * (l + 2) * B * x) * k;
      T m11 = 1 - a, m12 = -e, m21 = -b, m22 = 1 + a, det = m11 * m22 - m12 * m21;
      t.p = (m22 * p - m12 * r) / det; t.r = (m11 * r - m21 * p) / det;
      t.x -= fx * k; t.y -= fy * k; t.z -= (t.p * fx + t.r * fy) * k * k;
      break;
    }
    case ORBIT_OP_KICK: t.p += c[0]; t.r += c[1]; break;
    case ORBIT_OP_WRAP: if (t.z < -c[1]) t.z += c[0]; if (t.z > c[1]) t.z -= c[0]; break;
  }
}

// Largest and rms of a series.
struct Err {
  L big = 0, sq = 0;
  long n = 0;
  void add(L e) { e = std::fabs(e); big = std::max(big, e); sq += e * e; ++n; }
  void print() const { std::printf(" %.3Lg %.3Lg", big, n ? std::sqrt(sq / n) : 0.0L); }
};

int main(int argc, char** argv) {
  const int nseg = argc > 1 ? atoi(argv[1]) : 2000;
  std::mt19937_64 g(argc > 2 ? atoi(argv[2]) : 1);
  auto U = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(g); };
  auto E = [&](double a, double b) { return std::exp(U(std::log(a), std::log(b))); };
  const int codes[] = {ORBIT_OP_DRIFT, ORBIT_OP_QUAD1, ORBIT_OP_QUAD2, ORBIT_OP_QFRIN, ORBIT_OP_BEND1, ORBIT_OP_BEND3,
                       ORBIT_OP_BEND4, ORBIT_OP_BFRIN, ORBIT_OP_MULTP, ORBIT_OP_MPFRIN, ORBIT_OP_KICK, ORBIT_OP_WRAP};
  Err fxx, fxp, fxz, dbx, dbp, dbz;
  int fixed = 0;
  for (int q = 0; q < nseg; ++q) {
    const double g2 = U(0.05, 0.9), bx = E(1e-5, 5e-2), bp = bx * E(1e-3, 3.0), bd = E(1e-6, 0.1);
    std::vector<DevOp> ops;
    const int n = 1 + (int)(g() % 10);
    for (int k = 0; k < n; ++k) {
      DevOp o;
      std::memset(&o, 0, sizeof(o));
      // half the segments of one map only, so that each is exercised alone
      o.code = codes[(q % 2 ? (unsigned)(q / 2) : (unsigned)g()) % 12u];
      double* c = o.c;
      const double len = E(0.01, 3.0), k1 = U(-1.5, 1.5), th = U(-0.2, 0.2);
      switch (o.code) {
        case ORBIT_OP_QUAD1: {
          const double s = std::sqrt(std::fabs(k1) + 1e-9), l = len / 3;
          const double a[4] = {std::cos(s * l), std::sin(s * l) / s, -std::sin(s * l) * s, std::cos(s * l)};
          const double b[4] = {std::cosh(s * l), std::sinh(s * l) / s, std::sinh(s * l) * s, std::cosh(s * l)};
          for (int i = 0; i < 4; ++i) { c[i] = k1 > 0 ? a[i] : b[i]; c[4 + i] = k1 > 0 ? b[i] : a[i]; }
          c[8] = g2 * l;
          break;
        }
        case ORBIT_OP_QFRIN: c[0] = k1 / 4; c[1] = k1 / 12; break;
        case ORBIT_OP_BEND1: {
          const double rho = len / th, cx = std::cos(th), sx = std::sin(th);
          const double a[10] = {cx, rho * sx, rho * (1 - cx), -sx / rho, cx, sx, -sx, -rho * (1 - cx),
                                -(1 - g2) * len + rho * sx, len};
          for (int i = 0; i < 10; ++i) c[i] = a[i];
          break;
        }
        case ORBIT_OP_BEND3: case ORBIT_OP_BEND4: c[0] = th; break;
        case ORBIT_OP_BFRIN: c[1] = th / len; c[0] = c[1] / 2; break;
        case ORBIT_OP_MULTP: o.i0 = (int)(g() % 4); o.i1 = (int)(g() % 2); c[0] = U(-1, 1) * (o.i0 ? 1.0 : bp); break;
        case ORBIT_OP_MPFRIN: {
          o.i0 = 1 + (int)(g() % 3);
          const double kf = U(-3, 3) / (4.0 * std::tgamma(o.i0 + 3.0)), l = o.i0 + 1;
          c[g() % 2] = kf;
          c[2] = l; c[3] = l + 2; c[4] = l * (l + 1); c[5] = (l + 1) * (l + 2); c[6] = (l + 1) * (l - 2);
          break;
        }
        case ORBIT_OP_KICK: c[0] = U(-1, 1) * bp; c[1] = U(-1, 1) * bp; break;
        case ORBIT_OP_WRAP: c[0] = 10.0; c[1] = 5.0; break;
        default: c[0] = len;
      }
      ops.push_back(o);
    }
    fx::Bounds b = {(float)bx * 1.001f, (float)bp * 1.001f, (float)bd * 1.001f, 0.f, 0.f, 0};
    fx::Scales s;
    std::vector<fx::Op> fo(ops.size() + 1);
    bool ok = true;
    std::vector<DevOp> seg(1);
    seg.insert(seg.end(), ops.begin(), ops.end());
    fx::compile_segment(seg.data(), n, g2);
    for (int k = 1; k <= n; ++k) { ok = ok && fx::supported(seg[k]); fx::bound_op(seg[k].code, seg[k].i0, seg[k].f, b); }
    ok = ok && fx::choose_scales(b, s);
    if (!ok) continue;
    int md = 80;
    for (size_t k = 0; k < seg.size(); ++k) md = std::min(md, fx::consts_op(seg[k], s, fo[k], true));
    s.d = md;
    for (size_t k = 0; k < seg.size(); ++k) { fx::consts_op(seg[k], s, fo[k], false); ok = ok && !fo[k].bad; }
    if (!ok || s.d < 50) continue;
    ++fixed;
    for (int i = 0; i < 64; ++i) {
      // corners of the bound, zeros and the inside
      const double e[6] = {0.0, 1.0, -1.0, U(-1, 1), U(-1, 1), U(-1e-3, 1e-3)};
      const double x = bx * e[g() % 6], p = bp * e[g() % 6], y = bx * e[g() % 6], r = bp * e[g() % 6];
      const double z = U(-5, 5), dp = bd * e[g() % 6], knl = 1.0 / (1.0 + dp);
      P<L> t = {x, p, y, r, z, 1.0L / (L)knl - 1.0L};
      fx::Part f;
      int64_t dpf;
      bool in = fx::to_fix(x, s.x, &f.x) && fx::to_fix(p, s.p, &f.p) && fx::to_fix(y, s.x, &f.y) &&
                fx::to_fix(r, s.p, &f.r) && fx::to_fix((double)t.dp, s.k, &dpf);
      if (!in) { std::printf("conversion refused\n"); return 1; }
      if (i % 4 == 0) {  // low words of -2^31, which have no negative
        for (int64_t* v : {&f.x, &f.p, &f.y, &f.r}) *v = (*v & ~0xffffffffll) / 2 + 0x80000000ll;
        t.x = std::ldexp((L)f.x, -s.x); t.y = std::ldexp((L)f.y, -s.x);
        t.p = std::ldexp((L)f.p, -s.p); t.r = std::ldexp((L)f.r, -s.p);
      }
      f.z = z;
      fx::part_init(f, fx::kappa_of(knl), dpf, s.k);
      P<double> d = {(double)t.x, (double)t.p, (double)t.y, (double)t.r, z, (double)t.dp};
      for (auto& o : ops) { map<L>(t, o, g2); map<double>(d, o, g2); }
      fx::apply(f, fo.data(), n, s);
      auto wrapped = [](L e) { return std::fabs(e) > 5 ? std::fabs(e) - 10 : e; };  // the wrap's two sides
      fxx.add((std::ldexp((L)f.x, -s.x) - t.x) / b.x); fxx.add((std::ldexp((L)f.y, -s.x) - t.y) / b.x);
      fxp.add((std::ldexp((L)f.p, -s.p) - t.p) / b.p); fxp.add((std::ldexp((L)f.r, -s.p) - t.r) / b.p);
      fxz.add(wrapped((L)(f.z + fx::from_fix(f.d, s.d)) - t.z));
      dbx.add((d.x - t.x) / b.x); dbx.add((d.y - t.y) / b.x);
      dbp.add((d.p - t.p) / b.p); dbp.add((d.r - t.r) / b.p);
      dbz.add(wrapped(d.z - t.z));
      for (int64_t v : {f.x, f.p, f.y, f.r}) {  // conversions out: half an ulp
        const double o = fx::from_fix(v, s.x);
        if (std::fabs((L)o - std::ldexp((L)v, -s.x)) > std::fabs((L)o) * std::ldexp(1.0L, -53) * 1.0000001L) {
          std::printf("from_fix off\n");
          return 1;
        }
      }
    }
  }
  std::printf("%d %d", nseg, fixed);
  for (const Err* e : {&fxx, &fxp, &fxz, &dbx, &dbp, &dbz}) e->print();
  std::printf("\n");
  return 0;
}
