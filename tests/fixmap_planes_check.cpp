// Host check of which beams the fixed-point maps (csrc/fixmap.cuh) take:
// Gaussian beams whose planes differ by up to five decades through segments of
// drifts, quadrupoles with fringes, sextupoles and bends.  Prints the segments
// with a fixed-point form that are taken and refused (fx::fine_enough), the largest ratio of the rms error of a
// coordinate to binary64's on the same particles, both against long double,
// over the segments taken; and of those of round beams the share taken, and of
// beams with planes three decades apart.
#include <algorithm>
#include <initializer_list>

#define main fixmap_check_main
#include "fixmap_check.cpp"
#undef main

int main(int argc, char** argv) {
  const int nseg = argc > 1 ? atoi(argv[1]) : 2000, np = 400;
  std::mt19937_64 g(argc > 2 ? atoi(argv[2]) : 1);
  auto U = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(g); };
  auto E = [&](double a, double b) { return std::exp(U(std::log(a), std::log(b))); };
  std::normal_distribution<double> N;
  const double g2 = 0.234;
  int taken = 0, refused = 0, round_n = 0, round_ok = 0, flat_n = 0, flat_ok = 0;
  double worst = 0.0;
  for (int q = 0; q < nseg; ++q) {
    const double sx = E(1e-4, 2e-2), sp = sx * E(0.05, 1.0), sd = E(1e-5, 3e-3);
    const double ry = q % 3 == 0 ? 1.0 : E(1e-5, 1.0), rp = q % 3 == 0 ? 1.0 : ry * E(0.3, 3.0);
    std::vector<DevOp> seg(1);
    auto add = [&](int code, std::initializer_list<double> c, int i0 = 0) {
      DevOp o;
      std::memset(&o, 0, sizeof(o));
      o.code = code;
      o.i0 = i0;
      std::copy(c.begin(), c.end(), o.c);
      seg.push_back(o);
    };
    const double k1 = U(-0.8, 0.8), s = std::sqrt(std::fabs(k1) + 1e-9);
    auto quad1 = [&](double l) {
      const double a = std::cos(s * l), b = std::sin(s * l), c = std::cosh(s * l), d = std::sinh(s * l);
      if (k1 > 0) add(ORBIT_OP_QUAD1, {a, b / s, -b * s, a, c, d / s, d * s, c, g2 * l});
      else add(ORBIT_OP_QUAD1, {c, d / s, d * s, c, a, b / s, -b * s, a, g2 * l});
    };
    switch (g() % 4) {
      case 0:
        add(ORBIT_OP_DRIFT, {E(0.1, 2.0)});
        break;
      case 1:
        add(ORBIT_OP_QFRIN, {k1 / 4, k1 / 12});
        quad1(0.25);
        add(ORBIT_OP_QUAD2, {0.5});
        quad1(0.25);
        add(ORBIT_OP_QFROUT, {-k1 / 4, -k1 / 12});
        add(ORBIT_OP_DRIFT, {E(0.1, 2.0)});
        break;
      case 2: {
        const double th = U(0.05, 0.15), rho = 1.0 / th, c = std::cos(th), d = std::sin(th);
        add(ORBIT_OP_MULTP, {U(-0.4, 0.4)}, 2);
        add(ORBIT_OP_DRIFT, {0.5});
        add(ORBIT_OP_BEND1, {c, rho * d, rho * (1 - c), -d / rho, c, d, -d, -rho * (1 - c), -(1 - g2) + rho * d, 1.0});
        add(ORBIT_OP_BEND2, {1.0});
        add(ORBIT_OP_BEND3, {th});
        add(ORBIT_OP_BEND4, {th});
        break;
      }
      default:
        add(ORBIT_OP_DRIFT, {1.0});
        quad1(0.25);
        add(ORBIT_OP_QUAD2, {0.25});
    }
    const int n = (int)seg.size() - 1;
    std::vector<P<double>> beam(np);
    double mx = 0, mp = 0, md = 0, e[4] = {0, 0, 0, 0};
    for (auto& b : beam) {
      b = {sx * N(g), sp * N(g), sx * ry * N(g), sp * rp * N(g), U(-5, 5), sd * N(g)};
      mx = std::max({mx, std::fabs(b.x), std::fabs(b.y)});
      mp = std::max({mp, std::fabs(b.p), std::fabs(b.r)});
      md = std::max(md, std::fabs(b.dp));
      const double v[4] = {b.x, b.p, b.y, b.r};
      for (int k = 0; k < 4; ++k) e[k] += std::floor(std::log2(std::fabs(v[k]))) / np;
    }
    fx::Typical t = {std::exp2((float)e[0]), std::exp2((float)e[1]), std::exp2((float)e[2]), std::exp2((float)e[3])};
    fx::Bounds b = {(float)mx * 1.001f, 1.25f * (float)mp, (float)md * 1.001f, 0.f, 0.f, 0};
    fx::compile_segment(seg.data(), n, g2);
    for (int k = 1; k <= n; ++k) {
      fx::bound_op(seg[k].code, seg[k].i0, seg[k].f, b);
      fx::typical_op(seg[k].code, seg[k].i0, seg[k].f, t);
    }
    fx::Scales sc;
    std::vector<fx::Op> fo(n + 1);
    bool ok = fx::choose_scales(b, sc);
    if (ok) {
      sc.d = 80;
      for (int k = 0; k <= n; ++k) sc.d = std::min(sc.d, fx::consts_op(seg[k], sc, fo[k], true));
      for (int k = 0; k <= n; ++k) { fx::consts_op(seg[k], sc, fo[k], false); ok = ok && !fo[k].bad; }
    }
    if (!ok) continue;  // the maps mix x and p too strongly for any beam
    ok = fx::fine_enough(t, sc);
    if (q % 3 == 0) { ++round_n; round_ok += ok; }
    if (ry < 1e-3) { ++flat_n; flat_ok += ok; }
    if (!ok) { ++refused; continue; }
    ++taken;
    double ef[4] = {0, 0, 0, 0}, ed[4] = {0, 0, 0, 0};
    for (auto& B : beam) {
      const double knl = 1.0 / (1.0 + B.dp);
      const L dp = 1.0L / (L)knl - 1.0L;
      auto fix = [](double v, int S) {  // the kernel's conversions: half a unit in, half an ulp back
        const int64_t f = fx::cvt_to(v, S);
        const double o = fx::cvt_from(f, S);
        if (std::fabs((L)f - std::ldexp((L)v, S)) > 0.5L ||
            std::fabs((L)o - std::ldexp((L)f, -S)) > std::fabs((L)o) * std::ldexp(1.0L, -53) * 1.0000001L) {
          std::printf("conversion off\n");
          std::exit(1);
        }
        return f;
      };
      fx::Part f;
      f.x = fix(B.x, sc.x); f.p = fix(B.p, sc.p); f.y = fix(B.y, sc.x); f.r = fix(B.r, sc.p); f.z = B.z;
      fx::part_init(f, fx::kappa_of(knl), fix((double)dp, sc.k), sc.k);
      P<L> T = {B.x, B.p, B.y, B.r, B.z, dp};
      P<double> D = {B.x, B.p, B.y, B.r, B.z, (double)dp};
      for (int k = 1; k <= n; ++k) { map<L>(T, seg[k], g2); map<double>(D, seg[k], g2); }
      fx::apply(f, fo.data(), n, sc);
      const double o[4] = {fx::cvt_from(f.x, sc.x), fx::cvt_from(f.p, sc.p), fx::cvt_from(f.y, sc.x), fx::cvt_from(f.r, sc.p)};
      const double d[4] = {D.x, D.p, D.y, D.r};
      const L w[4] = {T.x, T.p, T.y, T.r};
      for (int k = 0; k < 4; ++k) {
        ef[k] += (double)((o[k] - w[k]) * (o[k] - w[k]));
        ed[k] += (double)((d[k] - w[k]) * (d[k] - w[k]));
      }
    }
    for (int k = 0; k < 4; ++k)
      if (ed[k] > 0.0) worst = std::max(worst, std::sqrt(ef[k] / ed[k]));
  }
  std::printf("%d %d %.4f %.4f %.4f\n", taken, refused, worst, (double)round_ok / round_n, (double)flat_ok / flat_n);
  return 0;
}
