// The constants of the lattice pass that follows a kick: the kick's own, and
// the scales, bounds and map constants of the fixed-point pass.  They hang on
// the bunch's magnitudes, the grids and the line density only, all known
// before the potential, so one warp makes them beside the solve (prep_pass)
// and every block of the pass copies them; what hangs on max |phi| is added
// there (load_prep).  Made in the pass itself, by warp 0 of every block
// before its first particle, they took about 8 us of each pass.
#pragma once

#include "fixmap.cuh"
#include "sc_device.cuh"

namespace orbit {

struct FxGrid {      // t = x / step - min / step in units of 2^-F
  fx::V a;
  long long c;
  int F, lo, hi, half;  // high words: a quarter cell inside the edges, 1/2
};
struct alignas(16) FxPass {
  int ok;             // the pass runs in fixed point: its scales and maps fit
  int kick_ok;        // and so do the kick's constants
  int n;              // maps
  int check;          // some particles lie beyond the bounds
  fx::Scales s;
  int limx, limp, limd;  // high words of the bounds of |x|, |xp| and |dp_p| as doubles
  int limk;              // and of the kick in the pass's units
  FxGrid gx, gy;
  int ny, nz, j, limj;
  fx::V Cx, Cy;       // kick = (gradient lambda) C 2^j
  int ce;             // C is -factor / step over 2^(ce - 61)
  double az, cz;      // line density: z / dz - zmin / dz + 1/2, units 2^-Fz
  int Fz;
  alignas(16) fx::Op op[fx::kMaxOps];
};
struct alignas(16) PassPrep {
  KickConst k;
  KickFix kf;
  FxPass fx;
};

// The scales, the maps' constants and the grids' (one warp): nothing here hangs
// on the solve.
__device__ __forceinline__ void prep_maps(const PrepJob& J, const ScState* st, int nx, int ny, int nz) {
  const int lane = threadIdx.x & 31, nops = J.b - J.a;
  FxPass* f = &J.out->fx;
  // lane 0 the segment's start entry, lanes 1..nops its maps
  bool ok = nops < fx::kMaxOps && st->mag.pmax != 0u && !st->skip;
  const DevOp* o = J.ops + J.a - 1 + (lane <= nops ? lane : 0);
  const int code = lane <= nops ? o->code : 0, i0 = lane <= nops ? o->i0 : 0;
  float c[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) c[q] = lane <= nops ? o->f[q] : 0.f;
  // typical magnitudes of x, xp, y, yp: the geometric mean, in whole exponents,
  // of 256 particles spread over the bunch, of those that are not zero, which have
  // to be half of them.  (Sampled by the pass in its loop they cost 1 to 2 us of
  // every pass of 1e6 particles.)
  unsigned sum[4] = {0u, 0u, 0u, 0u};  // exponents from 2^-60, and the count (2^20)
  {
    unsigned hw[8][4];  // high words, every load in flight at once
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int i = (int)(((long long)(r * 32 + lane) * J.n) >> 8);
#pragma unroll
      for (int q = 0; q < 4; ++q) hw[r][q] = ok ? __ldcg(reinterpret_cast<const unsigned*>(J.c[q] + i) + 1) : 0u;
    }
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const unsigned e = hw[r][q] >> 20 & 0x7ffu;
        if (e != 0u) sum[q] += (1u << 20) + min(max(e, 963u), 1083u) - 963u;
      }
  }
  for (int q = 0; q < 4; ++q) sum[q] = __reduce_add_sync(0xffffffffu, sum[q]);
  // (lane q of every four takes coordinate q)
  const int lq = lane & 3;
  const unsigned sq = lq == 0 ? sum[0] : lq == 1 ? sum[1] : lq == 2 ? sum[2] : sum[3], cnt = sq >> 20;
  ok = ok && __reduce_min_sync(0xffffffffu, cnt) >= 128u;
  const float typ_q = exp2f(__fdividef((float)(sq & 0xfffffu), (float)max(cnt, 1u)) - 60.f);
  auto of = [](float v, int q) { return __shfl_sync(0xffffffffu, v, q); };
  fx::Typical ty = {of(typ_q, 0), of(typ_q, 1), of(typ_q, 2), of(typ_q, 3)};
  // bounds: the extent, or 24 times the larger plane's typical size (9 standard
  // deviations of a Gaussian) where a few particles lie further out.  16 made a
  // batch of tracked bunches, whose tails it cut, 1% slower, since one particle's
  // way through the FP64 routines takes 15 us; 50 leaves a beam with a halo too few
  // units
  const float xm = (float)st->mag.xmax * 1.0001f;
  const float pm = (float)__hiloint2double((int)st->mag.pmax, -1) * 1.0001f;
  const float dm = (float)__hiloint2double((int)st->mag.emax, -1) * fabsf((float)J.dp_p_coeff) * 1.0001f;
  const float x0 = fminf(xm, 24.f * fmaxf(ty.x, ty.y)), p0 = fminf(pm, 24.f * fmaxf(ty.p, ty.r)), d0 = fminf(dm, 0.124f);
  fx::Bounds bd = {x0, 1.25f * p0, d0, 0.f, 0.f, 0};
  if (ok) {
    for (int q = 1; q <= nops; ++q) {
      float g[8];
#pragma unroll
      for (int w = 0; w < 8; ++w) g[w] = __shfl_sync(0xffffffffu, c[w], q);
      const int cq = __shfl_sync(0xffffffffu, code, q), iq = __shfl_sync(0xffffffffu, i0, q);
      fx::bound_op(cq, iq, g, bd);
      fx::typical_op(cq, iq, g, ty);
    }
    fx::Scales s;
    ok = fx::choose_scales(bd, s);
    // a constant too large for the units of xp (a sextupole's, for a beam with
    // little slope) may fit coarser ones
    for (int t = 0; ok; ++t, --s.p) {
      ok = fx::fine_enough(ty, s);
      fx::Op out;
      out.bad = 0;
      int md = 80;
      if (ok && lane <= nops) md = fx::consts_op(*o, s, out, true);
      s.d = __reduce_min_sync(0xffffffffu, md);
      if (ok && lane <= nops) {
        fx::consts_op(*o, s, out, false);
        f->op[lane] = out;
      }
      const bool fits = __all_sync(0xffffffffu, ok && out.bad == 0 && s.d >= 50);
      if (fits) break;
      ok = ok && t < 2;
    }
    if (lane == 0 && ok) {
      f->n = nops;
      f->s = s;
      f->check = !(x0 >= xm && p0 >= pm && d0 >= dm);  // (NaN among them, too)
      f->limx = __double2hiint((double)x0);
      f->limp = __double2hiint((double)p0);
      f->limd = __double2hiint((double)d0);
      int64_t v;  // a kick of at most a quarter of the momentum bound
      if (!fx::fixc(0.25 * (double)p0, s.p, &v)) ok = false;
      f->limk = (int)(v >> 32);
      auto width = [](int ncell) {
        int w = 0;
        while ((1 << w) < ncell + 2) ++w;
        return w;
      };
      // grid coordinate in units of 2^-F, at most 2^57; no coarser than binary64
      // at the far edge
      auto grid = [&](double inv_d, double cc, int ncell, FxGrid* g) {
        int ff = 57 - width(ncell);
        const int room = 61 - fx::exp_of(inv_d) + s.x - 64;
        if (room < ff) ff = room;
        int64_t t;
        if (ff < 53 - width(ncell) || !fx::fixv(inv_d, ff - s.x + 64, &g->a) || !fx::fixc(cc - 0.5, ff, &t)) {
          ok = false;
          return;
        }
        g->c = t;
        g->F = ff;
        // t + 1/2 within [1/4, ncell - 1/4]
        g->half = 1 << (ff - 33);
        g->lo = (1 << (ff - 34)) - g->half;
        g->hi = (int)(((long long)(4 * ncell - 1) << (ff - 2)) >> 32) - g->half;
      };
      grid(st->inv_dx, 0.5 - st->xmin * st->inv_dx, nx, &f->gx);
      grid(st->inv_dy, 0.5 - st->ymin * st->inv_dy, ny, &f->gy);
      f->ny = ny;
      f->nz = nz;
      f->az = st->inv_dz;
      f->cz = 0.5 - st->zmin * st->inv_dz;
      f->Fz = 57 - width(nz);
    }
  }
  if (lane == 0) f->ok = ok ? 1 : 0;
}

// The kick's constants (one thread), which hang on the finished line density.
__device__ __forceinline__ void prep_kick(const PrepJob& J, const ScState* st, int nx, int ny, int nz) {
  FxPass* f = &J.out->fx;
  KickConst kc;
  KickFix kx;
  load_kick_const(kc, st, J.host_factor, nx, ny, nz, false);
  J.out->k = kc;
  load_kick_fix(kx, st, kc.fac, nx, ny, nz);
  J.out->kf = kx;
  const double gx = -kc.fac * kx.ax, gy = -kc.fac * kx.ay;
  const int e = max(fx::exp_of(gx), fx::exp_of(gy));
  f->ce = e;
  bool ok = true;
  if (e < -2000) {  // no kick
    f->Cx = f->Cy = fx::V{0, 0};
  } else {
    ok = fx::fixv(gx, 61 - e, &f->Cx) && fx::fixv(gy, 61 - e, &f->Cy);
  }
  f->kick_ok = ok ? 1 : 0;
}

// Executed by one warp: `maps`, then `kick`, the latter with `bar` after nblk
// blocks have arrived there.  The fused convolution gives both to one block; the
// separate forward rows give them to two, which run side by side.
static __device__ __noinline__ void prep_pass(const PrepJob& J, const ScState* st, int nx, int ny, int nz, bool maps,
                                              bool kick, unsigned* bar, unsigned nblk, long long polls,
                                              unsigned* status) {
  if (maps) prep_maps(J, st, nx, ny, nz);
  if (bar) {
    if ((threadIdx.x & 31) == 0) counter_wait(bar, nblk, polls, status);
    __syncwarp();
  }
  if (kick && (threadIdx.x & 31) == 0) prep_kick(J, st, nx, ny, nz);
}

// Executed by warp 0 of a block: the constants (with those of nops maps) into
// shared memory, with the potential's scale.
__device__ __forceinline__ void load_prep(const PassPrep* __restrict__ prep, const ScState* st, int nops,
                                          PassPrep* s) {
  const int lane = threadIdx.x & 31;
  const int n16 = (int)((offsetof(PassPrep, fx) + offsetof(FxPass, op) + (nops < fx::kMaxOps ? nops + 1 : 0) * sizeof(fx::Op)) / 16);
  const int sphi = scale_bits(__ldcg(&st->phi_absmax));
  const int skip = __ldcg(&st->skip);  // a skipped kick made no constants
  constexpr int U = 4;  // loads in flight
  for (int i = lane; i < n16; i += 32 * U) {
    int4 v[U];
#pragma unroll
    for (int q = 0; q < U; ++q)
      if (i + 32 * q < n16) v[q] = __ldcg(reinterpret_cast<const int4*>(prep) + i + 32 * q);
#pragma unroll
    for (int q = 0; q < U; ++q)
      if (i + 32 * q < n16) reinterpret_cast<int4*>(s)[i + 32 * q] = v[q];
  }
  __syncwarp();
  if (lane == 0 && skip) {
    s->k.skip = skip;
    s->fx.ok = 0;
  } else if (lane == 0) {
    KickFix* kf = &s->kf;
    FxPass* f = &s->fx;
    kf->sphi = sphi;
    kf->gxs = sf::pow2mul(kf->ax, 5 - sphi);
    kf->gys = sf::pow2mul(kf->ay, 5 - sphi);
    // kick = (gx 2^4) (lambda 2^2) 2^-64 C 2^(j-64), C = -factor / step in the
    // kick's units over 2^j
    int j = f->ce + 129 - sphi - kf->slam + f->s.p - 61;
    if (f->ce < -2000) j = 0;
    if (j < 0) {
      const int r = -j > 62 ? 62 : -j;
      f->Cx = fx::sp(fx::join(f->Cx) >> r);
      f->Cy = fx::sp(fx::join(f->Cy) >> r);
      j = 0;
    }
    f->j = j;
    if (j > 29 || !f->kick_ok) f->ok = 0;
    else f->limj = 1 << (29 - j);
  }
}

}  // namespace orbit
