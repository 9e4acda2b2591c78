// Lattice programs: a recorded node sequence (the order AccNode.trackActions
// produces, py/orbit/lattice/AccNode.py:302-350) compiled into fused device
// passes and replayed from a CUDA graph.
//
// A turn with SC kicks S_0..S_{m-1} between map segments M_0..M_m runs as
//   [P_0]  solve(S_0) P_1 solve(S_1) ... solve(S_{m-1}) P_m
// where P_0 = M_0 + extrema(S_0), P_i = kick(S_{i-1}) + M_i + extrema(S_i) and
// the last pass of a turn that is followed by another turn also applies M_0
// of the next turn and the extrema scan for its first kick.  Every pass reads
// and writes the six coordinates once; the deposit reads x, y, z once more.
#include <cstring>
#include <vector>

#include "common.cuh"
#include "sc2p5d.cuh"
#include "passprep.cuh"
#include "sc_device.cuh"
#include "teapot.cuh"
#include "batch.cuh"
#include "program.cuh"

namespace orbit {

static const int kPassSmem = 220 * 1024;

// Threads per block of the fused pass (one block per SM when the kick keeps
// its potential in shared memory); the register budget per thread is
// 65536 / ORBIT_PASS_THREADS.
#ifndef ORBIT_PASS_THREADS
#define ORBIT_PASS_THREADS 512
#endif
// The same of the fixed-point pass.
#ifndef ORBIT_FX_THREADS
#define ORBIT_FX_THREADS 640
#endif

// The kick constants of a pass (one thread), out of line so that their
// registers do not weigh on the particle loop's.
__device__ __noinline__ void kick_consts_into(KickConst* k, KickFix* kf, const KickArgs& kick) {
  load_kick_const(*k, kick.st, kick.host_factor, kick.nx, kick.ny, kick.nz, kf == nullptr);
  if (kf) load_kick_fix(*kf, kick.st, k->fac, kick.nx, kick.ny, kick.nz);
}

// Cell and fraction (Q62) of tsc_fixed; false within a quarter cell of the
// grid's edge or outside.
__device__ __forceinline__ bool cell_fx(const FxGrid& g, long long x, int ncell, int& ic, long long& f) {
  const long long t = fx::mul(g.a, fx::sp(x), g.c);
  const int h = (int)(t >> 32);
  const int i = (h + g.half) >> (g.F - 32);
  ic = min(max(i, 1), ncell - 2);
  f = (long long)((unsigned long long)t << (62 - g.F)) - ((long long)ic << 62);
  return (h >= g.lo) & (h <= g.hi);
}

// The plain kick in fixed point; false: the particle takes the FP64 path.
// Every particle lies in [zmin, zmax], the extent of the scan before it.
__device__ __forceinline__ bool kick_fx(const FxPass& f, int nx, const long long* __restrict__ P,
                                        const long long* __restrict__ Lm, fx::Part& t) {
  int ix, iy;
  long long gfx, gfy, gx, gy, lv;
  const bool in = cell_fx(f.gx, t.x, nx, ix, gfx) & cell_fx(f.gy, t.y, f.ny, iy, gfy);
  if (!in) return false;
  if (f.nz > 1) {
    const long long v = fx::cvt_to(fma(t.z, f.az, f.cz), f.Fz);
    const int i = min(max((int)(v >> f.Fz), 0), f.nz);
    const long long w = (long long)((unsigned long long)(v - ((long long)i << f.Fz)) << (62 - f.Fz));
    lv = fx::mul2(fx::sp((1ll << 62) - w), fx_of_pair(Lm[(i == 0 ? f.nz : i) - 1]), fx::sp(w),
                  fx_of_pair(Lm[i == f.nz ? 0 : i]));
  } else {
    lv = fx::join(fx_of_pair(Lm[0])) >> 2;
  }
  grad_fixed(P, f.ny, ix, iy, gfx, gfy, gx, gy);
  const fx::V l2 = fx::sp(lv << 2);
  const long long px = fx::mul(fx::sp(gx << 4), l2), py = fx::mul(fx::sp(gy << 4), l2);
  const long long dx = fx::mul(fx::sp(px << f.j), f.Cx), dy = fx::mul(fx::sp(py << f.j), f.Cy);
  t.p += dx;
  t.r += dy;
  return fx::within(gx, (1 << 26) - 1) & fx::within(gy, (1 << 26) - 1) & fx::within(px, f.limj) &
         fx::within(py, f.limj) & fx::within(dx, f.limk) & fx::within(dy, f.limk);
}

// What the FP64 routines of a fixed-point pass need, kept in shared memory,
// with the extrema and magnitudes of the particles they take.
struct FxFallback {
  const KickConst* k;
  const KickFix* kf;
  const long long* P;
  const long long* Lm;
  double* c[5];
  const double* dE;
  double* knl;
  const KickArgs* kick;
  const MapCtx* m;
  const DevOp* ops;
  int a, b;
  unsigned long long mn[3], mx[3];
  unsigned pm;
  int bad;
  unsigned taken;  // particles the FP64 routines took
  int fixed;       // the pass runs in fixed point
  int declined;    // some of the block's particles are left to the FP64 routines
};

static_assert(kPassSmem + sizeof(FxFallback) + sizeof(PassPrep) + kCommitSmem + 64 <= kBlockSmem,
              "k_pass_fx: its own shared memory beside the largest copy of the potential");

// A declined particle's 1/(1+dp_p) until the FP64 routines take it: minus
// infinity, which the reciprocal of a sum never is.
__device__ __forceinline__ double declined_mark() { return __hiloint2double((int)0xfff00000u, 0); }
__device__ __forceinline__ bool declined(double knl) { return knl == declined_mark(); }

// One particle by the FP64 routines: those the fixed-point form declines,
// and all of a pass it cannot run.
template <bool EXT>
__device__ __noinline__ void pass_particle(FxFallback* f, int i) {
  Part p;
  p.x = f->c[0][i]; p.xp = f->c[1][i]; p.y = f->c[2][i]; p.yp = f->c[3][i]; p.z = f->c[4][i]; p.dE = f->dE[i];
  p.knl = f->knl[i];
  p.dp_p = dmul<ORBIT_SOFT_MUL & 1>(p.dE, f->m->dp_p_coeff);
  p.knl_ok = !declined(p.knl);
  if (!p.knl_ok) {  // the mark stands in its place
    ensure_knl<ORBIT_SOFT_MUL & 1>(p, *f->m);
    f->knl[i] = p.knl;
  }
  if (!f->k->skip && bnd_inside(f->kick->bnd, p.x, p.y)) {
    if (!kick_fixed(*f->kf, f->P, f->Lm, p.x, p.y, p.z, p.xp, p.yp)) {
      kick_plain(*f->k, f->kick->phi, f->kick->lam, p.x, p.y, p.z, p.xp, p.yp);
    }
  }
  apply_ops<ORBIT_SOFT_MUL>(p, f->ops, f->a, f->b, *f->m);
  if (EXT) {
    ExtAcc e;
    e.init();
    e.add(p.x, p.y, p.z);
    e.finish();
    for (int c = 0; c < 3; ++c) {
      atomicMin(&f->mn[c], e.mn[c]);
      atomicMax(&f->mx[c], e.mx[c]);
    }
    if (e.bad) f->bad = 1;
    MagAcc g;
    g.init();
    g.bound(p.xp, p.yp);
    atomicMax(&f->pm, g.pm);
  }
  f->c[0][i] = p.x; f->c[1][i] = p.xp; f->c[2][i] = p.y; f->c[3][i] = p.yp; f->c[4][i] = p.z;
}

// Leaves particle i to the FP64 routines.  Out of line: with a call in its loop
// the pass keeps its constants in shared memory (hoisted out of the loop they
// spill) and its other registers as they are; marking in place was 1 to 3% slower.
__device__ __noinline__ void fx_decline(FxFallback* f, int i) {
  if (f->fixed) f->knl[i] = declined_mark();
  f->declined = 1;
}

// Extrema of a pass run in fixed point: x and y as integers (their
// conversion to the stored doubles is monotonic), z as a key.
struct ExtFx {
  long long mn[2], mx[2];
  unsigned long long zn, zx;
  __device__ __forceinline__ void init() {
    mn[0] = mn[1] = 0x7fffffffffffffffll;
    mx[0] = mx[1] = -0x7fffffffffffffffll;
    zn = ~0ull;
    zx = 0ull;
  }
  __device__ __forceinline__ void add(long long x, long long y, double z) {
    mn[0] = min(mn[0], x);
    mx[0] = max(mx[0], x);
    mn[1] = min(mn[1], y);
    mx[1] = max(mx[1], y);
    const unsigned long long k = dkey(z);
    zn = min(zn, k);
    zx = max(zx, k);
  }
  // As keys of the stored doubles.
  __device__ __forceinline__ void join(ExtAcc& a, int S) const {
    for (int c = 0; c < 2; ++c) {
      if (mn[c] > mx[c]) continue;
      a.mn[c] = dkey(fx::cvt_from(mn[c], S));
      a.mx[c] = dkey(fx::cvt_from(mx[c], S));
    }
    a.mn[2] = zn;
    a.mx[2] = zx;
  }
};

// Copies the potential and line density the kick reads into the block's
// shared memory (threads t0.. of the block): KF 1 as fixed-point pairs made
// from the FP64 values at the scales the kick constants use.
template <int KF>
__device__ __forceinline__ void fill_kick_grids(const KickArgs& kick, unsigned char* s_raw, int t0) {
  const int ng = kick.nx * kick.ny;
  if (KF == 1) {
    const int sphi = scale_bits(kick.st->phi_absmax), slam = scale_bits(kick.st->lam_absmax);
    double* sd = reinterpret_cast<double*>(s_raw);  // the FP64 values land in place and become integers there
    copy_smem_async(sd, kick.phi, ng,
                    [sphi](double v) { return __longlong_as_double(fx_pair(phi_fixed(v, sphi))); }, t0);
    copy_smem_async(sd + ng, kick.lam, kick.nz,
                    [slam](double v) { return __longlong_as_double(fx_pair(phi_fixed(v, slam))); }, t0);
  } else {
    float* s = reinterpret_cast<float*>(s_raw);
    copy_smem_async(s, kick.phi_f, ng, [](float v) { return v; }, t0);
    copy_smem_async(s + ng, kick.lam_f, kick.nz, [](float v) { return v; }, t0);
  }
}

// KF: 0 no kick, 1 plain kick, 2 fp32 kick.  EXT: accumulate extrema.
// Blocks blk = 0..nblk-1 share the bunch's particles.  The FP64 pass: the
// first of a run, and those whose maps or kick (2.5Drb) have no fixed-point
// form.
template <int KF, bool EXT, bool KSMEM>
__device__ __forceinline__ void pass_body(double* __restrict__ cx, double* __restrict__ cxp,
                                          double* __restrict__ cy, double* __restrict__ cyp,
                                          double* __restrict__ cz, double* __restrict__ cdE, int n,
                                          const DevOp* __restrict__ ops, int a, int b, const MapCtx& m,
                                          const KickArgs& kick, ScState* ext_st, unsigned* status,
                                          const SetupArgs& sa, double* __restrict__ knl_buf, int km, int blk,
                                          int nblk) {
  KickConst k;
  KickFix kf;
  const long long* P = kick.phi_fix;
  const long long* Lm = kick.lam_fix;
  const float* Pf = kick.phi_f;
  const float* Lf = kick.lam_f;
  extern __shared__ __align__(16) unsigned char s_raw[];
  if (KF != 0) {
    // thread 0 computes the kick constants (two FP64 divisions among
    // them) while warps 1.. fill the block's copy of the potential and the
    // line density; one barrier completes both
    __shared__ KickConst s_k;
    __shared__ KickFix s_kf;
    if (threadIdx.x == 0) kick_consts_into(&s_k, KF == 1 ? &s_kf : nullptr, kick);
    if (KSMEM) {
      fill_kick_grids<KF>(kick, s_raw, blockDim.x > 64 ? 32 : 0);
      P = reinterpret_cast<const long long*>(s_raw);
      Lm = P + kick.nx * kick.ny;
      Pf = reinterpret_cast<const float*>(s_raw);
      Lf = Pf + kick.nx * kick.ny;
    }
    __syncthreads();
    k = s_k;
    if (KF == 1) kf = s_kf;
  }
  ExtAcc acc;
  MagAcc mag;
  if (EXT) {
    acc.init();
    mag.init();
  }
  for (int i = blk * blockDim.x + threadIdx.x; i < n; i += nblk * blockDim.x) {
    Part p;
    p.x = cx[i]; p.xp = cxp[i]; p.y = cy[i]; p.yp = cyp[i]; p.z = cz[i]; p.dE = cdE[i];
    p.knl_ok = false;
    if (km & KNL_LOAD) {  // 1/(1+dp_p) as an earlier pass of this run computed it from the same dE
      p.dp_p = dmul<ORBIT_SOFT_MUL & 1>(p.dE, m.dp_p_coeff);
      p.knl = knl_buf[i];
      p.knl_ok = true;
    }
    if (KF == 1 && !k.skip && bnd_inside(kick.bnd, p.x, p.y)) {
      if (!kick_fixed(kf, P, Lm, p.x, p.y, p.z, p.xp, p.yp))
        kick_plain(k, kick.phi, kick.lam, p.x, p.y, p.z, p.xp, p.yp);
      if (kick.lamd) {  // 2.5Drb: longitudinal kick; dE changed
        RbConst r;
        load_rb_const(r, kick.st, kick.rb_lsf);
        kick_rb_long(k, r, kick.lamd, p.x, p.y, p.z, p.dE);
        p.knl_ok = false;
      }
    }
    if (KF == 2 && !k.skip && bnd_inside(kick.bnd, p.x, p.y)) kick_fp32(k, Pf, Lf, p.x, p.y, p.z, p.xp, p.yp);
    apply_ops<ORBIT_SOFT_MUL>(p, ops, a, b, m);
    if (EXT) {
      acc.add(p.x, p.y, p.z);
      if (sa.mag) {
        mag.bound(p.xp, p.yp);
        mag.em = max(mag.em, MagAcc::hi(p.dE));
      }
    }
    if (km & KNL_STORE) {
      ensure_knl<ORBIT_SOFT_MUL & 1>(p, m);
      knl_buf[i] = p.knl;
    }
    cx[i] = p.x; cxp[i] = p.xp; cy[i] = p.y; cyp[i] = p.yp; cz[i] = p.z; cdE[i] = p.dE;
  }
  // the last block sets up the grids of the next kick
  if (EXT) {
    if (sa.mag) mag_block_commit(mag, ext_st);
    ext_commit_and_setup(acc, ext_st, status, sa, nblk);
  }
}

// The pass in fixed point: maps that all have a fixed-point form, dE and
// 1/(1+dp_p) unchanged, the plain form's kick.  A pass whose magnitudes or
// constants do not fit (FxPass::ok, the same in every block) goes particle by
// particle through the FP64 routines: 1e6 particles, 128 x 128 x 64, quadrupole
// fringes beyond their limits, 327 us a kick (359 before the fixed-point form).
//
// Bound by the issue of integer instructions: 777 a particle for a kick and a
// drift, about 1300 with two half quadrupoles and their fringes, at half an
// instruction a clock per sub-partition with 5 warps there (512, 640 and 768
// threads are within 3% of one another).  At 1e6 particles, 128 x 128 x 64, a
// FODO segment: 53 us against 140 us of the FP64 pass; at 16e6 particles,
// 256 x 256 x 64, ring segments: 2.0 ms against 4.3 ms.
//
// The FP32 form keeps the FP64 pass: a rounding of its fields that flips
// moves the whole potential by 5e-8, so coordinates that differ in the last
// bit give beams that differ at the form's own error, 2e-5 after 16 kicks.
template <bool EXT, bool KSMEM>
__device__ __forceinline__ void pass_fx_body(double* __restrict__ cx, double* __restrict__ cxp,
                                             double* __restrict__ cy, double* __restrict__ cyp,
                                             double* __restrict__ cz, const double* __restrict__ cdE, int n,
                                             const DevOp* __restrict__ ops, int a, int b, const MapCtx& m,
                                             const KickArgs& kick, ScState* ext_st, unsigned* status,
                                             const SetupArgs& sa, double* __restrict__ knl_buf,
                                             const PassPrep* __restrict__ prep, int blk, int nblk) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  __shared__ FxFallback s_f;
  __shared__ PassPrep s_prep;
  FxPass& s_fx = s_prep.fx;
  // warp 0 takes the constants made beside the solve and adds what hangs on
  // the potential's maximum while warps 1.. fill the block's copy of the
  // potential and the line density; one barrier completes both
  if (threadIdx.x < 32) {
    load_prep(prep, kick.st, b - a, &s_prep);
    if (threadIdx.x == 0) {
      const size_t ng = (size_t)kick.nx * kick.ny;
      s_f.P = KSMEM ? reinterpret_cast<const long long*>(s_raw) : kick.phi_fix;
      s_f.Lm = KSMEM ? s_f.P + ng : kick.lam_fix;
      s_f.c[0] = cx; s_f.c[1] = cxp; s_f.c[2] = cy; s_f.c[3] = cyp; s_f.c[4] = cz;
      s_f.k = &s_prep.k; s_f.kf = &s_prep.kf;
      s_f.dE = cdE; s_f.knl = knl_buf; s_f.kick = &kick; s_f.m = &m; s_f.ops = ops; s_f.a = a; s_f.b = b;
      for (int c = 0; c < 3; ++c) { s_f.mn[c] = ~0ull; s_f.mx[c] = 0ull; }
      s_f.pm = 0u;
      s_f.bad = 0;
      s_f.taken = 0u;
      s_f.fixed = s_fx.ok;
      s_f.declined = 0;
    }
  }
  if (KSMEM) fill_kick_grids<1>(kick, s_raw, blockDim.x > 64 ? 32 : 0);
  __syncthreads();
  const long long* P = KSMEM ? reinterpret_cast<const long long*>(s_raw) : kick.phi_fix;
  const long long* Lm = KSMEM ? P + (size_t)kick.nx * kick.ny : kick.lam_fix;
  const bool fixed = s_fx.ok != 0, bound = kick.bnd.type >= 0;
  if (fixed && blk == 0 && threadIdx.x == 0) atomicAdd(&kick.st->n_fixed, 1ull);
  const fx::Scales s = s_fx.s;
  ExtFx ext;
  MagAcc mag;
  if (EXT) {
    ext.init();
    mag.init();
  }
  const int di = nblk * blockDim.x;
  for (int i = first_particle(blk, nblk); i < n; i += nblk * blockDim.x) {
    bool ok = fixed;
    fx::Part t;
    if (ok) {
      const double x = cx[i], xp = cxp[i], y = cy[i], yp = cyp[i], dE = cdE[i];
      const double knl = knl_buf[i];  // as an earlier pass of this run computed it from the same dE
      const double dp = __dmul_rn(dE, m.dp_p_coeff);
      t.z = cz[i];
      t.x = fx::cvt_to(x, s.x);
      t.p = fx::cvt_to(xp, s.p);
      t.y = fx::cvt_to(y, s.x);
      t.r = fx::cvt_to(yp, s.p);
      if (s_fx.check) {
        auto inside = [](double v, int lim) { return (__double2hiint(v) & 0x7fffffff) <= lim; };
        ok = inside(x, s_fx.limx) & inside(y, s_fx.limx) & inside(xp, s_fx.limp) & inside(yp, s_fx.limp) &
             inside(dp, s_fx.limd);
      }
      if (ok && (!bound || bnd_inside(kick.bnd, x, y))) {
        ok = kick_fx(s_fx, kick.nx, P, Lm, t);
      }
      fx::part_init(t, fx::kappa_of(knl), fx::cvt_to(dp, s.k), s.k);
    }
    if (!ok) {
      fx_decline(&s_f, i);
      continue;
    }
    fx::apply(t, s_fx.op, s_fx.n, s);
    const double x = fx::cvt_from(t.x, s.x), xp = fx::cvt_from(t.p, s.p), y = fx::cvt_from(t.y, s.x), yp = fx::cvt_from(t.r, s.p);
    const double z = t.z + fx::cvt_from(t.d, s.d);
    if (EXT) {
      ext.add(t.x, t.y, z);
      mag.bound(xp, yp);
    }
    cx[i] = x; cxp[i] = xp; cy[i] = y; cyp[i] = yp; cz[i] = z;
  }
  __syncthreads();
  // A warp goes through the FP64 routines, 64 clocks an instruction, for any one
  // of its lanes: the declined particles wait for the end of the loop, and every
  // 32 rounds' are then taken lane by lane together.  Taken at once, 5% of 1e6
  // particles far out made a kick 290 us (251 when every pass was of FP64), so
  // 216.
  if (s_f.declined) {
    for (int i = first_particle(blk, nblk); i < n;) {
      unsigned todo = 0u;
      const int i0 = i;
      for (int r = 0; r < 32 && i < n; ++r, i += di)
        if (!fixed || declined(knl_buf[i])) todo |= 1u << r;
      if (todo) atomicAdd(&s_f.taken, (unsigned)__popc(todo));
      for (; todo; todo &= todo - 1u) pass_particle<EXT>(&s_f, i0 + (__ffs(todo) - 1) * di);
    }
    __syncthreads();  // their extrema and count
    if (threadIdx.x == 0) atomicAdd(&kick.st->n_fp64, (unsigned long long)s_f.taken);
  }
  // the last block sets up the grids of the next kick
  if (EXT) {
    ExtAcc acc;
    acc.init();
    ext.join(acc, s.x);
    if (threadIdx.x == 0) {
      for (int c = 0; c < 3; ++c) {
        acc.mn[c] = min(acc.mn[c], s_f.mn[c]);
        acc.mx[c] = max(acc.mx[c], s_f.mx[c]);
      }
      acc.bad = s_f.bad != 0;
      mag.pm = max(mag.pm, s_f.pm);
      // dE is unchanged; without magnitudes before, none are claimed
      mag.em = kick.st->mag.pmax ? kick.st->mag.emax : 0x7fefffffu;
    }
    if (sa.mag) mag_block_commit(mag, ext_st);
    ext_commit_and_setup(acc, ext_st, status, sa, nblk);
  }
}

template <int KF, bool EXT, bool KSMEM>
__global__ void __launch_bounds__(ORBIT_PASS_THREADS) k_pass(double* __restrict__ cx, double* __restrict__ cxp,
                                              double* __restrict__ cy, double* __restrict__ cyp,
                                              double* __restrict__ cz, double* __restrict__ cdE, int n,
                                              const DevOp* __restrict__ ops, int a, int b, MapCtx m,
                                              KickArgs kick, ScState* ext_st, unsigned* status,
                                              const __grid_constant__ SetupArgs sa,
                                              double* __restrict__ knl_buf, int km) {
  pass_body<KF, EXT, KSMEM>(cx, cxp, cy, cyp, cz, cdE, n, ops, a, b, m, kick, ext_st, status, sa, knl_buf, km,
                            blockIdx.x, gridDim.x);
}

template <bool EXT, bool KSMEM>
__global__ void __launch_bounds__(ORBIT_FX_THREADS) k_pass_fx(double* __restrict__ cx, double* __restrict__ cxp,
                                              double* __restrict__ cy, double* __restrict__ cyp,
                                              double* __restrict__ cz, const double* __restrict__ cdE, int n,
                                              const DevOp* __restrict__ ops, int a, int b,
                                              const __grid_constant__ MapCtx m,
                                              const __grid_constant__ KickArgs kick, ScState* ext_st,
                                              unsigned* status, const __grid_constant__ SetupArgs sa,
                                              double* __restrict__ knl_buf,
                                              const PassPrep* __restrict__ prep) {
  pass_fx_body<EXT, KSMEM>(cx, cxp, cy, cyp, cz, cdE, n, ops, a, b, m, kick, ext_st, status, sa, knl_buf,
                               prep, blockIdx.x, gridDim.x);
}

// The same passes for the members of a batch class; each block finds its
// member in the block table.
template <int KF, bool EXT, bool KSMEM>
__global__ void __launch_bounds__(ORBIT_PASS_THREADS) kb_pass(const PassJob* __restrict__ jobs,
                                               const unsigned short* __restrict__ blk_job,
                                               const int2* __restrict__ mblk, int a, int b, int km) {
  const int j = blk_job[blockIdx.x];
  const PassJob& J = jobs[j];
  const int2 mb = mblk[j];
  pass_body<KF, EXT, KSMEM>(J.c[0], J.c[1], J.c[2], J.c[3], J.c[4], J.c[5], J.n, J.ops, a, b, J.m, J.ka, J.ext,
                            J.status, J.sa, J.knl, km, blockIdx.x - mb.x, mb.y);
}

template <bool EXT, bool KSMEM>
__global__ void __launch_bounds__(ORBIT_FX_THREADS) kb_pass_fx(const PassJob* __restrict__ jobs,
                                               const unsigned short* __restrict__ blk_job,
                                               const int2* __restrict__ mblk, int a, int b) {
  const int j = blk_job[blockIdx.x];
  const PassJob& J = jobs[j];
  const int2 mb = mblk[j];
  pass_fx_body<EXT, KSMEM>(J.c[0], J.c[1], J.c[2], J.c[3], J.c[4], J.c[5], J.n, J.ops, a, b, J.m, J.ka, J.ext,
                              J.status, J.sa, J.knl, J.prep, blockIdx.x - mb.x, mb.y);
}

// Shared-memory limits are raised once, outside any stream capture.
static int init_pass_attrs() {
  static bool done = false;
  if (done) return ORBIT_OK;
  ORBIT_CUDA(cudaFuncSetAttribute(k_pass<1, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPassSmem));
  ORBIT_CUDA(cudaFuncSetAttribute(k_pass<1, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPassSmem));
  ORBIT_CUDA(cudaFuncSetAttribute(k_pass<2, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPassSmem));
  ORBIT_CUDA(cudaFuncSetAttribute(k_pass<2, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPassSmem));
  ORBIT_CUDA(cudaFuncSetAttribute(kb_pass<1, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPassSmem));
  ORBIT_CUDA(cudaFuncSetAttribute(kb_pass<1, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPassSmem));
  ORBIT_CUDA(cudaFuncSetAttribute(k_pass_fx<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPassSmem));
  ORBIT_CUDA(cudaFuncSetAttribute(k_pass_fx<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPassSmem));
  ORBIT_CUDA(cudaFuncSetAttribute(kb_pass_fx<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPassSmem));
  ORBIT_CUDA(cudaFuncSetAttribute(kb_pass_fx<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPassSmem));
  done = true;
  return ORBIT_OK;
}

template <int KF, bool EXT, bool KSMEM>
static int launch_pass(orbit_bunch_t* bu, cudaStream_t s, size_t smem, const DevOp* ops, int a, int b,
                       const MapCtx& m, const KickArgs& ka, ScState* ext, const SetupArgs& sa, double* knl_buf,
                       int km, bool fixed, const PassPrep* prep) {
  const int threads = spread_threads(bu->n, fixed ? ORBIT_FX_THREADS : ORBIT_PASS_THREADS);
  int bps = KSMEM ? (int)(kPassSmem / (smem > 0 ? smem : 1)) : 4;
  if (bps < 1) bps = 1;
  if (bps > 4) bps = 4;
  int blocks = num_sms() * bps;
  int need = (bu->n + threads - 1) / threads;
  if (need < blocks) blocks = need < 1 ? 1 : need;
  ORBIT_PB(KF == 0 ? "pass_maps" : "pass_kick_maps", s);
  if constexpr (KF == 1) {
    if (fixed) {
      k_pass_fx<EXT, KSMEM><<<blocks, threads, KSMEM ? smem : 0, s>>>(
          bu->coord(0), bu->coord(1), bu->coord(2), bu->coord(3), bu->coord(4), bu->coord(5), bu->n, ops, a, b, m,
          ka, ext, bu->d_status, sa, knl_buf, prep);
      ORBIT_PE(s);
      ORBIT_LAUNCH_CHECK("k_pass_fx");
      return ORBIT_OK;
    }
  }
  k_pass<KF, EXT, KSMEM><<<blocks, threads, KSMEM ? smem : 0, s>>>(
      bu->coord(0), bu->coord(1), bu->coord(2), bu->coord(3), bu->coord(4), bu->coord(5), bu->n, ops, a, b, m, ka,
      ext, bu->d_status, sa, knl_buf, km);
  ORBIT_PE(s);
  ORBIT_LAUNCH_CHECK("k_pass");
  return ORBIT_OK;
}

size_t batch_pass_smem_limit() { return kPassSmem; }

int batch_enqueue_pass(const PassJob* jobs, const BlockMap& bm, int threads, int kf, bool ext, bool ksmem,
                       size_t smem, int a, int b, int km, bool fixed, cudaStream_t s, const char* tag) {
  int arc = init_pass_attrs();
  if (arc) return arc;
  const int nb = bm.nblk;
  ORBIT_PB(kf == 0 ? "batch_pass_maps" : tag, s);
  if (kf == 0) {
    if (ext) kb_pass<0, true, false><<<nb, threads, 0, s>>>(jobs, bm.blk_job, bm.mblk, a, b, km);
    else kb_pass<0, false, false><<<nb, threads, 0, s>>>(jobs, bm.blk_job, bm.mblk, a, b, km);
  } else if (fixed) {
    const int t = ORBIT_FX_THREADS;
    if (ksmem) {
      if (ext) kb_pass_fx<true, true><<<nb, t, smem, s>>>(jobs, bm.blk_job, bm.mblk, a, b);
      else kb_pass_fx<false, true><<<nb, t, smem, s>>>(jobs, bm.blk_job, bm.mblk, a, b);
    } else {
      if (ext) kb_pass_fx<true, false><<<nb, t, 0, s>>>(jobs, bm.blk_job, bm.mblk, a, b);
      else kb_pass_fx<false, false><<<nb, t, 0, s>>>(jobs, bm.blk_job, bm.mblk, a, b);
    }
  } else if (ksmem) {
    if (ext) kb_pass<1, true, true><<<nb, threads, smem, s>>>(jobs, bm.blk_job, bm.mblk, a, b, km);
    else kb_pass<1, false, true><<<nb, threads, smem, s>>>(jobs, bm.blk_job, bm.mblk, a, b, km);
  } else {
    if (ext) kb_pass<1, true, false><<<nb, threads, 0, s>>>(jobs, bm.blk_job, bm.mblk, a, b, km);
    else kb_pass<1, false, false><<<nb, threads, 0, s>>>(jobs, bm.blk_job, bm.mblk, a, b, km);
  }
  ORBIT_PE(s);
  ORBIT_LAUNCH_CHECK("batch pass");
  return ORBIT_OK;
}

}  // namespace orbit

using namespace orbit;

namespace orbit {

static void free_graphs(orbit_program_t* p) {
  cudaGraphExec_t* gs[] = {&p->g_first, &p->g_mid, &p->g_last, &p->g_single};
  for (auto g : gs)
    if (*g) { cudaGraphExecDestroy(*g); *g = nullptr; }
}

static bool sync_equal(const orbit_sync_t& a, const orbit_sync_t& b) {
  return a.beta == b.beta && a.gamma == b.gamma && a.momentum == b.momentum && a.charge == b.charge &&
         a.classical_radius == b.classical_radius && a.macrosize == b.macrosize && a.mass == b.mass;
}

KickArgs kick_args(orbit_sc2p5d_t* c, const orbit_sync_t& s, double length, const orbit_boundary* bnd) {
  KickArgs ka;
  ka.st = c->d_st;
  ka.phi = c->d_phi;
  ka.lam = c->d_lam;
  ka.phi_f = c->d_phi_f;
  ka.lam_f = c->d_lam_f;
  ka.phi_fix = c->d_phi_fix;
  ka.lam_fix = c->d_lam_fix;
  ka.host_factor = sc_host_factor(s, length);
  ka.nx = c->nx; ka.ny = c->ny; ka.nz = c->nz; ka.form = c->form;
  ka.lamd = c->rb ? c->d_lamd : nullptr;
  ka.rb_lsf = c->rb ? sc_rb_long_factor(s, length) : 0.0;
  ka.bnd = bnd_shape_of(bnd);
  return ka;
}

// One fused pass: optional kick of calculator kc, maps [a,b), optional
// extrema for calculator ec.
// ec_here: the kick of ec is enqueued next in this same stream (and graph),
// so a graph branch for its Green rebuild can be set up by this pass.
static int enqueue_pass(orbit_bunch_t* bu, cudaStream_t s, const DevOp* ops, Seg seg, const MapCtx& m,
                        orbit_sc2p5d_t* kc, double klen, const orbit_boundary* kb, orbit_sc2p5d_t* ec,
                        const orbit_boundary* eb, bool ec_here, double* knl_buf, int km, int* nl) {
  KickArgs ka;
  std::memset(&ka, 0, sizeof(ka));
  int kf = 0;
  size_t smem = 0;
  bool ksm = false;
  if (kc) {
    ka = kick_args(kc, bu->sync, klen, kb);
    kf = kc->form == ORBIT_FORM_PLAIN ? 1 : 2;
    smem = (kf == 1 ? 8 : 4) * ((size_t)kc->nx * kc->ny + kc->nz);
    ksm = kc->smem_kick && smem <= (size_t)kPassSmem;  // else the kick reads phi_fix, converted by the solve
  }
  if (!kc && !ec && seg.a == seg.b) return ORBIT_OK;  // nothing to do
  const bool fixed = fixed_pass(seg, kc && kc->form == ORBIT_FORM_PLAIN && !kc->rb, km);
  const PassPrep* prep = kc ? kc->d_prep : nullptr;
  ScState* ext = ec ? ec->d_st : nullptr;
  bool e = ext != nullptr;
  SetupArgs sa;
  std::memset(&sa, 0, sizeof(sa));
  if (ec) {
    sa = sc_setup_args(ec, sc_dep_scales(ec, bu), eb);
    if (ec_here) sa.cond = sc_green_cond(ec, s, true);
  }
  int rc;
  if (kf == 0) rc = e ? launch_pass<0, true, false>(bu, s, 0, ops, seg.a, seg.b, m, ka, ext, sa, knl_buf, km, fixed, prep)
                      : launch_pass<0, false, false>(bu, s, 0, ops, seg.a, seg.b, m, ka, ext, sa, knl_buf, km, fixed, prep);
  else if (kf == 1) {
    if (ksm) rc = e ? launch_pass<1, true, true>(bu, s, smem, ops, seg.a, seg.b, m, ka, ext, sa, knl_buf, km, fixed, prep)
                    : launch_pass<1, false, true>(bu, s, smem, ops, seg.a, seg.b, m, ka, ext, sa, knl_buf, km, fixed, prep);
    else rc = e ? launch_pass<1, true, false>(bu, s, 0, ops, seg.a, seg.b, m, ka, ext, sa, knl_buf, km, fixed, prep)
                : launch_pass<1, false, false>(bu, s, 0, ops, seg.a, seg.b, m, ka, ext, sa, knl_buf, km, fixed, prep);
  } else {
    if (ksm) rc = e ? launch_pass<2, true, true>(bu, s, smem, ops, seg.a, seg.b, m, ka, ext, sa, knl_buf, km, fixed, prep)
                    : launch_pass<2, false, true>(bu, s, smem, ops, seg.a, seg.b, m, ka, ext, sa, knl_buf, km, fixed, prep);
    else rc = e ? launch_pass<2, true, false>(bu, s, 0, ops, seg.a, seg.b, m, ka, ext, sa, knl_buf, km, fixed, prep)
                : launch_pass<2, false, false>(bu, s, 0, ops, seg.a, seg.b, m, ka, ext, sa, knl_buf, km, fixed, prep);
  }
  if (rc == ORBIT_OK) ++*nl;
  return rc;
}

// Builds the device op array: all non-SC ops of the turn in order, then the
// wrap segment (last segment followed by the first).
int compile(orbit_program_t* p, orbit_bunch_t* bu, Plan& plan) {
  std::vector<DevOp> dev;
  p->time_adv.assign(p->ops.size(), 0.0);
  int start = 0;
  std::vector<std::pair<int, int>> seg_ops;  // [first op, last op) in p->ops for each segment
  for (size_t k = 0; k < p->ops.size(); ++k) {
    if (p->ops[k].code == ORBIT_OP_SC) {
      seg_ops.push_back({start, (int)k});
      plan.sc_idx.push_back((int)k);
      start = (int)k + 1;
    }
  }
  seg_ops.push_back({start, (int)p->ops.size()});
  // Maps that add to x, y and z a term linear in their length and change
  // neither xp, yp nor dE (drift; quad2 = bend2) compose by adding lengths:
  // drift(L1) drift(L2) = drift(L1+L2) and quad2(L1) quad2(L2) =
  // quad2(L1+L2), equal in exact arithmetic (each reads only xp, yp and
  // dp_p, which the other leaves alone), one rounding per coordinate instead
  // of two.  The reference's quad schedule issues quad2(L) twice in a row
  // when the element has no multipoles (teapot.py:945-960).
  auto lengthwise = [](int code) {
    return code == ORBIT_OP_DRIFT ? 1 : (code == ORBIT_OP_QUAD2 || code == ORBIT_OP_BEND2) ? 2 : 0;
  };
  auto emit = [&](int a, int b, bool start) -> Seg {
    Seg s;
    if (start) dev.push_back(DevOp{});  // the segment's start entry (fx::compile_segment)
    s.a = (int)dev.size();
    s.dE = false;
    for (int k = a; k < b; ++k) {
      DevOp d;
      double adv = 0.0;
      if (!compile_op(p->ops[k], bu->sync, d, &adv)) return Seg{-1, -1, false, false};
      p->time_adv[k] = adv;
      if (d.code == ORBIT_OP_WEDGEROT || (d.code == ORBIT_OP_KICK && d.c[2] != 0.)) s.dE = true;
      if (d.code == 0) continue;
      if (lengthwise(d.code) && (int)dev.size() > s.a && lengthwise(dev.back().code) == lengthwise(d.code)) {
        dev.back().c[0] += d.c[0];
        continue;
      }
      dev.push_back(d);
    }
    s.b = (int)dev.size();
    return s;
  };
  for (auto& so : seg_ops) {
    Seg s = emit(so.first, so.second, true);
    if (s.a < 0) return set_error(ORBIT_ERR_ARG, "orbit_program: bad op parameters");
    plan.segs.push_back(s);
  }
  Seg w;
  {
    Seg s1 = emit(seg_ops.back().first, seg_ops.back().second, true);
    w.a = s1.a;
    Seg s2 = emit(seg_ops.front().first, seg_ops.front().second, false);
    if (s1.a < 0 || s2.a < 0) return set_error(ORBIT_ERR_ARG, "orbit_program: bad op parameters");
  }
  w.b = (int)dev.size();
  w.dE = plan.segs.back().dE || plan.segs.front().dE;
  plan.wrap = w;
  const double g2 = make_ctx(bu->sync).gamma2i;
  auto mark = [&](Seg& sg) {
    fx::compile_segment(&dev[sg.a - 1], sg.b - sg.a, g2);
    bool moves = false;
    sg.fx = sg.b - sg.a < fx::kMaxOps;
    for (int k = sg.a; k < sg.b; ++k) {
      // multipoles do nothing to a neutral bunch (teapotbase.cc:340, 397, 510): left to the FP64 routines
      const bool pole = dev[k].code == ORBIT_OP_MULTP || dev[k].code == ORBIT_OP_MPFRIN || dev[k].code == ORBIT_OP_MPFROUT;
      sg.fx = sg.fx && fx::supported(dev[k]) && !(pole && bu->sync.charge == 0.);
      moves = moves || fx::moves_x(dev[k]);
    }
    sg.fx = sg.fx && moves;  // x and y are rewritten: thin kicks alone leave them as they are
  };
  for (Seg& sg : plan.segs) mark(sg);
  mark(plan.wrap);
  if (p->knl_n < (size_t)bu->n) {
    if (p->d_knl) { cudaFree(p->d_knl); p->d_knl = nullptr; }
    p->knl_n = 0;
    if (bu->n > 0) {
      ORBIT_CUDA(cudaMalloc(&p->d_knl, sizeof(double) * (size_t)bu->n));
      p->knl_n = (size_t)bu->n;
    }
  }
  if (p->d_ops) { cudaFree(p->d_ops); p->d_ops = nullptr; }
  p->n_devops = (int)dev.size();
  if (!dev.empty()) {
    ORBIT_CUDA(cudaMalloc(&p->d_ops, sizeof(DevOp) * dev.size()));
    ORBIT_CUDA(cudaMemcpy(p->d_ops, dev.data(), sizeof(DevOp) * dev.size(), cudaMemcpyHostToDevice));
  }
  return ORBIT_OK;
}

// Enqueues one turn.  prologue: run P_0 first.  wrap: end with the pass
// that also applies M_0 of the next turn and its extrema scan.
static int enqueue_turn(orbit_program_t* p, orbit_bunch_t* bu, cudaStream_t s, const Plan& plan, bool prologue,
                        bool wrap, int* nl) {
  const DevOp* ops = p->d_ops;
  MapCtx m = make_ctx(bu->sync);
  int nsc = (int)plan.sc_idx.size();
  bool sc_active = bu->n >= 2;  // SpaceChargeCalc2p5D.cc:79-80
  auto calc_of = [&](int i) -> orbit_sc2p5d_t* { return p->calcs[p->ops[plan.sc_idx[i]].i0]; };
  auto len_of = [&](int i) -> double { return p->ops[plan.sc_idx[i]].d[0]; };
  auto pipe_of = [&](int i) -> double { return p->ops[plan.sc_idx[i]].d[1]; };
  int rc;
  // the first pass of the run stores 1/(1+dp_p); later passes load it and
  // store it again only when their ops change dE
  bool first = true;
  // (a 2.5Drb kick at the start of a pass also changes dE)
  auto km_of = [&](const Seg& sg, bool sc, orbit_sc2p5d_t* kc = nullptr) -> int {
    if (!sc && sg.a == sg.b) return 0;  // enqueue_pass launches nothing
    bool dE = sg.dE || (kc && kc->rb);
    int km = first ? (int)KNL_STORE : (KNL_LOAD | (dE ? KNL_STORE : 0));
    first = false;
    return km;
  };
  double* knl = p->d_knl;
  auto bnd_of = [&](int i) -> const orbit_boundary* {
    int k = p->ops[plan.sc_idx[i]].i1;
    return (k >= 1 && k <= (int)p->bnds.size()) ? p->bnds[k - 1] : nullptr;
  };
  if (nsc == 0 || !sc_active) {
    // no kicks: one pass over all maps of the turn
    for (size_t i = 0; i < plan.segs.size(); ++i) {
      rc = enqueue_pass(bu, s, ops, plan.segs[i], m, nullptr, 0.0, nullptr, nullptr, nullptr, false, knl,
                        km_of(plan.segs[i], false), nl);
      if (rc) return rc;
    }
    return ORBIT_OK;
  }
  if (prologue) {
    rc = enqueue_pass(bu, s, ops, plan.segs[0], m, nullptr, 0.0, nullptr, calc_of(0), bnd_of(0), true, knl,
                      km_of(plan.segs[0], true), nl);
    if (rc) return rc;
  }
  for (int i = 0; i < nsc; ++i) {
    const bool last = (i == nsc - 1);
    const Seg& sg = !last ? plan.segs[i + 1] : (wrap ? plan.wrap : plan.segs[nsc]);
    orbit_sc2p5d_t* kc = calc_of(i);
    const int km = km_of(sg, true, kc);
    PrepJob job;
    std::memset(&job, 0, sizeof(job));
    if (fixed_pass(sg, kc->form == ORBIT_FORM_PLAIN && !kc->rb, km)) {
      job.ops = ops; job.a = sg.a; job.b = sg.b;
      for (int q = 0; q < 4; ++q) job.c[q] = bu->coord(q);
      job.n = bu->n;
      job.dp_p_coeff = m.dp_p_coeff;
      job.host_factor = sc_host_factor(bu->sync, len_of(i));
      job.out = kc->d_prep;
    }
    rc = sc_enqueue_kick(kc, bu, len_of(i), s, false, false, nl, pipe_of(i), bnd_of(i), &job);
    if (rc) return rc;
    // the last pass of a turn that another one follows also applies M_0 and
    // scans for the next turn's first kick
    orbit_sc2p5d_t* ec = !last ? calc_of(i + 1) : (wrap ? calc_of(0) : nullptr);
    rc = enqueue_pass(bu, s, ops, sg, m, kc, len_of(i), bnd_of(i), ec, !last ? bnd_of(i + 1) : bnd_of(0), !last, knl,
                      km, nl);
    if (rc) return rc;
  }
  return ORBIT_OK;
}

static int capture(orbit_program_t* p, orbit_bunch_t* bu, const Plan& plan, bool prologue, bool wrap,
                   cudaGraphExec_t* out, int* nl) {
  cudaStream_t s = bu->stream;
  for (auto c : p->calcs) sc_clear_pending(c);
  ORBIT_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  int rc = enqueue_turn(p, bu, s, plan, prologue, wrap, nl);
  for (auto c : p->calcs) sc_clear_pending(c);
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaStreamEndCapture(s, &g);
  if (rc) {
    if (g) cudaGraphDestroy(g);
    return rc;
  }
  if (e != cudaSuccess) return cuda_error(e, "cudaStreamEndCapture");
  e = cudaGraphInstantiate(out, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return cuda_error(e, "cudaGraphInstantiate");
  return ORBIT_OK;
}

static int prepare(orbit_program_t* p, orbit_bunch_t* bu) {
  auto dnv = [](const orbit_sc2p5d_t* c) { return c && c->dn ? dn_version(c->dn) : 0ull; };
  bool same = p->key_bunch == bu && p->key_n == bu->n && p->key_coords == bu->d_coords &&
              p->key_msize == bu->has_msize && sync_equal(p->key_sync, bu->sync) && p->g_mid &&
              p->key_gen.size() == p->calcs.size() && p->key_dnv.size() == p->calcs.size();
  for (size_t i = 0; same && i < p->calcs.size(); ++i)
    same = p->key_gen[i] == (p->calcs[i] ? p->calcs[i]->cfg_gen : 0ull) && p->key_dnv[i] == dnv(p->calcs[i]);
  if (same) return ORBIT_OK;
  free_graphs(p);
  for (auto c : p->calcs)
    if (c && c->dn) {
      int prc = dn_prepare_capture(c->dn);
      if (prc) return prc;
    }
  Plan plan;
  int rc = compile(p, bu, plan);
  if (rc) return rc;
  int nl = 0;
  rc = capture(p, bu, plan, true, true, &p->g_first, &nl);
  if (!rc) { nl = 0; rc = capture(p, bu, plan, false, true, &p->g_mid, &nl); }
  if (!rc) { p->launches_per_turn = nl; nl = 0; rc = capture(p, bu, plan, false, false, &p->g_last, &nl); }
  if (!rc) { nl = 0; rc = capture(p, bu, plan, true, false, &p->g_single, &nl); }
  if (rc) { free_graphs(p); return rc; }
  p->key_bunch = bu;
  p->key_n = bu->n;
  p->key_coords = bu->d_coords;
  p->key_sync = bu->sync;
  p->key_msize = bu->has_msize;
  p->key_gen.resize(p->calcs.size());
  p->key_dnv.resize(p->calcs.size());
  for (size_t i = 0; i < p->calcs.size(); ++i) {
    p->key_gen[i] = p->calcs[i] ? p->calcs[i]->cfg_gen : 0ull;
    p->key_dnv[i] = dnv(p->calcs[i]);
  }
  return ORBIT_OK;
}

}  // namespace orbit

extern "C" {

int orbit_program_create(orbit_program_t** out, const orbit_op_t* ops, int nops, orbit_sc2p5d_t* const* calcs,
                         int ncalcs) {
  if (!out || nops < 0 || (nops > 0 && !ops) || ncalcs < 0 || (ncalcs > 0 && !calcs))
    return set_error(ORBIT_ERR_ARG, "orbit_program_create: bad argument");
  int arc = init_pass_attrs();
  if (arc) return arc;
  num_sms();
  orbit_program_t* p = new orbit_program_t();
  p->ops.assign(ops, ops + nops);
  p->calcs.assign(calcs, calcs + ncalcs);
  for (auto& o : p->ops) {
    if (o.code == ORBIT_OP_SC && (o.i0 < 0 || o.i0 >= ncalcs || !p->calcs[o.i0])) {
      delete p;
      return set_error(ORBIT_ERR_ARG, "orbit_program_create: SC op refers to a missing calculator");
    }
  }
  cudaError_t e = cudaEventCreateWithFlags(&p->done, cudaEventDisableTiming);
  if (e != cudaSuccess) {
    delete p;
    return cuda_error(e, "orbit_program_create");
  }
  *out = p;
  return ORBIT_OK;
}

int orbit_program_set_boundaries(orbit_program_t* p, orbit_boundary_t* const* bnds, int n) {
  if (!p || n < 0 || (n > 0 && !bnds)) return set_error(ORBIT_ERR_ARG, "orbit_program_set_boundaries: bad argument");
  for (int i = 0; i < n; ++i) {
    int init = 0;
    if (!bnds[i] || orbit_boundary_info(bnds[i], nullptr, nullptr, nullptr, nullptr, &init) || !init)
      return set_error(ORBIT_ERR_ARG, "Boundary2D: the boundary was not initialized, call initialize()");
    int rc = bnd_ensure_device(bnds[i]);
    if (rc) return rc;
  }
  if (p->used) ORBIT_CUDA(cudaEventSynchronize(p->done));
  p->bnds.assign(bnds, bnds + n);
  free_graphs(p);
  p->key_bunch = nullptr;
  return ORBIT_OK;
}

int orbit_program_destroy(orbit_program_t* p) {
  if (!p) return ORBIT_OK;
  if (p->used) cudaEventSynchronize(p->done);  // graphs in flight read d_ops
  if (p->done) cudaEventDestroy(p->done);
  free_graphs(p);
  if (p->d_ops) cudaFree(p->d_ops);
  if (p->d_knl) cudaFree(p->d_knl);
  delete p;
  return ORBIT_OK;
}

int orbit_program_run(orbit_program_t* p, orbit_bunch_t* b, int turns) {
  int rc = orbit_program_enqueue(p, b, turns);
  if (rc) return rc;
  return check_status(b);
}

int orbit_program_enqueue(orbit_program_t* p, orbit_bunch_t* b, int turns) {
  ORBIT_NVTX("lattice program turns");
  if (!p || !b || turns < 0) return set_error(ORBIT_ERR_ARG, "orbit_program_enqueue: bad argument");
  if (turns == 0) return ORBIT_OK;
  // work already queued on a calculator by another bunch comes first
  for (auto c : p->calcs)
    ORBIT_CUDA(sc_order_before(c, b->stream));
  int rc = prepare(p, b);
  if (rc) return rc;
  if (turns == 1) {
    ORBIT_CUDA(cudaGraphLaunch(p->g_single, b->stream));
  } else {
    ORBIT_CUDA(cudaGraphLaunch(p->g_first, b->stream));
    for (int t = 1; t < turns - 1; ++t) ORBIT_CUDA(cudaGraphLaunch(p->g_mid, b->stream));
    ORBIT_CUDA(cudaGraphLaunch(p->g_last, b->stream));
  }
  for (auto c : p->calcs) ORBIT_CUDA(sc_mark_used(c, b->stream));
  p->used = true;
  ORBIT_CUDA(cudaEventRecord(p->done, b->stream));
  // SyncPart time, advanced in op order as each map would (teapotbase.cc:165)
  for (int t = 0; t < turns; ++t)
    for (double a : p->time_adv)
      if (a != 0.0) b->sync.time = b->sync.time + a;
  return ORBIT_OK;
}

int orbit_program_profile(orbit_program_t* p, orbit_bunch_t* b, int max_kinds, char* names, double* total_ms,
                          int* launches, int* nkinds) {
  if (!p || !b || max_kinds <= 0 || !names || !total_ms || !launches || !nkinds)
    return set_error(ORBIT_ERR_ARG, "orbit_program_profile: bad argument");
  for (auto c : p->calcs)
    ORBIT_CUDA(sc_order_before(c, b->stream));
  // an eager (uncaptured) turn; the captured graphs are rebuilt on the next run
  ORBIT_CUDA(cudaStreamSynchronize(b->stream));
  free_graphs(p);
  p->key_bunch = nullptr;
  Plan plan;
  int rc = compile(p, b, plan);
  if (rc) return rc;
  Profiler* prof = prof_install();
  int nl = 0;
  rc = enqueue_turn(p, b, b->stream, plan, true, false, &nl);
  int rc2 = prof_collect(prof, max_kinds, names, total_ms, launches, nkinds);
  for (auto c : p->calcs) ORBIT_CUDA(sc_mark_used(c, b->stream));
  for (double a : p->time_adv)
    if (a != 0.0) b->sync.time = b->sync.time + a;
  if (rc) return rc;
  if (rc2) return rc2;
  return check_status(b);
}

int orbit_program_launches(const orbit_program_t* p, int* launches) {
  if (!p || !launches) return set_error(ORBIT_ERR_ARG, "orbit_program_launches: bad argument");
  *launches = p->launches_per_turn;
  return ORBIT_OK;
}

}  // extern "C"
