// Per-particle device routines of the 2.5D space-charge kick, shared by the
// stand-alone kernels (sc2p5d.cu) and the fused lattice passes (program.cu).
#pragma once

#include "common.cuh"
#include "fixlog.cuh"
#include "fixmap.cuh"
#include "softf64.cuh"
#include "sc2p5d.cuh"

namespace orbit {

// ---------------------------------------------------------------------
// extrema (BunchExtremaCalculator::getExtremaXYZ, src/utils/bunch/
// BunchExtremaCalculator.cc:37-83) on order-preserving integer keys
// ---------------------------------------------------------------------
struct ExtAcc {
  unsigned long long mn[3], mx[3];
  bool bad;
  __device__ __forceinline__ void init() {
    for (int c = 0; c < 3; ++c) { mn[c] = ~0ull; mx[c] = 0ull; }
    bad = false;
  }
  __device__ __forceinline__ void add(double x, double y, double z) {
    double v[3] = {x, y, z};
    for (int c = 0; c < 3; ++c) {
      unsigned long long k = dkey(v[c]);
      mn[c] = k < mn[c] ? k : mn[c];
      mx[c] = k > mx[c] ? k : mx[c];
    }
  }
  // After the last add: infinities and NaN are beyond every finite key, so one
  // among the particles shows in the extrema.
  __device__ __forceinline__ void finish() {
    for (int c = 0; c < 3; ++c)
      if (mn[c] <= mx[c] && (!dfinite_bits(dkey_inv(mn[c])) || !dfinite_bits(dkey_inv(mx[c])))) bad = true;
  }
};

// Magnitudes of a bunch (ScState::mag): largest high words of |xp|, |yp| and of
// |dE|.
struct MagAcc {
  unsigned pm, em;
  __device__ __forceinline__ void init() { pm = em = 0u; }
  static __device__ __forceinline__ unsigned hi(double v) {
    return (unsigned)__double2hiint(v) & 0x7fffffffu;
  }
  __device__ __forceinline__ void bound(double xp, double yp) { pm = max(pm, max(hi(xp), hi(yp))); }
};

// Block-wide reduction, one atomic per quantity per block.
__device__ __forceinline__ void mag_block_commit(const MagAcc& a, ScState* st) {
  __shared__ unsigned s_m[2][32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
  const unsigned full = 0xffffffffu, pm = __reduce_max_sync(full, a.pm), em = __reduce_max_sync(full, a.em);
  if (lane == 0) {
    s_m[0][w] = pm;
    s_m[1][w] = em;
  }
  __syncthreads();
  if (w == 0) {
    const unsigned r0 = __reduce_max_sync(full, lane < nw ? s_m[0][lane] : 0u);
    const unsigned r1 = __reduce_max_sync(full, lane < nw ? s_m[1][lane] : 0u);
    if (lane == 0) atomicMax(&st->acc_pmax, r0);
    if (lane == 1) atomicMax(&st->acc_emax, r1);
  }
}

// Static shared memory of mag_block_commit, ext_block_commit and last_block_done.
static const size_t kCommitSmem = 32 * (2 * sizeof(unsigned) + 6 * sizeof(unsigned long long)) + 16;

// Smallest 64-bit key of a warp, from two 32-bit reductions.
__device__ __forceinline__ unsigned long long warp_min_key(unsigned long long k) {
  const unsigned h = __reduce_min_sync(0xffffffffu, (unsigned)(k >> 32));
  const unsigned l = __reduce_min_sync(0xffffffffu, (unsigned)(k >> 32) == h ? (unsigned)k : ~0u);
  return ((unsigned long long)h << 32) | l;
}

// Block-wide reduction, then one atomic per key per block (a maximum is the
// complement's minimum).
__device__ __forceinline__ void ext_block_commit(ExtAcc& a, ScState* st, unsigned* status) {
  a.finish();
  __shared__ unsigned long long s_k[6][32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    const unsigned long long lo = c == 0 ? a.mn[0] : c == 1 ? a.mn[1] : a.mn[2];
    const unsigned long long hi = c == 0 ? a.mx[0] : c == 1 ? a.mx[1] : a.mx[2];
    const unsigned long long v0 = warp_min_key(lo), v1 = warp_min_key(~hi);
    if (lane == 0) {
      s_k[2 * c][w] = v0;
      s_k[2 * c + 1][w] = v1;
    }
  }
  const int bad = __syncthreads_or(a.bad);
#pragma unroll 1
  for (int k = w; k < 6; k += nw) {
    const unsigned long long v = warp_min_key(lane < nw ? s_k[k][lane] : ~0ull);
    if (lane == 0) {
      if (k & 1) atomicMax(&st->key[k], ~v);
      else atomicMin(&st->key[k], v);
    }
  }
  if (threadIdx.x == 0 && bad) atomicOr(status, (unsigned)ST_NAN);
}

// ---------------------------------------------------------------------
// Grid set-up of bunchAnalysis (SpaceChargeCalc2p5D.cc:126-216), run by
// one warp of the last block of the kernel that scanned the extrema.
// ---------------------------------------------------------------------
// Explicitly rounded operations (no contraction), so that the grid limits
// and the persistent xy_ratio evolve exactly as the reference's.  The keys
// and the status word were written by atomics of other blocks: they are
// read from L2.
//
// The set-up is a chain of divisions on the critical path of every kick.  They
// run on the integer pipes (sf::div, correctly rounded as the instruction);
// every lane follows the same steps, and divisions that do not hang on one
// another go to different lanes of one division (four in a row instead of
// fourteen); halves are products by 0.5 (the same value), and the logarithm of
// the solver's scale is left to a block beside the forward rows.
static __device__ __noinline__ void sc_setup_warp(ScState* st, unsigned* status, const SetupArgs& sa) {
  const int lane = threadIdx.x & 31;
  unsigned long long key[6];
  for (int c = 0; c < 6; ++c) key[c] = __ldcg(&st->key[c]);
  const double xy0 = st->xy_ratio, sxmin = st->sxmin, sxmax = st->sxmax, symin = st->symin, symax = st->symax;
  const double sdx0 = st->sdx;
  const unsigned stat = __ldcg(status);
  // every load before the first store: one trip to L2, not one each
  const unsigned pmax = __ldcg(&st->acc_pmax), emax = __ldcg(&st->acc_emax);
  const int dirty = st->green_dirty;
  double xMin = dkey_inv(key[0]), xMax = dkey_inv(key[1]);
  double yMin = dkey_inv(key[2]), yMax = dkey_inv(key[3]);
  double zMin = dkey_inv(key[4]), zMax = dkey_inv(key[5]);
  __syncwarp();
  if (lane == 0) {
    for (int c = 0; c < 3; ++c) { st->key[2 * c] = ~0ull; st->key[2 * c + 1] = 0ull; }
    st->mag.pmax = pmax;
    st->mag.emax = emax;
    st->mag.xmax = fmax(fmax(fabs(xMin), fabs(xMax)), fmax(fabs(yMin), fabs(yMax)));
    st->acc_pmax = st->acc_emax = 0u;
    st->conv_bar[0] = 0u;
    st->conv_bar[1] = 0u;
  }
  if (sa.bnd) {
    // a boundary fixes the transverse grid to its extents; only z comes
    // from the bunch (SpaceChargeCalc2p5D.cc:174-196)
    xMin = sa.bxmin; xMax = sa.bxmax; yMin = sa.bymin; yMax = sa.bymax;
  }
  if (stat & ST_NAN) {
    // a non-finite coordinate was met by the extrema scan: no kick
    if (lane == 0) st->skip = 1;
    return;
  }
  if (!(xMin < xMax) || !(yMin < yMax) || !(zMin < zMax)) {  // :131 (also catches an empty scan)
    if (lane == 0) {
      st->skip = 1;
      atomicOr(status, (unsigned)ST_EXTENT);
    }
    return;
  }
  // lane q divides num by den; the quotients of lanes 0..3
  auto div4 = [](double n0, double d0, double n1, double d1, double n2, double d2, double n3, double d3, double q[4]) {
    const int l = threadIdx.x & 3;
    const double v = sf::div(l == 0 ? n0 : l == 1 ? n1 : l == 2 ? n2 : n3, l == 0 ? d0 : l == 1 ? d1 : l == 2 ? d2 : d3);
    for (int k = 0; k < 4; ++k) q[k] = __shfl_sync(0xffffffffu, v, k);
  };
  double q[4];
  double xy = xy0;
  div4(__dsub_rn(xMax, xMin), __dsub_rn(yMax, yMin), __dsub_rn(sxmax, sxmin), __dsub_rn(symax, symin),
       __dsub_rn(zMax, zMin), (double)sa.nz, 1.0, 1.0, q);
  const double ratio_beam = q[0], sr = q[1], dz = q[2];
  int set_solver = 0;
  if (sa.bnd) {
    xy = ratio_beam;  // :180
  } else if (sa.rb || fabs(__dsub_rn(ratio_beam, xy)) < __dmul_rn(0.25, xy)) {
    // :152-168; SpaceChargeCalc2p5Drb::bunchAnalysis (SpaceChargeCalc2p5Drb.cc:188-203)
    // always stretches to the calculator's own ratio, which never changes
    const double rr = sf::div(ratio_beam, xy);
    double width, center;
    if (ratio_beam > xy) {
      center = __dmul_rn(__dadd_rn(yMax, yMin), 0.5);
      width = __dmul_rn(__dmul_rn(__dsub_rn(yMax, yMin), rr), 0.5);
      yMin = __dsub_rn(center, width);
      yMax = __dadd_rn(center, width);
    } else {
      center = __dmul_rn(__dadd_rn(xMax, xMin), 0.5);
      width = __dmul_rn(sf::div(__dsub_rn(xMax, xMin), rr), 0.5);
      xMin = __dsub_rn(center, width);
      xMax = __dadd_rn(center, width);
    }
  } else {  // :169-173
    xy = ratio_beam;
    set_solver = 1;
  }
  // Grid2D::setGridX/Y (Grid2D.cc:422-433), Grid1D::setGridZ (Grid1D.cc:89-94)
  div4(__dsub_rn(xMax, xMin), (double)(sa.nx - 1), __dsub_rn(yMax, yMin), (double)(sa.ny - 1),
       __dsub_rn(xMax, xMin), __dsub_rn(yMax, yMin), 1.0, dz, q);
  const double dx = q[0], dy = q[1], inv_dz = q[3];
  if (!sa.bnd && !sa.rb && !set_solver) xy = q[2];
  // solver-shape check (SpaceChargeCalc2p5D.cc:208-216); the 2.5Drb
  // calculator keeps its solver grid
  if (!set_solver && !sa.rb && fabs(__dsub_rn(sr, xy)) > 0.00000001) set_solver = 1;
  div4(1.0, dx, 1.0, dy, set_solver ? dx : sdx0, dx, 1.0, 1.0, q);
  if (lane != 0) return;
  st->xmin = xMin; st->xmax = xMax; st->ymin = yMin; st->ymax = yMax;
  st->dx = dx; st->dy = dy; st->inv_dx = q[0]; st->inv_dy = q[1];
  st->zmin = zMin; st->zmax = zMax; st->dz = dz; st->inv_dz = inv_dz;
  if (!sa.rb) st->xy_ratio = xy;
  if (set_solver) {  // PoissonSolverFFT2D::setGridXY (PoissonSolverFFT2D.cc:103-111)
    st->sxmin = xMin; st->sxmax = xMax; st->symin = yMin; st->symax = yMax;
    st->sdx = dx; st->sdy = dy;
    st->green_dirty = 1;
  }
  st->scale_arg = q[2];  // its logarithm: PoissonSolverFFT2D.cc:213
  st->inv_qscale = sa.inv_qscale;
  st->phi_absmax = 0ull;
  st->lam_absmax = 0ull;
  if (sa.cond) cudaGraphSetConditional(sa.cond, (set_solver || dirty) ? 1u : 0u);
  st->skip = 0;
}

// True in exactly one of the nblk blocks that share `counter` (all blocks
// of the grid, or of one bunch of a batched launch): the last to call it.
// Every thread's earlier global writes and atomics come before the block is
// counted (one fence behind the barrier, where every thread's own waited for all
// its stores); `counter` is left at zero for the next launch.
__device__ __forceinline__ bool last_block_done(unsigned* counter, unsigned nblk) {
  __shared__ int s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();  // cumulative: what the barrier ordered before it, too
    unsigned prev = atomicAdd(counter, 1u);
    s_last = prev == nblk - 1;
    if (s_last) {
      *counter = 0u;
      __threadfence();
    }
  }
  __syncthreads();
  return s_last != 0;
}

// Waits until *cnt reaches n, for at most `polls` polls; a wait that runs out
// sets ST_SYNC and returns 0.  One thread; what the others wrote before they
// arrived is visible after it.
__device__ __forceinline__ int counter_wait(unsigned* cnt, unsigned n, long long polls, unsigned* status) {
  int ok = 1;
  long long i = 0;
  for (;;) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(cnt) : "memory");
    if (v >= n) break;
    if (++i > polls) {
      ok = 0;
      break;
    }
    __nanosleep(32);
  }
  if (!ok) atomicOr(status, (unsigned)ST_SYNC);
  __threadfence();
  return ok;
}

// Extrema commit followed, in the last of the nblk blocks scanning this
// bunch, by the grid set-up.
__device__ __forceinline__ void ext_commit_and_setup(ExtAcc& a, ScState* st, unsigned* status,
                                                     const SetupArgs& sa, unsigned nblk) {
  ext_block_commit(a, st, status);
  if (last_block_done(&st->ext_count, nblk) && threadIdx.x < 32) sc_setup_warp(st, status, sa);
}

// ---------------------------------------------------------------------
// 9-point TSC weights (Grid2D.cc:147-156, 220-233)
// ---------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void tsc_index(T t, int n, int& ind, T& frac) {
  // ind = int(t + 0.5) clamped to [1, n-2]; frac = t - ind  (Grid2D.cc:337-349)
  int i = (int)(t + (T)0.5);
  i = i < 1 ? 1 : i;
  i = i > n - 2 ? n - 2 : i;
  ind = i;
  frac = t - (T)i;
}

template <typename T>
__device__ __forceinline__ void tsc_weights(T f, T& wm, T& w0, T& wp) {
  T f2 = f * f;
  wm = (T)0.5 * ((T)0.25 - f + f2);
  w0 = (T)0.75 - f2;
  wp = (T)0.5 * ((T)0.25 + f + f2);
}

// ---------------------------------------------------------------------
// line density index (Grid1D::getIndAndWZ, Grid1D.cc:568-627)
// ---------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void g1_index(T z, T zmin, T inv_dz, int nz, int& i0, int& ip, T& w0, T& wp) {
  if (nz > 1) {
    T ind_dbl = (z - zmin) * inv_dz - (T)0.5;
    int iz0 = (int)ind_dbl;
    iz0 = iz0 > nz - 1 ? nz - 1 : iz0;
    T zf = ind_dbl - (T)iz0;
    if (iz0 == 0 && zf < (T)0) {
      i0 = nz - 1; ip = 0; w0 = -zf; wp = (T)1 + zf;
      return;
    }
    if (iz0 == nz - 1) {
      if (zf > (T)0) { i0 = iz0; ip = 0; w0 = (T)1 - zf; wp = zf; return; }
      ip = iz0; i0 = nz - 2; w0 = -zf; wp = (T)1 + zf;
      return;
    }
    i0 = iz0; ip = iz0 + 1; w0 = (T)1 - zf; wp = zf;
    return;
  }
  i0 = 0; ip = 0; w0 = (T)1; wp = (T)0;
}

// ---------------------------------------------------------------------
// kick (SpaceChargeCalc2p5D.cc:104-119 with Grid2D::calcGradient and
// Grid1D::getValue)
// ---------------------------------------------------------------------
struct KickConst {
  double xmin, ymin, inv_dx, inv_dy, zmin, zmax, inv_dz, fac;
  // FP32 form: grid coordinates t = x inv_dx + c; the z range test on
  // order-preserving integer keys; the float constants.  f32: the grid
  // origin lies within four grid extents of the coordinate origin, so t is
  // formed in float from the coordinate converted on the integer pipes:
  // t = fma(xf, ih, ch) + fma(xf, il, cl), 1/dx = ih + il and c = ch + cl
  // as float pairs, so that no rounding of a per-kick constant shifts or
  // stretches the whole grid (the kick would then sample the field away
  // from where the deposit put the charge); what is left are the unbiased
  // roundings of x and of the two operations, a few 2^-24 x n cells.
  // Otherwise one FP64 FMA and a conversion per coordinate.
  double cx, cy, cz;
  unsigned long long kzmin, kzmax;
  float inv_dx_f, inv_dy_f, fac_f;
  float ihx, ilx, chx, clx, ihy, ily, chy, cly, ihz, ilz, chz, clz;
  int f32;
  int nx, ny, nz;
  int skip;
};

// v as a float pair hi + lo (hi = float(v), lo = float(v - hi)).
__device__ __forceinline__ void split_f(double v, float& hi, float& lo) {
  hi = (float)v;
  lo = (float)(v - (double)hi);
}

// Grid coordinate of the FP32 form from a float coordinate and the float
// pairs of 1/dx and the offset.
__device__ __forceinline__ float grid_t_f32(float xf, float ih, float il, float ch, float cl) {
  return fmaf(xf, ih, ch) + fmaf(xf, il, cl);
}

// Whether the FP32 form's grid coordinates can be formed in float (see
// KickConst::f32).
__device__ __forceinline__ int grid_f32_ok(double cx, double cy, double cz, int nx, int ny, int nz) {
  return fabs(cx) <= 4.0 * nx && fabs(cy) <= 4.0 * ny && fabs(cz) <= 4.0 * nz + 4.0;
}

// f32: also the FP32 form's constants (a dozen FP64 operations the plain
// form does not need; one thread computes them while the block waits).
__device__ __forceinline__ void load_kick_const(KickConst& k, const ScState* st, double host_factor,
                                                int nx, int ny, int nz, bool f32 = true) {
  k.xmin = st->xmin; k.ymin = st->ymin; k.inv_dx = st->inv_dx; k.inv_dy = st->inv_dy;
  k.zmin = st->zmin; k.zmax = st->zmax; k.inv_dz = st->inv_dz;
  // factor = 2 L r_c/(beta^2 gamma^3) / (z_step * totalMacrosize)  (:96-100)
  // (the sum may come from another block of the same launch: from L2)
  k.fac = sf::div(host_factor, __dmul_rn(st->dz, __ldcg(&st->total_m)));
  k.nx = nx; k.ny = ny; k.nz = nz;
  k.skip = st->skip;
  if (!f32) return;
  k.cx = -k.xmin * k.inv_dx;
  k.cy = -k.ymin * k.inv_dy;
  k.cz = -k.zmin * k.inv_dz;
  k.kzmin = dkey(k.zmin);
  k.kzmax = dkey(k.zmax);
  k.inv_dx_f = (float)k.inv_dx;
  k.inv_dy_f = (float)k.inv_dy;
  k.fac_f = (float)k.fac;
  split_f(k.inv_dx, k.ihx, k.ilx);
  split_f(k.cx, k.chx, k.clx);
  split_f(k.inv_dy, k.ihy, k.ily);
  split_f(k.cy, k.chy, k.cly);
  split_f(k.inv_dz, k.ihz, k.ilz);
  split_f(k.cz, k.chz, k.clz);
  k.f32 = grid_f32_ok(k.cx, k.cy, k.cz, nx, ny, nz);
}

// 2.5Drb longitudinal kick (SpaceChargeCalc2p5Drb.cc:132-154):
// dE += ez(z) * lsf * coeff(r^2), ez the smoothed derivative of the line
// density (Grid1D::getValue), r measured from the beam centre, coeff =
// 1 + 2 ln(R/a) - r^2/a^2 inside a = a_bunch, 2 ln R - ln r^2 outside.
struct RbConst {
  double xc, yc, a2, inv_a2, lin, lout, lsf;
};

__device__ __forceinline__ void load_rb_const(RbConst& r, const ScState* st, double lsf) {
  r.xc = st->rb_xc; r.yc = st->rb_yc; r.a2 = st->rb_a2; r.inv_a2 = st->rb_inv_a2;
  r.lin = st->rb_lin; r.lout = st->rb_lout; r.lsf = lsf;
}

__device__ __forceinline__ void kick_rb_long(const KickConst& k, const RbConst& r, const double* __restrict__ lamd,
                                             double x, double y, double z, double& dE) {
  double ez = 0.0;
  if (!(z < k.zmin || z > k.zmax)) {
    int i0, ip;
    double w0, wp;
    g1_index<double>(z, k.zmin, k.inv_dz, k.nz, i0, ip, w0, wp);
    ez = (k.nz > 1) ? (w0 * lamd[i0] + wp * lamd[ip]) : lamd[0];
  }
  double ddx = x - r.xc, ddy = y - r.yc;
  double r2 = ddx * ddx + ddy * ddy;
  double coeff = (r2 <= r.a2) ? r.lin - r2 / r.a2 : r.lout - log(r2);
  dE += ez * r.lsf * coeff;
}

// FP64 plain form: phi/lam may be in shared or global memory.
__device__ __forceinline__ void kick_plain(const KickConst& k, const double* __restrict__ phi,
                                           const double* __restrict__ lam, double x, double y, double z,
                                           double& xp, double& yp) {
  int ix, iy;
  double fx, fy;
  tsc_index<double>((x - k.xmin) * k.inv_dx, k.nx, ix, fx);
  tsc_index<double>((y - k.ymin) * k.inv_dy, k.ny, iy, fy);
  double wxm, wx0, wxp, wym, wy0, wyp;
  tsc_weights<double>(fx, wxm, wx0, wxp);
  tsc_weights<double>(fy, wym, wy0, wyp);
  // dW = -(0.5 - f), -2f, 0.5 + f  (Grid2D.cc:228-233)
  double dxm = fx - 0.5, dx0 = -2.0 * fx, dxp = 0.5 + fx;
  double dym = fy - 0.5, dy0 = -2.0 * fy, dyp = 0.5 + fy;
  const double* r0 = phi + (ix - 1) * k.ny + (iy - 1);
  const double* r1 = r0 + k.ny;
  const double* r2 = r1 + k.ny;
  double a00 = r0[0], a01 = r0[1], a02 = r0[2];
  double a10 = r1[0], a11 = r1[1], a12 = r1[2];
  double a20 = r2[0], a21 = r2[1], a22 = r2[2];
  // separable sums: rows weighted along y, then along x
  double s0 = wym * a00 + wy0 * a01 + wyp * a02;
  double s1 = wym * a10 + wy0 * a11 + wyp * a12;
  double s2 = wym * a20 + wy0 * a21 + wyp * a22;
  double t0 = dym * a00 + dy0 * a01 + dyp * a02;
  double t1 = dym * a10 + dy0 * a11 + dyp * a12;
  double t2 = dym * a20 + dy0 * a21 + dyp * a22;
  double gx = dxm * s0 + dx0 * s1 + dxp * s2;
  double gy = wxm * t0 + wx0 * t1 + wxp * t2;
  // lambda(z)  (Grid1D.cc:191-209)
  double lv = 0.0;
  if (!(z < k.zmin || z > k.zmax)) {
    int i0, ip;
    double w0, wp;
    g1_index<double>(z, k.zmin, k.inv_dz, k.nz, i0, ip, w0, wp);
    lv = (k.nz > 1) ? (w0 * lam[i0] + wp * lam[ip]) : lam[0];
  }
  double lf = -lv * k.fac;
  xp += gx * k.inv_dx * lf;
  yp += gy * k.inv_dy * lf;
}

// FP32 form: gradient and line density in FP32, accumulation into FP64.
__device__ __forceinline__ void kick_fp32(const KickConst& k, const float* __restrict__ phi,
                                          const float* __restrict__ lam, double x, double y, double z,
                                          double& xp, double& yp) {
  // the FP64 pipe bounds the pass: the coordinates converted to float on
  // the integer pipes (or one FMA and a conversion each, far from the
  // origin), the z range test on integer keys
  float tx, ty;
  if (k.f32) {
    tx = grid_t_f32(sf::to_float(x), k.ihx, k.ilx, k.chx, k.clx);
    ty = grid_t_f32(sf::to_float(y), k.ihy, k.ily, k.chy, k.cly);
  } else {
    tx = (float)fma(x, k.inv_dx, k.cx);
    ty = (float)fma(y, k.inv_dy, k.cy);
  }
  int ix, iy;
  float fx, fy;
  tsc_index<float>(tx, k.nx, ix, fx);
  tsc_index<float>(ty, k.ny, iy, fy);
  float wxm, wx0, wxp, wym, wy0, wyp;
  tsc_weights<float>(fx, wxm, wx0, wxp);
  tsc_weights<float>(fy, wym, wy0, wyp);
  float dxm = fx - 0.5f, dx0 = -2.0f * fx, dxp = 0.5f + fx;
  float dym = fy - 0.5f, dy0 = -2.0f * fy, dyp = 0.5f + fy;
  const float* r0 = phi + (ix - 1) * k.ny + (iy - 1);
  const float* r1 = r0 + k.ny;
  const float* r2 = r1 + k.ny;
  float a00 = r0[0], a01 = r0[1], a02 = r0[2];
  float a10 = r1[0], a11 = r1[1], a12 = r1[2];
  float a20 = r2[0], a21 = r2[1], a22 = r2[2];
  float s0 = wym * a00 + wy0 * a01 + wyp * a02;
  float s1 = wym * a10 + wy0 * a11 + wyp * a12;
  float s2 = wym * a20 + wy0 * a21 + wyp * a22;
  float t0 = dym * a00 + dy0 * a01 + dyp * a02;
  float t1 = dym * a10 + dy0 * a11 + dyp * a12;
  float t2 = dym * a20 + dy0 * a21 + dyp * a22;
  float gx = dxm * s0 + dx0 * s1 + dxp * s2;
  float gy = wxm * t0 + wx0 * t1 + wxp * t2;
  float lv = 0.0f;
  const unsigned long long kz = dkey(z);
  if (kz >= k.kzmin && kz <= k.kzmax) {
    float zt = k.f32 ? grid_t_f32(sf::to_float(z), k.ihz, k.ilz, k.chz, k.clz) : (float)fma(z, k.inv_dz, k.cz);
    int i0, ip;
    float w0, wp;
    g1_index<float>(zt, 0.0f, 1.0f, k.nz, i0, ip, w0, wp);
    lv = (k.nz > 1) ? (w0 * lam[i0] + wp * lam[ip]) : lam[0];
  }
  float lf = -lv * k.fac_f;
  xp += sf::from_float(gx * k.inv_dx_f * lf);
  yp += sf::from_float(gy * k.inv_dy_f * lf);
}

// ---------------------------------------------------------------------
// deposit (Grid2D::binValue, Grid2D.cc:141-166; Grid1D::binValue,
// Grid1D.cc:422-439)
// ---------------------------------------------------------------------
struct DepConst {
  double xmin, xmax, ymin, ymax, inv_dx, inv_dy, zmin, zmax, inv_dz;
  int nx, ny, nz;
  int skip;
};

__device__ __forceinline__ void load_dep_const(DepConst& d, const ScState* st, int nx, int ny, int nz) {
  d.xmin = st->xmin; d.xmax = st->xmax; d.ymin = st->ymin; d.ymax = st->ymax;
  d.inv_dx = st->inv_dx; d.inv_dy = st->inv_dy;
  d.zmin = st->zmin; d.zmax = st->zmax; d.inv_dz = st->inv_dz;
  d.nx = nx; d.ny = ny; d.nz = nz;
  d.skip = st->skip;
}

// A thread's first particle, the rest follow every nblk * blockDim: the blocks'
// warps take turns, so that the last, partial round spreads over all blocks.
// (With block after block, the 27,200 particles of 1e6 that 152 blocks of 640
// leave for an eleventh round were 42 blocks' alone.)  The FP64 pass keeps block
// after block: 16 kicks of the FP32 form 2597 us against 2665.
__device__ __forceinline__ int first_particle(int blk, int nblk) {
  return (((int)threadIdx.x >> 5) * nblk + blk) * 32 + ((int)threadIdx.x & 31);
}

// Copies n elements of global memory (written by an earlier kernel) into
// shared memory with asynchronous 16-byte copies (cp.async.cg: no
// registers held, every copy of the thread in flight at once), then applies
// f in place to the elements this thread copied, once they have landed
// (cp.async.wait_all waits for the thread's own copies).  Threads t0.. of
// the block take part.  Where either address is not 16-byte aligned the
// thread copies element by element instead.  Returns with this thread's
// elements final; the caller synchronises the block.
template <typename T, typename F>
__device__ __forceinline__ void copy_smem_async(T* s, const T* g, int n, F f, int t0) {
  const int t = (int)threadIdx.x - t0, nt = (int)blockDim.x - t0;
  if (t < 0) return;
  constexpr int E = 16 / (int)sizeof(T);  // elements per 16-byte copy
  const uint32_t sb = (uint32_t)__cvta_generic_to_shared(s);
  const bool aligned = ((sb | (uint32_t)(size_t)g) & 15u) == 0u;
  const int nb = aligned ? n / E : 0;
  for (int i = t; i < nb; i += nt)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sb + 16u * (uint32_t)i),
                 "l"(reinterpret_cast<const char*>(g) + 16 * (size_t)i)
                 : "memory");
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_all;" ::: "memory");
  for (int i = t; i < nb; i += nt) {
#pragma unroll
    for (int q = 0; q < E; ++q) s[i * E + q] = f(s[i * E + q]);
  }
  for (int i = nb * E + t; i < n; i += nt) s[i] = f(__ldcg(g + i));
}

// 64-bit accumulation grids.  Global: native 64-bit atomics.  Shared: each
// cell is a low and a high 32-bit word in two separate arrays (so that
// random cells spread over all 32 banks), added with native 32-bit atomics:
// the low word wraps modulo 2^32 and the add that wraps carries 1 into the
// high word, so hi * 2^32 + lo, read once all adds are done, is the exact
// sum modulo 2^64.
//
// row(i) addresses cell i for adds at i + j with j known to the compiler.
template <bool SHARED> struct GridAcc;

// v at the low word lo and the high word hi of a cell, as shared-memory
// addresses: two atomics and the carry between them (left to atomicAdd and a
// test for a high word of zero, a cell takes a branch besides).
__device__ __forceinline__ void add_lo_hi(unsigned lo, unsigned hi, unsigned long long v) {
  asm volatile(
      "{\n\t.reg .u32 o, c, h;\n\t"
      "atom.shared.add.u32 o, [%0], %2;\n\t"
      "add.cc.u32 c, o, %2;\n\t"
      "addc.u32 h, %3, 0;\n\t"
      "red.shared.add.u32 [%1], h;\n\t}" ::"r"(lo),
      "r"(hi), "r"((unsigned)v), "r"((unsigned)(v >> 32))
      : "memory");
}
struct SharedRow {
  unsigned lo, hi;
  __device__ __forceinline__ void add(int j, unsigned long long v) const { add_lo_hi(lo + 4 * j, hi + 4 * j, v); }
};

template <> struct GridAcc<false> {
  unsigned long long* p;
  struct Row {
    unsigned long long* p;
    __device__ __forceinline__ void add(int j, unsigned long long v) const { atomicAdd(p + j, v); }
  };
  __device__ __forceinline__ Row row(int i) const { return Row{p + i}; }
  __device__ __forceinline__ void add(int i, unsigned long long v) const { atomicAdd(p + i, v); }
  // every particle is deposited by the block that reads it
  __device__ __forceinline__ bool owns(int) const { return true; }
  __device__ __forceinline__ bool owns_outside() const { return true; }
};

template <> struct GridAcc<true> {
  unsigned* lo;  // low words; the high words are at lo + hi_off
  int hi_off;
  __device__ __forceinline__ SharedRow row(int i) const {
    const unsigned a = (unsigned)__cvta_generic_to_shared(lo) + 4 * i;
    return SharedRow{a, a + 4 * hi_off};
  }
  __device__ __forceinline__ void add(int i, unsigned long long v) const { row(i).add(0, v); }
  __device__ __forceinline__ unsigned long long get(int i) const {
    return ((unsigned long long)lo[hi_off + i] << 32) | lo[i];
  }
  __device__ __forceinline__ bool owns(int) const { return true; }
  __device__ __forceinline__ bool owns_outside() const { return true; }
};

// Rows r0..r1-1 of a grid too large for one block's shared memory, plus
// one halo row on each side (the 9-point stencil of a particle whose
// centre row is owned).  A particle is deposited by the block that owns its
// centre row, whole (its line-density contribution included); particles
// outside the transverse grid belong to the first band.  Cell i of the
// grid is local cell i - base, base = first local row * ny.
struct BandAcc {
  unsigned* lo;  // low words; the high words at lo + hi_off
  int hi_off;
  int base;
  int r0, r1;
  bool first;
  __device__ __forceinline__ SharedRow row(int i) const {
    const unsigned a = (unsigned)__cvta_generic_to_shared(lo) + 4 * (i - base);
    return SharedRow{a, a + 4 * hi_off};
  }
  __device__ __forceinline__ void add(int i, unsigned long long v) const { row(i).add(0, v); }
  __device__ __forceinline__ unsigned long long get(int i) const {
    return ((unsigned long long)lo[hi_off + i] << 32) | lo[i];
  }
  __device__ __forceinline__ bool owns(int ix) const { return ix >= r0 && ix < r1; }
  __device__ __forceinline__ bool owns_outside() const { return first; }
};

// Plain form: contributions are rounded to a fixed-point grid of step 1/S
// (S a power of two with S * total macrosize <= 2^62) and summed as 64-bit
// integers, so the deposit is exact and independent of summation order.
template <class RA, class ZA>
__device__ __forceinline__ void deposit_plain(const DepConst& d, const RA& rho, const ZA& zg, double x, double y,
                                              double z, double ms) {
  const bool in2 = !(x < d.xmin || x > d.xmax || y < d.ymin || y > d.ymax);
  int ix = 0, iy;
  double fx, fy;
  if (in2) tsc_index<double>((x - d.xmin) * d.inv_dx, d.nx, ix, fx);
  if (in2 ? !rho.owns(ix) : !rho.owns_outside()) return;  // another block's particle
  if (in2) {
    tsc_index<double>((y - d.ymin) * d.inv_dy, d.ny, iy, fy);
    double wxm, wx0, wxp, wym, wy0, wyp;
    tsc_weights<double>(fx, wxm, wx0, wxp);
    tsc_weights<double>(fy, wym, wy0, wyp);
    double ax[3] = {wxm * ms, wx0 * ms, wxp * ms};
    double wy[3] = {wym, wy0, wyp};
    const int base = (ix - 1) * d.ny + (iy - 1);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) rho.add(base + i * d.ny + j, (unsigned long long)__double2ll_rn(ax[i] * wy[j]));
  }
  if (!(z < d.zmin || z > d.zmax)) {
    int i0, ip;
    double w0, wp;
    g1_index<double>(z, d.zmin, d.inv_dz, d.nz, i0, ip, w0, wp);
    if (d.nz > 1) {
      zg.add(i0, (unsigned long long)__double2ll_rn(w0 * ms));
      zg.add(ip, (unsigned long long)__double2ll_rn(wp * ms));
    } else {
      zg.add(0, (unsigned long long)__double2ll_rn(ms));
    }
  }
}

// ---------------------------------------------------------------------
// Exact fixed-point arithmetic on the integer pipe (plain form).
//
// After one FP64 fused multiply-add per coordinate, v = t + 0.5 with
// t = (x - xmin)/dx in cell units, the index, the fraction and the 9-point
// weights are computed as 64-bit fixed-point integers: the fraction
// f = t - ind exactly as rounded into v (Q56), the weights W = (f -+ 0.5)^2/2
// and 0.75 - f^2 in Q58 (absolute error below 2^-58), the derivative
// weights exactly.  GB300 issues two FP64 FMAs per SM per cycle but dozens
// of integer operations, so this keeps the FP64 pipe for the coordinates.
// ---------------------------------------------------------------------

// v * 2^F truncated toward zero; false when |v| * 2^F could reach 2^63 or v
// is not finite.
__device__ __forceinline__ bool fix_of(double v, int F, long long& out) {
  long long u = __double_as_longlong(v);
  int e = (int)((u >> 52) & 0x7ff);
  long long m = (u & 0x000FFFFFFFFFFFFFll) | 0x0010000000000000ll;
  int sh = e - 1075 + F;
  long long r;
  if (e == 0) {
    r = 0;
  } else if (sh >= 0) {
    if (sh > 10) return false;
    r = m << sh;
  } else {
    r = (sh > -63) ? (m >> (-sh)) : 0;
  }
  out = (u < 0) ? -r : r;
  return true;
}

// Fraction bits F for values below n + 1 (n >= 2): v * 2^F < 2^63.
__host__ __device__ __forceinline__ int fix_bits(int n) {
  int b = 0;
  while ((1 << b) < n + 2) ++b;
  int F = 63 - b;
  return F > 60 ? 60 : F;
}

// g in Q56 with |g| <= 2^57: g^2 in Q58.
__device__ __forceinline__ long long sq_q58(long long g) {
  unsigned long long a = (unsigned long long)(g < 0 ? -g : g) << 5;
  return (long long)__umul64hi(a, a);
}

// Grid2D::getIndAndFracX/Y on v = t + 0.5: ind = floor(v) clamped to
// [1, n-2], f = t - ind in Q56.  False outside 0 <= floor(v) <= n-1.
__device__ __forceinline__ bool tsc_fixed(double v, int n, int F, int& ind, long long& f56) {
  long long V;
  // |f| <= 1.25 keeps every product below 2^63; particles inside the grid
  // limits have 0.5 <= v <= n - 0.5
  if (!fix_of(v, F, V) || V < (1ll << (F - 2)) || V > ((long long)n << F) - (1ll << (F - 2))) return false;
  long long i = V >> F;
  long long fr = V - (i << F) - (1ll << (F - 1));
  long long f = (F <= 56) ? (fr << (56 - F)) : (fr >> (F - 56));
  if (i < 1) { f -= (1ll << 56); i = 1; }
  if (i > n - 2) { f += (1ll << 56); i = n - 2; }
  ind = (int)i;
  f56 = f;
  return true;
}

// 9-point weights Wm, W0, Wp (Q58).
__device__ __forceinline__ void tsc_w_fixed(long long f, long long w[3]) {
  w[0] = sq_q58(f - (1ll << 55)) >> 1;
  w[1] = (3ll << 56) - sq_q58(f);
  w[2] = sq_q58(f + (1ll << 55)) >> 1;
}
// Grid1D index on u = (z - zmin)/dz + 0.5 (nz > 1): floor semantics with
// periodic neighbours reproduce every wrap rule of Grid1D::getIndAndWZ;
// wp (weight of ip) in Q56.
__device__ __forceinline__ bool g1_fixed(double u, int nz, int F, int& i0, int& ip, long long& wp56) {
  long long V;
  if (!fix_of(u, F, V) || V < 0) return false;
  long long i = V >> F;
  if (i > nz) return false;
  long long fr = V - (i << F);
  wp56 = (F <= 56) ? (fr << (56 - F)) : (fr >> (F - 56));
  int a = (int)i - 1;
  i0 = a < 0 ? nz - 1 : a;
  ip = (int)i >= nz ? 0 : (int)i;
  return true;
}

struct DepFix {
  unsigned long long kxmin, kxmax, kymin, kymax, kzmin, kzmax;  // ordered keys of the limits
  double ax, cx, ay, cy, az, cz;   // v = x * ax + cx etc.
  int nx, ny, nz, Fx, Fy, Fz, K;
  int skip;
};

__device__ __forceinline__ void load_dep_fix(DepFix& d, const ScState* st, int nx, int ny, int nz, int K) {
  d.kxmin = dkey(st->xmin); d.kxmax = dkey(st->xmax);
  d.kymin = dkey(st->ymin); d.kymax = dkey(st->ymax);
  d.kzmin = dkey(st->zmin); d.kzmax = dkey(st->zmax);
  d.ax = st->inv_dx; d.cx = 0.5 - st->xmin * st->inv_dx;
  d.ay = st->inv_dy; d.cy = 0.5 - st->ymin * st->inv_dy;
  d.az = st->inv_dz; d.cz = 0.5 - st->zmin * st->inv_dz;
  d.nx = nx; d.ny = ny; d.nz = nz;
  d.Fx = fix_bits(nx); d.Fy = fix_bits(ny); d.Fz = fix_bits(nz);
  d.K = K;
  d.skip = st->skip;
}

// Integer deposit of one particle with unit weight scaled by 2^K (the
// macrosize multiplies the grid afterwards).  Returns false when the
// particle needs the FP64 path (never for finite coordinates in range).
// SHARED: the grids are block-private shared memory.
template <class RA, class ZA>
__device__ __forceinline__ bool deposit_fixed(const DepFix& d, const RA& rho, const ZA& zg, double x, double y,
                                              double z) {
  unsigned long long kx = dkey(x), ky = dkey(y), kz = dkey(z);
  bool in2 = kx >= d.kxmin && kx <= d.kxmax && ky >= d.kymin && ky <= d.kymax;
  bool in1 = kz >= d.kzmin && kz <= d.kzmax;
  int ix = 0, iy = 0, i0 = 0, ip = 0;
  long long fx = 0, fy = 0, wp = 0;
  if (in2) {
    if (!tsc_fixed(fma(x, d.ax, d.cx), d.nx, d.Fx, ix, fx)) return false;
    if (!tsc_fixed(fma(y, d.ay, d.cy), d.ny, d.Fy, iy, fy)) return false;
  }
  if (in1 && d.nz > 1) {
    if (!g1_fixed(fma(z, d.az, d.cz), d.nz, d.Fz, i0, ip, wp)) return false;
  }
  if (in2 ? !rho.owns(ix) : !rho.owns_outside()) return true;  // another block's particle
  if (in2) {
    long long wx[3], wy[3];
    tsc_w_fixed(fx, wx);
    tsc_w_fixed(fy, wy);
    const int sh = 60 - d.K;
    const long long half = 1ll << (sh - 1);
    const int base = (ix - 1) * d.ny + (iy - 1);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      long long a = wx[i] << 4;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        long long p = __mul64hi(a, wy[j] << 4);  // Wx Wy in Q60
        rho.add(base + i * d.ny + j, (unsigned long long)((p + half) >> sh));
      }
    }
  }
  if (in1) {
    const int sh = 56 - d.K;
    const long long half = 1ll << (sh - 1);
    if (d.nz > 1) {
      zg.add(i0, (unsigned long long)((((1ll << 56) - wp) + half) >> sh));
      zg.add(ip, (unsigned long long)((wp + half) >> sh));
    } else {
      zg.add(0, (unsigned long long)(1ll << d.K));
    }
  }
  return true;
}

// The constants of a block's deposit: v 2^F is the coordinate in cells plus
// 1/2, x a + c for a uniform macrosize and (x - c) a + 2^(F-1) for others (as
// deposit_fixed and deposit_plain round it), its high word within [lo, lo + span] where the particle is
// surely inside the grid's limits.
struct DepFast {
  double a[3], c[3];
  int F[3], lo[3];
  unsigned span[3];
  int none;               // every particle goes the general way
  double min[3], max[3];  // the limits themselves
};

// g: extra bits of a per-particle macrosize (K = 0): about 2^58 units at the
// mean of n particles; 0: none fit, every particle goes the general way.
__host__ __device__ __forceinline__ int dep_ms_bits(int n) {
  int b = 0;
  while (b < 30 && (n >> (b + 1)) != 0) ++b;
  return b >= 9 ? b - 4 : 0;
}

// Executed by lanes 0..2 of one warp, one coordinate each.
__device__ __forceinline__ void load_dep_fast(DepFast* d, const ScState* st, int nx, int ny, int nz, int K, int n) {
  const int k = threadIdx.x;
  const int nc = k == 0 ? nx : k == 1 ? ny : nz;
  const double inv = k == 0 ? st->inv_dx : k == 1 ? st->inv_dy : st->inv_dz;
  const double mn = k == 0 ? st->xmin : k == 1 ? st->ymin : st->zmin;
  const int F = fix_bits(nc);
  const double scale = __hiloint2double((1023 + F) << 20, 0);
  const double c = 0.5 - mn * inv;
  d->a[k] = inv * scale;
  d->c[k] = K > 0 ? c * scale : mn;
  d->F[k] = F;
  d->min[k] = mn;
  d->max[k] = k == 0 ? st->xmax : k == 1 ? st->ymax : st->zmax;
  // cells [0, n - 1] of x and y, [0, nz] of z, less 2^(32 - F) at each end: far
  // above the rounding of v unless the grid lies 2^16 cells off the origin
  const int lo = (1 << (F - 33)) + 1;
  const int hi = (int)((((long long)nc << F) - (1ll << (F - 1))) >> 32) + (k == 2 ? 1 << (F - 32) : 0) - 1;
  d->lo[k] = lo;
  d->span[k] = (unsigned)(hi - lo);
  const bool ok = (K > 0 ? fabs(c) < 65536.0 : dep_ms_bits(n) > 0) && hi >= lo;
  const bool all = __all_sync(7u, ok);
  if (k == 0) d->none = !all;
}

// A particle next to a limit: inside all three, and its cell coordinate where
// deposit_fixed takes it.
static __device__ __noinline__ bool dep_edge(const DepFast* d, double x, double y, double z, int hx, int hy, int hz) {
  const double v[3] = {x, y, z};
  const int h[3] = {hx, hy, hz};
  bool in = true;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int q = 1 << (d->F[k] - 34);  // a quarter cell
    in = in && v[k] >= d->min[k] && v[k] <= d->max[k] && h[k] >= q && h[k] < d->lo[k] + (int)d->span[k] + q;
  }
  return in;
}

// One particle inside the grid.  MS: M is its macrosize in units of
// 2^-(g) / S, else every particle counts 2^K.  The sums are deposit_fixed's,
// bit for bit, for K > 0.  Returns false, with nothing done, for the others.
//
// Bound by the issue of instructions (with the fields of the doubles taken
// apart, keys compared and every product formed from unsigned halves a particle
// took 740): the conversions run on the otherwise idle FP64 pipe (three
// multiply-adds and three conversions, 64 clocks a warp each), one square gives
// the three weights, and the nine products take four multiply-adds each.  1e6
// particles, 128 x 128 x 64: 44 -> 27 us; 333,333 with their own macrosizes on
// 96 x 80 x 48, whose FP64 sums became integer ones: 60 -> 25 us.
template <bool MS, class RA, class ZA>
__device__ __forceinline__ bool deposit_fast(const DepFast& d, const DepFast* sd, const RA& rho, const ZA& zg, double x, double y,
                                             double z, long long M, int nx, int ny, int nz, int K) {
  auto cells = [&](double v, int k) -> long long {
    if (MS) return __double2ll_rz((v - d.c[k]) * d.a[k]) + (1ll << (d.F[k] - 1));
    return __double2ll_rz(fma(v, d.a[k], d.c[k]));
  };
  const long long vx = cells(x, 0), vy = cells(y, 1), vz = cells(z, 2);
  const int hx = (int)(vx >> 32), hy = (int)(vy >> 32), hz = (int)(vz >> 32);
  const bool in = ((unsigned)(hx - d.lo[0]) <= d.span[0]) & ((unsigned)(hy - d.lo[1]) <= d.span[1]) &
                  ((unsigned)(hz - d.lo[2]) <= d.span[2]);
  if (!in && !dep_edge(sd, x, y, z, hx, hy, hz)) return false;
  if (MS && !fx::within(M, 1 << 29)) return false;
  const int ix = min(max(hx >> (d.F[0] - 32), 1), nx - 2), iy = min(max(hy >> (d.F[1] - 32), 1), ny - 2);
  if (!rho.owns(ix)) return true;  // another block's particle
  // f = v - i - 1/2 in Q61, to 2^-56
  auto frac = [](long long v, int F, int i) {
    const unsigned long long t = (unsigned long long)v << (62 - F);
    const long long f = (long long)(t - ((unsigned long long)(unsigned)((i << 30) + (1 << 29)) << 32));
    return (f >> 1) & ~31ll;
  };
  fx::V wx[3], wy[3];
  fx::tsc_weights_q58(frac(vx, d.F[0], ix), 4, wx);
  fx::tsc_weights_q58(frac(vy, d.F[1], iy), 1, wy);
  const fx::V m = fx::sp(M);
  int sh = 57 - K;  // products Wx Wy in Q57
  if (MS) {
    sh = K - 4;
#pragma unroll
    for (int i = 0; i < 3; ++i) wx[i] = fx::sp(fx::mul_floor(wx[i], m) << 3);  // 2 Wx M
  }
  const int half = 1 << (sh - 1);  // sh <= 28
  const int base = (ix - 1) * ny + (iy - 1);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const auto row = rho.row(base + i * ny);
#pragma unroll
    for (int j = 0; j < 3; ++j) row.add(j, (unsigned long long)(fx::mul_floor_r(wx[i], wy[j], half) >> sh));
  }
  if (nz > 1) {
    const int iz = hz >> (d.F[2] - 32);
    const long long w = (long long)(((unsigned long long)vz << (62 - d.F[2])) -
                                    ((unsigned long long)(unsigned)(iz << 30) << 32));  // Q62
    const int i0 = iz == 0 ? nz - 1 : iz - 1, ip = iz >= nz ? 0 : iz;
    if (MS) {
      const long long hz2 = 1ll << (K - 3);
      zg.add(i0, (unsigned long long)(fx::mul_floor(fx::sp((1ll << 62) - w), m, hz2) >> (K - 2)));
      zg.add(ip, (unsigned long long)(fx::mul_floor(fx::sp(w), m, hz2) >> (K - 2)));
    } else {
      const int sz = 56 - K;
      const long long hz1 = 1ll << (sz - 1), wp = w >> 6;
      zg.add(i0, (unsigned long long)(((1ll << 56) - wp + hz1) >> sz));
      zg.add(ip, (unsigned long long)((wp + hz1) >> sz));
    }
  } else {
    zg.add(0, MS ? (unsigned long long)((M + (1ll << (K - 1))) >> K) : 1ull << K);
  }
  return true;
}

// A particle outside the grid, or whose macrosize is far above the mean: the
// general way.
template <class RA, class ZA>
struct DepSlow {
  RA rho;
  ZA zg;
  const ScState* st;
  const double* c[3];
  const double* msize;
  double ms_uniform, qscale;
  int nx, ny, nz, K;
};

template <class RA, class ZA>
__device__ __noinline__ void deposit_slow(const DepSlow<RA, ZA>* s, int i) {
  const double x = s->c[0][i], y = s->c[1][i], z = s->c[2][i];
  if (s->K > 0) {
    DepFix df;
    load_dep_fix(df, s->st, s->nx, s->ny, s->nz, s->K);
    if (deposit_fixed(df, s->rho, s->zg, x, y, z)) return;
  }
  DepConst d;
  load_dep_const(d, s->st, s->nx, s->ny, s->nz);
  deposit_plain(d, s->rho, s->zg, x, y, z, s->msize ? s->msize[i] * s->qscale : s->ms_uniform);
}

// Deposits particle i one way or the other.  g: dep_ms_bits, q: qscale 2^g.
template <class RA, class ZA>
__device__ __forceinline__ void deposit_one(const DepFast& d, const DepFast* sd, const DepSlow<RA, ZA>* ss,
                                            const RA& rho, const ZA& zg, const double* __restrict__ x,
                                            const double* __restrict__ y, const double* __restrict__ z,
                                            const double* __restrict__ msize, int g, double q, int nx, int ny, int nz,
                                            int K, int i) {
  const bool done = K > 0 ? deposit_fast<false>(d, sd, rho, zg, x[i], y[i], z[i], 0, nx, ny, nz, K)
                          : deposit_fast<true>(d, sd, rho, zg, x[i], y[i], z[i], __double2ll_rn(msize[i] * q), nx, ny,
                                               nz, g);
  if (!done) deposit_slow(ss, i);
}

// The particles blk * blockDim + thread, ... of a block's deposit.
template <class RA, class ZA>
__device__ __forceinline__ void deposit_particles(const DepFast* sd, const DepSlow<RA, ZA>* ss, const RA& rho,
                                                  const ZA& zg, const double* __restrict__ x,
                                                  const double* __restrict__ y, const double* __restrict__ z,
                                                  const double* __restrict__ msize, int n, double qscale, int nx,
                                                  int ny, int nz, int K, int blk, int nblk) {
  const DepFast d = *sd;
  const int i0 = first_particle(blk, nblk), di = nblk * blockDim.x, g = dep_ms_bits(n);
  const double q = sf::pow2mul(qscale, g);
  if (d.none) {
    for (int i = i0; i < n; i += di) deposit_slow(ss, i);
  } else if (K > 0) {  // two loops: the test stays outside
    for (int i = i0; i < n; i += di) deposit_one(d, sd, ss, rho, zg, x, y, z, msize, g, q, nx, ny, nz, K, i);
  } else {
    for (int i = i0; i < n; i += di) deposit_one(d, sd, ss, rho, zg, x, y, z, msize, g, q, nx, ny, nz, 0, i);
  }
}

// Which particles a band looks at, by the order of the high words of the
// doubles alone (widened by 1/16 cell, so none of its own is missed): those
// whose centre row may be its own, and for the first band also those that may
// lie outside the transverse grid.  Centre rows are clamped to [1, nx - 2], so
// the owner of row 1 takes all below it and the owner of row nx - 2 all above.
struct BandKeys {
  int xlo, xhi, ylo, yhi, xout;
};

__device__ __forceinline__ int hi_key(double v) {
  const int h = __double2hiint(v);
  return h ^ ((h >> 31) & 0x7fffffff);
}

__device__ __forceinline__ void load_band_keys(BandKeys* k, const ScState* st, int nx, const BandAcc& a) {
  const double dx = 1.0 / st->inv_dx, dy = 1.0 / st->inv_dy;
  k->xlo = a.r0 <= 1 ? -0x7fffffff - 1 : hi_key(st->xmin + (a.r0 - 0.5625) * dx);
  k->xhi = a.r1 >= nx - 1 ? 0x7fffffff : hi_key(st->xmin + (a.r1 - 0.4375) * dx);
  k->ylo = a.first ? hi_key(st->ymin + 0.0625 * dy) : -0x7fffffff - 1;
  k->yhi = a.first ? hi_key(st->ymax - 0.0625 * dy) : 0x7fffffff;
  k->xout = a.first ? hi_key(st->xmax - 0.0625 * dx) : 0x7fffffff;
}

// The same particles for a band: a warp sets aside those that may be the
// band's own until it has 32, and deposits them together.  With every lane
// testing and depositing its own, a warp went through the whole deposit in
// every band for the lanes that own theirs: 835 against 572 us for 16e6
// particles on 256 x 256 in three bands.
static __device__ __forceinline__ void deposit_band_particles(const DepFast* sd, const DepSlow<BandAcc, GridAcc<true>>* ss,
                                                       const BandKeys* bk, int* queue, const BandAcc& rho,
                                                       const GridAcc<true>& zg, const double* __restrict__ x,
                                                       const double* __restrict__ y, const double* __restrict__ z,
                                                       const double* __restrict__ msize, int n, double qscale, int nx,
                                                       int ny, int nz, int K, int blk, int nblk) {
  const DepFast d = *sd;
  const BandKeys k = *bk;
  const int lane = threadIdx.x & 31, g = dep_ms_bits(n);
  const double q = sf::pow2mul(qscale, g);
  int* mine = queue + 64 * (threadIdx.x >> 5);
  int have = 0;
  auto flush = [&](int cnt) {
    __syncwarp();
    if (lane < cnt) {
      const int i = mine[lane];
      if (d.none) deposit_slow(ss, i);
      else if (K > 0) deposit_one(d, sd, ss, rho, zg, x, y, z, msize, g, q, nx, ny, nz, K, i);
      else deposit_one(d, sd, ss, rho, zg, x, y, z, msize, g, q, nx, ny, nz, 0, i);
    }
    __syncwarp();
  };
  const int di = nblk * blockDim.x;
  for (int i = first_particle(blk, nblk); i - lane < n; i += di) {
    bool own = false;
    if (i < n) {
      const int kx = hi_key(x[i]);
      own = kx >= k.xlo && kx <= k.xhi;
      if (rho.first && !own) {
        const int ky = hi_key(y[i]);
        own = kx >= k.xout || ky <= k.ylo || ky >= k.yhi;
      }
    }
    const unsigned m = __ballot_sync(0xffffffffu, own);
    if (own) mine[have + __popc(m & ((1u << lane) - 1u))] = i;
    have += __popc(m);
    if (have >= 32) {
      flush(32);
      have -= 32;
      if (lane < have) mine[lane] = mine[32 + lane];
      __syncwarp();  // the slots above `have` are written next
    }
  }
  flush(have);
}

// Fixed-point kick: phi and lambda as 64-bit integers with per-kick scales
// (phi * 2^sphi, lambda * 2^slam, both below 2^61).
struct KickFix {
  double ax, cx, ay, cy, az, cz;
  unsigned long long kzmin, kzmax;
  double gxs, gys;   // inv_dx * 2^-(sphi-5), inv_dy * 2^-(sphi-5)
  double lfs;        // -factor * 2^-(slam-2)
  int nx, ny, nz, Fx, Fy, Fz;
  int sphi, slam;
  int skip;
};

__device__ __forceinline__ int scale_bits(unsigned long long absmax_bits) {
  int e = (int)((absmax_bits >> 52) & 0x7ff);
  return absmax_bits == 0 ? 0 : 1083 - e;  // max * 2^s < 2^61
}

// fac: the kick factor of load_kick_const (the same division).
__device__ __forceinline__ void load_kick_fix(KickFix& k, const ScState* st, double fac, int nx, int ny, int nz) {
  k.ax = st->inv_dx; k.cx = 0.5 - st->xmin * st->inv_dx;
  k.ay = st->inv_dy; k.cy = 0.5 - st->ymin * st->inv_dy;
  k.az = st->inv_dz; k.cz = 0.5 - st->zmin * st->inv_dz;
  k.kzmin = dkey(st->zmin); k.kzmax = dkey(st->zmax);
  k.sphi = scale_bits(st->phi_absmax);
  k.slam = scale_bits(__ldcg(&st->lam_absmax));
  k.gxs = sf::pow2mul(st->inv_dx, 5 - k.sphi);
  k.gys = sf::pow2mul(st->inv_dy, 5 - k.sphi);
  k.lfs = sf::pow2mul(-fac, 2 - k.slam);
  k.nx = nx; k.ny = ny; k.nz = nz;
  k.Fx = fix_bits(nx); k.Fy = fix_bits(ny); k.Fz = fix_bits(nz);
  k.skip = st->skip;
}

__device__ __forceinline__ long long phi_fixed(double v, int s) {
  long long r;
  return fix_of(v, s, r) ? r : 0;
}

// A fixed-point grid value as the fx::V pair the kick multiplies (high word
// above, signed low word below).
__device__ __forceinline__ long long fx_pair(long long v) {
  const fx::V p = fx::sp(v);
  return (long long)(((unsigned long long)(unsigned)p.h << 32) | (unsigned)p.l);
}
__device__ __forceinline__ fx::V fx_of_pair(long long v) {
  fx::V p;
  p.l = (int)(unsigned)v;
  p.h = (int)(v >> 32);
  return p;
}

// Gradient of the fixed-point potential (Grid2D::calcGradient) at cell (ix,
// iy) and fractions fx, fy (Q62, |f| <= 1.25): gx, gy in Q(sphi-5) cells.
// The weights come from one square per axis, each row's two sums and the two
// column sums are rounded once (fx::mul3): about 90 instructions for the 24
// products against ~400 as separate 64-bit high products.
__device__ __forceinline__ void grad_fixed(const long long* __restrict__ P, int ny, int ix, int iy, long long fx_,
                                           long long fy_, long long& gx, long long& gy) {
  const fx::V fx1 = fx::sp(fx_), fy1 = fx::sp(fy_);
  const long long x2 = fx::mul(fx1, fx1) << 2, y2 = fx::mul(fy1, fy1) << 2;  // f^2, Q62
  const long long e8 = 1ll << 59, half = 1ll << 60;
  // W = (f -+ 1/2)^2 / 2, 3/4 - f^2 (Q62); dW = f -+ 1/2, -2 f (Q61)
  const fx::V wxm = fx::sp((x2 >> 1) - (fx_ >> 1) + e8), wx0 = fx::sp((3ll << 60) - x2), wxp = fx::sp((x2 >> 1) + (fx_ >> 1) + e8);
  const fx::V wym = fx::sp((y2 >> 1) - (fy_ >> 1) + e8), wy0 = fx::sp((3ll << 60) - y2), wyp = fx::sp((y2 >> 1) + (fy_ >> 1) + e8);
  const fx::V dxm = fx::sp((fx_ >> 1) - half), dx0 = fx::sp(-fx_), dxp = fx::sp((fx_ >> 1) + half);
  const fx::V dym = fx::sp((fy_ >> 1) - half), dy0 = fx::sp(-fy_), dyp = fx::sp((fy_ >> 1) + half);
  fx::V s[3], t[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const long long* r = P + (ix - 1 + i) * ny + (iy - 1);
    const fx::V a0 = fx_of_pair(r[0]), a1 = fx_of_pair(r[1]), a2 = fx_of_pair(r[2]);
    s[i] = fx::sp(fx::mul3(wym, a0, wy0, a1, wyp, a2));  // Q(sphi-2)
    t[i] = fx::sp(fx::mul3(dym, a0, dy0, a1, dyp, a2));  // Q(sphi-3)
  }
  gx = fx::mul3(dxm, s[0], dx0, s[1], dxp, s[2]);  // Q(sphi-5)
  gy = fx::mul3(wxm, t[0], wx0, t[1], wxp, t[2]);  // Q(sphi-5)
}

// Line density at z in Q(slam-2) (Grid1D::getValue); false when the particle
// needs the FP64 path.
__device__ __forceinline__ bool lam_fixed(const KickFix& k, const long long* __restrict__ Lm, double z,
                                          long long& lv) {
  lv = 0;
  const unsigned long long kz = dkey(z);
  if (kz >= k.kzmin && kz <= k.kzmax) {
    if (k.nz > 1) {
      int i0, ip;
      long long wp;
      if (!g1_fixed(fma(z, k.az, k.cz), k.nz, k.Fz, i0, ip, wp)) return false;
      wp <<= 6;
      lv = fx::mul2(fx::sp((1ll << 62) - wp), fx_of_pair(Lm[i0]), fx::sp(wp), fx_of_pair(Lm[ip]));
    } else {
      lv = fx::join(fx_of_pair(Lm[0])) >> 2;
    }
  }
  return true;
}

// Returns false when the particle needs the FP64 path.
__device__ __forceinline__ bool kick_fixed(const KickFix& k, const long long* __restrict__ P,
                                           const long long* __restrict__ Lm, double x, double y, double z,
                                           double& xp, double& yp) {
  int ix, iy;
  long long fx, fy, lv, gx, gy;
  if (!tsc_fixed(fma(x, k.ax, k.cx), k.nx, k.Fx, ix, fx)) return false;
  if (!tsc_fixed(fma(y, k.ay, k.cy), k.ny, k.Fy, iy, fy)) return false;
  if (!lam_fixed(k, Lm, z, lv)) return false;
  grad_fixed(P, k.ny, ix, iy, fx << 6, fy << 6, gx, gy);
  const double lf = dmul<(ORBIT_SOFT_MUL >> 4) & 1>((double)lv, k.lfs);  // -lambda(z) * factor
  xp = fma((double)gx, dmul<(ORBIT_SOFT_MUL >> 4) & 1>(k.gxs, lf), xp);
  yp = fma((double)gy, dmul<(ORBIT_SOFT_MUL >> 4) & 1>(k.gys, lf), yp);
  return true;
}

// The constants of kick_direct: cells as DepFast's, with limits a quarter cell
// outside those of x and y.
struct KickDirect {
  double a[3], c[3];
  int F[3], lo[3];
  unsigned span[3];
  double zmin, zmax;
  double gxs, gys, lfs;
};

// Executed by lanes 0..2 of one warp, one coordinate each.
__device__ __forceinline__ void load_kick_direct(KickDirect* d, const ScState* st, int nx, int ny, int nz) {
  const int k = threadIdx.x;
  const int nc = k == 0 ? nx : k == 1 ? ny : nz;
  const double inv = k == 0 ? st->inv_dx : k == 1 ? st->inv_dy : st->inv_dz;
  const double mn = k == 0 ? st->xmin : k == 1 ? st->ymin : st->zmin;
  const int F = fix_bits(nc);
  const double scale = __hiloint2double((1023 + F) << 20, 0);
  const double c = 0.5 - mn * inv;
  d->a[k] = inv * scale;
  d->c[k] = c * scale;
  d->F[k] = F;
  const int n32 = (int)(((long long)nc << F) >> 32), q = 1 << (F - 34);
  // x and y: v in [1/4, n - 1/4]; z: surely inside its limits
  const int lo = k < 2 ? q : 2 * q + 1, hi = k < 2 ? n32 - q - 1 : n32 + 2 * q - 1;
  const bool ok = k < 2 || (fabs(c) < 65536.0 && hi >= lo);
  d->lo[k] = ok ? lo : 0;
  d->span[k] = ok ? (unsigned)(hi - lo) : 0u;
  if (k == 2) {
    d->zmin = mn;
    d->zmax = st->zmax;
  }
}

// kick_fixed with the conversions on the FP64 pipe, for kernels that leave it
// idle.  iz, w: the particle's slice and fraction (Q62), for the longitudinal
// kick; iz = -1: outside the grid's length.
__device__ __forceinline__ bool kick_direct(const KickDirect& d, const long long* __restrict__ P,
                                            const long long* __restrict__ Lm, int nx, int ny, int nz, double x,
                                            double y, double z, double& xp, double& yp, int& iz, long long& w) {
  const long long vx = __double2ll_rz(fma(x, d.a[0], d.c[0])), vy = __double2ll_rz(fma(y, d.a[1], d.c[1]));
  const long long vz = __double2ll_rz(fma(z, d.a[2], d.c[2]));
  const int hx = (int)(vx >> 32), hy = (int)(vy >> 32), hz = (int)(vz >> 32);
  if (((unsigned)(hx - d.lo[0]) > d.span[0]) | ((unsigned)(hy - d.lo[1]) > d.span[1])) return false;
  const int ix = min(max(hx >> (d.F[0] - 32), 1), nx - 2), iy = min(max(hy >> (d.F[1] - 32), 1), ny - 2);
  auto frac = [](long long v, int F, int sub) {
    return (long long)(((unsigned long long)v << (62 - F)) - ((unsigned long long)(unsigned)sub << 32));
  };
  long long lv = 0;
  iz = -1;
  w = 0;
  if ((unsigned)(hz - d.lo[2]) <= d.span[2] || (z >= d.zmin && z <= d.zmax)) {
    iz = nz > 1 ? min(max(hz >> (d.F[2] - 32), 0), nz) : 0;
    if (nz > 1) {
      w = frac(vz, d.F[2], iz << 30);
      lv = fx::mul2(fx::sp((1ll << 62) - w), fx_of_pair(Lm[iz == 0 ? nz - 1 : iz - 1]), fx::sp(w),
                    fx_of_pair(Lm[iz == nz ? 0 : iz]));
    } else {
      lv = fx::join(fx_of_pair(Lm[0])) >> 2;
    }
  }
  long long gx, gy;
  grad_fixed(P, ny, ix, iy, frac(vx, d.F[0], (ix << 30) + (1 << 29)), frac(vy, d.F[1], (iy << 30) + (1 << 29)), gx, gy);
  const double lf = __ll2double_rn(lv) * d.lfs;  // -lambda(z) * factor
  xp = fma(__ll2double_rn(gx), d.gxs * lf, xp);
  yp = fma(__ll2double_rn(gy), d.gys * lf, yp);
  return true;
}

// kick_rb_long at slice iz and fraction w of kick_direct.
__device__ __forceinline__ void kick_rb_direct(const RbConst& r, const LogTab* lt, const double* __restrict__ lamd,
                                               int nz, double x, double y, int iz, long long w, double& dE) {
  if (iz < 0) return;
  double ez = lamd[0];
  if (nz > 1) {
    const double l0 = lamd[iz == 0 ? nz - 1 : iz - 1], l1 = lamd[iz == nz ? 0 : iz];
    const double f = __ll2double_rn(w);  // w 2^62
    const int h = __double2hiint(f);
    ez = fma(__hiloint2double(h == 0 ? 0 : h - (62 << 20), __double2loint(f)), l1 - l0, l0);
  }
  const double dx = x - r.xc, dy = y - r.yc;
  const double r2 = fma(dx, dx, dy * dy);
  double coeff;
  int64_t q;
  if (r2 <= r.a2) {
    coeff = fma(-r2, r.inv_a2, r.lin);
  } else if (log_q55(lt, r2, &q)) {
    const double f = __ll2double_rn(q);
    const int h = __double2hiint(f);
    coeff = r.lout - __hiloint2double(h == 0 ? 0 : h - (55 << 20), __double2loint(f));
  } else {
    coeff = r.lout - log(r2);
  }
  dE = fma(ez * r.lsf, coeff, dE);
}

}  // namespace orbit
