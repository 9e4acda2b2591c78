// Bunch diagnostics on the device (src/orbit/BunchDiagnostics): the first and
// second moments of BunchTwissAnalysis::analyzeBunch as a deterministic
// two-level reduction, and BunchTuneAnalysis::analyzeBunch per particle
// with its attributes kept on the device.  No coordinate leaves the GPU.
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "sc2p5d.cuh"
#include "sc_device.cuh"

namespace orbit {

static const int kMomThreads = 256;
static const int kNMom = 28;  // total macrosize, 6 first moments, 21 second moments (i >= j)

// out[k] = sum over the launch's blocks of part[block * ns + k], run by the
// last block: one warp per sum, each lane a fixed stride of blocks, then a
// fixed shuffle tree, so the result is the same on every run.
__device__ __forceinline__ void sum_parts(const double* __restrict__ part, int ns, double* __restrict__ out) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int k = threadIdx.x >> 5; k < ns; k += nw) {
    double t = 0.0;
    for (int bk = lane; bk < (int)gridDim.x; bk += 32) t += __ldcg(part + (size_t)bk * ns + k);
    for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
    if (lane == 0) out[k] = t;
  }
}

// Per-block sums of m, m c_i, m c_i c_j (i >= j), summed in a fixed order:
// the block results go to part[block], the last block adds them up into
// out[28].
template <bool MS>
__global__ void __launch_bounds__(kMomThreads) k_moments(const double* __restrict__ coords, int cap, int n,
                                                         const double* __restrict__ msize, double* part,
                                                         unsigned* counter, double* out) {
  double s[kNMom];
#pragma unroll
  for (int k = 0; k < kNMom; ++k) s[k] = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double c[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) c[q] = coords[(size_t)q * cap + i];
    double m = MS ? msize[i] : 1.0;
    s[0] += m;
    int k = 7;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      double mc = MS ? m * c[q] : c[q];
      s[1 + q] += mc;
#pragma unroll
      for (int r = 0; r <= q; ++r) s[k++] += mc * c[r];
    }
  }
  __shared__ double red[kMomThreads / 32][kNMom];
#pragma unroll
  for (int k = 0; k < kNMom; ++k)
    for (int off = 16; off > 0; off >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], off);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int k = 0; k < kNMom; ++k) red[threadIdx.x >> 5][k] = s[k];
  __syncthreads();
  if (threadIdx.x < kNMom) {
    double t = 0.0;
    for (int w = 0; w < kMomThreads / 32; ++w) t += red[w][threadIdx.x];
    part[(size_t)blockIdx.x * kNMom + threadIdx.x] = t;
  }
  if (last_block_done(counter, gridDim.x)) sum_parts(part, kNMom, out);
}

// Cells of the x-y moment table that computeBunchMoments accumulates
// (j < order, i <= order - j), and its stray cell.
__host__ __device__ constexpr int xy_cells(int order) { return order * (order + 3) / 2 + 1; }

struct XyArgs {
  double disp;    // D / (E_kin + m) / beta^2 (0 without the dispersion term)
  double xa, ya;  // the averages the moments are centred on
};

// BunchTwissAnalysis::computeBunchMoments (BunchTwissAnalysis.cc:146-340):
// the sums over the bunch of X^i Y^j for every cell (i, j) of the table, with
// X = m ((x - disp dE) - xa), Y = m (y - ya) (m = 1 for a uniform macrosize),
// then of X^2 Y^order, which the reference's uniform-macrosize loop adds to
// cell [2][order] once per particle.  The reference divides every term by
// sqrt(beta)^i and sqrt(beta)^j; the divisors do not depend on the particle,
// so the host divides the sums.
//
// One pass over the bunch for all cells, each particle's powers formed
// once, block partials in a fixed order and the last block summing them:
// bound by the FP64 pipe (22 operations per particle at order 4; DRAM is at
// 24 B per particle).  A block row per cell, each reading the whole bunch
// and dividing twice per term, took 2811 us for the 15 cells of order 4 on
// 4e6 particles; this takes 157 us (FP64 pipe 82% busy).  Orders up to kXyFused keep their sums
// in registers (28 at order 6).
static const int kXyFused = 6;

template <int ORDER, bool MS, bool DISP>
__global__ void __launch_bounds__(kMomThreads) k_xy_moments(const double* __restrict__ coords, int cap, int n,
                                                            const double* __restrict__ msize, XyArgs a,
                                                            double* part, unsigned* counter, double* out) {
  constexpr int NC = xy_cells(ORDER);
  double s[NC];
#pragma unroll
  for (int k = 0; k < NC; ++k) s[k] = 0.0;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    double x = coords[q], y = coords[(size_t)2 * cap + q];
    if (DISP) x = fma(-a.disp, coords[(size_t)5 * cap + q], x);
    double X[ORDER + 1], Y[ORDER + 1];
    X[1] = x - a.xa;
    Y[1] = y - a.ya;
    if (MS) {
      const double m = msize[q];
      X[1] *= m;
      Y[1] *= m;
    }
    X[0] = Y[0] = 1.0;
#pragma unroll
    for (int i = 2; i <= ORDER; ++i) {
      X[i] = X[i - 1] * X[1];
      Y[i] = Y[i - 1] * Y[1];
    }
    int k = 0;
#pragma unroll
    for (int j = 0; j < ORDER; ++j)
#pragma unroll
      for (int i = 0; i <= ORDER - j; ++i, ++k) {
        if (i + j < 2) continue;  // [0][0], [1][0] and [0][1] are fixed by the host
        s[k] = i == 0 ? s[k] + Y[j] : (j == 0 ? s[k] + X[i] : fma(X[i], Y[j], s[k]));
      }
    if (!MS) s[k] = fma(X[2], Y[ORDER], s[k]);
  }
  __shared__ double red[kMomThreads / 32][NC];
#pragma unroll
  for (int k = 0; k < NC; ++k)
    for (int off = 16; off > 0; off >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], off);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int k = 0; k < NC; ++k) red[threadIdx.x >> 5][k] = s[k];
  __syncthreads();
  if (threadIdx.x < NC) {
    double t = 0.0;
    for (int w = 0; w < kMomThreads / 32; ++w) t += red[w][threadIdx.x];
    part[(size_t)blockIdx.x * NC + threadIdx.x] = t;
  }
  if (last_block_done(counter, gridDim.x)) sum_parts(part, NC, out);
}

// The sums of one cell per blockIdx.y, for orders above kXyFused (their sums
// do not fit in one thread's registers); the last block adds the partials.
__global__ void __launch_bounds__(kMomThreads) k_xy_moments_cell(const double* __restrict__ coords, int cap, int n,
                                                                 const double* __restrict__ msize, XyArgs a,
                                                                 int order, double* part, unsigned* counter,
                                                                 double* out) {
  int j = 0, c = blockIdx.y;
  while (j < order && c > order - j) c -= order + 1 - j++;
  const int ci = j < order ? c : 2, cj = j;  // j = order: the stray cell
  double s = 0.0;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    double X = coords[q], Y = coords[(size_t)2 * cap + q] - a.ya;
    if (a.disp != 0.0) X = fma(-a.disp, coords[(size_t)5 * cap + q], X);
    X -= a.xa;
    if (msize) {
      X *= msize[q];
      Y *= msize[q];
    }
    double t = 1.0;
    for (int i = 0; i < ci; ++i) t *= X;
    for (int i = 0; i < cj; ++i) t *= Y;
    s += t;
  }
  __shared__ double red[kMomThreads / 32];
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kMomThreads / 32; ++w) t += red[w];
    part[(size_t)blockIdx.x * gridDim.y + blockIdx.y] = t;
  }
  if (last_block_done(counter, gridDim.x * gridDim.y)) sum_parts(part, gridDim.y, out);
}

struct TuneArgs {
  double betax, alphax, etax, etapx, betay, alphay;
  double beta, etot;
};

// BunchTuneAnalysis::analyzeBunch (BunchTuneAnalysis.cc:36-108): normalised
// phases, the phase advance since the last call and the actions; ph holds
// six rows {xLastPhase, yLastPhase, xLastTune, yLastTune, xAction, yAction}.
__global__ void k_tune(const double* __restrict__ coords, int cap, int n, TuneArgs a, double* ph, int pcap) {
  const double twopi = 2.0 * 3.14159265358979323846;  // 2 OrbitConst::PI
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double x = coords[i], xp = coords[(size_t)cap + i];
    double y = coords[2 * (size_t)cap + i], yp = coords[3 * (size_t)cap + i];
    double dE = coords[5 * (size_t)cap + i];
    double dpp = 1 / (a.beta * a.beta) * dE / a.etot;
    double sbx = sqrt(a.betax), sby = sqrt(a.betay);
    double xval = (x - a.etax * dpp) / sbx;
    double xpval = (xp - a.etapx * dpp) * sbx + xval * a.alphax;
    double yval = y / sby;
    double ypval = (yp + y * a.alphay / a.betay) * sby;
    double ang = atan2(xpval, xval);
    if (ang < 0.) ang += twopi;
    double xt = (ph[i] - ang) / twopi;
    if (xt < 0.) xt += 1.;
    ph[i] = ang;
    ph[2 * (size_t)pcap + i] = xt;
    ang = atan2(ypval, yval);
    if (ang < 0.) ang += twopi;
    double yt = (ph[(size_t)pcap + i] - ang) / twopi;
    if (yt < 0.) yt += 1.;
    ph[(size_t)pcap + i] = ang;
    ph[3 * (size_t)pcap + i] = yt;
    double xc = x - a.etax * dpp, yc = y;
    double pxc = (xp - a.etapx * dpp) + xc * (a.alphax / a.betax);
    double pyc = yp + yc * (a.alphay / a.betay);
    ph[4 * (size_t)pcap + i] = xc * xc / a.betax + pxc * pxc * a.betax;
    ph[5 * (size_t)pcap + i] = yc * yc / a.betay + pyc * pyc * a.betay;
  }
}

static int moment_blocks() { return num_sms() * 2; }

// Scratch of the moment sums, kept with the bunch: the block partials of
// the largest table, the results and the block counter.
static const int kMaxSums = xy_cells(16);

struct DiagScratch {
  double* part;
  double* res;
  unsigned* counter;
};

static int diag_scratch(orbit_bunch_t* b, DiagScratch* d) {
  const size_t np = (size_t)moment_blocks() * kMaxSums;
  if (!b->d_diag) {
    const size_t bytes = sizeof(double) * (np + kMaxSums + 1);
    ORBIT_CUDA(cudaMalloc(&b->d_diag, bytes));
    ORBIT_CUDA(cudaMemsetAsync(b->d_diag, 0, bytes, b->stream));
  }
  d->part = b->d_diag;
  d->res = d->part + np;
  d->counter = reinterpret_cast<unsigned*>(d->res + kMaxSums);
  return ORBIT_OK;
}

template <int ORDER>
static void launch_xy(orbit_bunch_t* b, const XyArgs& a, const DiagScratch& d) {
  const int nb = moment_blocks();
  const bool ms = b->has_msize != 0, disp = a.disp != 0.0;
  auto go = [&](auto kernel) {
    kernel<<<nb, kMomThreads, 0, b->stream>>>(b->d_coords, b->cap, b->n, b->d_msize, a, d.part, d.counter, d.res);
  };
  if (ms) disp ? go(k_xy_moments<ORDER, true, true>) : go(k_xy_moments<ORDER, true, false>);
  else disp ? go(k_xy_moments<ORDER, false, true>) : go(k_xy_moments<ORDER, false, false>);
}

// Phase rows of capacity >= n, zero for particles without a value yet.
static int ensure_phase(orbit_bunch_t* b) {
  if (b->d_phase && b->phase_cap >= b->n) return ORBIT_OK;
  int cap = b->cap > b->n ? b->cap : b->n;
  if (cap < 1) cap = 1;
  double* d = nullptr;
  ORBIT_CUDA(cudaMalloc(&d, sizeof(double) * 6 * (size_t)cap));
  ORBIT_CUDA(cudaMemsetAsync(d, 0, sizeof(double) * 6 * (size_t)cap, b->stream));
  if (b->d_phase) {
    int keep = b->phase_cap < b->n ? b->phase_cap : b->n;
    for (int r = 0; r < 6; ++r)
      ORBIT_CUDA(cudaMemcpyAsync(d + (size_t)r * cap, b->d_phase + (size_t)r * b->phase_cap, sizeof(double) * keep,
                                 cudaMemcpyDeviceToDevice, b->stream));
    ORBIT_CUDA(cudaStreamSynchronize(b->stream));
    cudaFree(b->d_phase);
  }
  b->d_phase = d;
  b->phase_cap = cap;
  return ORBIT_OK;
}

}  // namespace orbit

using namespace orbit;

extern "C" {

int orbit_bunch_moments(orbit_bunch_t* b, double* out) {
  if (!b || !out) return set_error(ORBIT_ERR_ARG, "orbit_bunch_moments: bad argument");
  const int nb = moment_blocks();
  std::lock_guard<std::mutex> lock(b->diag_mu);
  DiagScratch d;
  int rc = diag_scratch(b, &d);
  if (rc) return rc;
  double h[kNMom];
  if (b->n > 0) {
    if (b->has_msize)
      k_moments<true><<<nb, kMomThreads, 0, b->stream>>>(b->d_coords, b->cap, b->n, b->d_msize, d.part, d.counter,
                                                           d.res);
    else
      k_moments<false><<<nb, kMomThreads, 0, b->stream>>>(b->d_coords, b->cap, b->n, nullptr, d.part, d.counter,
                                                            d.res);
    ORBIT_LAUNCH_CHECK("moments");
    ORBIT_CUDA(cudaMemcpyAsync(h, d.res, sizeof(h), cudaMemcpyDeviceToHost, b->stream));
    ORBIT_CUDA(cudaStreamSynchronize(b->stream));
  } else {
    for (int k = 0; k < kNMom; ++k) h[k] = 0.0;
  }
  // BunchTwissAnalysis.cc:95-140: averages and correlations over the total macrosize
  const double total = h[0];
  out[0] = b->n;
  out[1] = total;
  for (int k = 1; k < kNMom; ++k) out[k + 1] = std::fabs(total) > 0. ? h[k] / total : 0.0;
  return ORBIT_OK;
}

int orbit_bunch_xy_moments(orbit_bunch_t* b, int order, const double* params, double* out) {
  if (!b || !params || !out || order < 2 || order > 16)
    return set_error(ORBIT_ERR_ARG, "orbit_bunch_xy_moments: bad argument (2 <= order <= 16)");
  const int nc = xy_cells(order);
  const bool uniform = !b->has_msize;
  std::unique_lock<std::mutex> lock(b->diag_mu);
  DiagScratch d;
  int rc = diag_scratch(b, &d);
  if (rc) return rc;
  XyArgs a;
  a.disp = params[0] != 0.0 ? params[0] / params[1] / params[2] : 0.0;
  a.xa = params[3];
  a.ya = params[4];
  double sum[kMaxSums] = {};
  if (b->n > 0) {
    switch (order) {
      case 2: launch_xy<2>(b, a, d); break;
      case 3: launch_xy<3>(b, a, d); break;
      case 4: launch_xy<4>(b, a, d); break;
      case 5: launch_xy<5>(b, a, d); break;
      case kXyFused: launch_xy<kXyFused>(b, a, d); break;
      default:
        k_xy_moments_cell<<<dim3(moment_blocks(), nc), kMomThreads, 0, b->stream>>>(
            b->d_coords, b->cap, b->n, uniform ? nullptr : b->d_msize, a, order, d.part, d.counter, d.res);
    }
    ORBIT_LAUNCH_CHECK("xy moments");
    ORBIT_CUDA(cudaMemcpyAsync(sum, d.res, sizeof(double) * nc, cudaMemcpyDeviceToHost, b->stream));
    ORBIT_CUDA(cudaStreamSynchronize(b->stream));
  }
  lock.unlock();
  // total macrosize: n for a uniform macrosize (the reference's m_size = 1
  // there), else the sum of the macrosizes
  double total = (double)b->n;
  if (!uniform) {
    double mom[29];
    rc = orbit_bunch_moments(b, mom);
    if (rc) return rc;
    total = mom[1];
  }
  const int w = order + 1;
  for (int k = 0; k < w * w; ++k) out[k] = 0.0;
  // pow(xbetaterm, double(i)) pow(ybetaterm, double(j)) (BunchTwissAnalysis.cc:249),
  // in long double: a term's divisions average out over the bunch, the sum's would not
  long double xb[17], yb[17];
  xb[0] = yb[0] = 1.0L;
  for (int i = 1; i <= order; ++i) {
    xb[i] = xb[i - 1] * params[5];
    yb[i] = yb[i - 1] * params[6];
  }
  int k = 0;
  for (int j = 0; j < order; ++j)
    for (int i = 0; i < order + 1 - j; ++i, ++k) {
      const long double t = sum[k] / (xb[i] * yb[j]);
      out[i * w + j] += (double)(uniform ? t : t + sum[k]);
    }
  if (uniform) out[2 * w + order] += sum[k];
  // BunchTwissAnalysis.cc:325-336: divided for i + j <= order (the stray
  // cell [2][order] is not), then the three fixed cells
  if (std::fabs(total) > 0.)
    for (int i = 0; i < w; ++i)
      for (int j = 0; j < w - i; ++j) out[i * w + j] /= total;
  out[0] = 1.0;
  out[1 * w + 0] = params[3];
  out[0 * w + 1] = params[4];
  return ORBIT_OK;
}

int orbit_bunch_tune_analysis(orbit_bunch_t* b, const double* twiss, double etot) {
  if (!b || !twiss) return set_error(ORBIT_ERR_ARG, "orbit_bunch_tune_analysis: bad argument");
  int rc = ensure_phase(b);
  if (rc) return rc;
  if (b->n == 0) return ORBIT_OK;
  TuneArgs a;
  a.betax = twiss[0]; a.alphax = twiss[1]; a.etax = twiss[2]; a.etapx = twiss[3];
  a.betay = twiss[4]; a.alphay = twiss[5];
  a.beta = b->sync.beta;
  a.etot = etot;
  int blocks = (b->n + 255) / 256;
  if (blocks > num_sms() * 8) blocks = num_sms() * 8;
  k_tune<<<blocks, 256, 0, b->stream>>>(b->d_coords, b->cap, b->n, a, b->d_phase, b->phase_cap);
  ORBIT_LAUNCH_CHECK("tune analysis");
  return ORBIT_OK;
}

int orbit_bunch_phase_get(orbit_bunch_t* b, double* host) {
  if (!b || (!host && b->n > 0)) return set_error(ORBIT_ERR_ARG, "orbit_bunch_phase_get: bad argument");
  if (!b->d_phase) return set_error(ORBIT_ERR_ARG, "orbit_bunch_phase_get: no tune analysis has run");
  for (int r = 0; r < 6; ++r)
    ORBIT_CUDA(cudaMemcpyAsync(host + (size_t)r * b->n, b->d_phase + (size_t)r * b->phase_cap,
                               sizeof(double) * b->n, cudaMemcpyDeviceToHost, b->stream));
  ORBIT_CUDA(cudaStreamSynchronize(b->stream));
  return ORBIT_OK;
}

int orbit_bunch_phase_set(orbit_bunch_t* b, const double* host) {
  if (!b || (!host && b->n > 0)) return set_error(ORBIT_ERR_ARG, "orbit_bunch_phase_set: bad argument");
  int rc = ensure_phase(b);
  if (rc) return rc;
  for (int r = 0; r < 6; ++r)
    ORBIT_CUDA(cudaMemcpyAsync(b->d_phase + (size_t)r * b->phase_cap, host + (size_t)r * b->n,
                               sizeof(double) * b->n, cudaMemcpyHostToDevice, b->stream));
  ORBIT_CUDA(cudaStreamSynchronize(b->stream));
  return ORBIT_OK;
}

}  // extern "C"
