// kernels.cu - sm_103a kernels of libswave (compiled with --fmad=false).
//
// Each kernel restates one reference loop nest with the same floating-point
// operation order; the comments give the reference file:line.  Paths are
// relative to the reference project root.
#include "../../include/swave.h"
#include "norms.cuh"
#include "swave_dev.cuh"

namespace swave {

// ---------------------------------------------------------------------------
// Padding and coefficients
// ---------------------------------------------------------------------------

// model_pad (libs/libwave/ReadSouVelRho.f90:545-596): edge replication is
// a clamp of every padded index onto the physical window.
__global__ void k_pad_velocity(Geom g, const float *__restrict__ vp, float *__restrict__ out) {
  const long long n = (long long)g.n1p * g.n2p * g.n3p;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x) {
    const int a = (int)(q % g.n1p);
    const long long r = q / g.n1p;
    const int b = (int)(r % g.n2p);
    const int c = (int)(r / g.n2p);
    const int i = g.lo1 + a, j = g.lo2 + b, k = g.lo3 + c;
    const int ii = min(max(i, 1), g.nz), jj = min(max(j, 1), g.nx), kk = min(max(k, 1), g.ny);
    out[g.idx(i, j, k)] = vp[g.pidx(ii, jj, kk)];
  }
}

// Higdon_coeff (libs/libwave/Boundary.f90:66-87).
__device__ __forceinline__ void higdon_coeff(float nu, float *c, int stride) {
  const float beta1 = 1.0f, beta2 = 0.7f, weight = 0.5f;
  float fdum = (beta1 + nu) * (1.0f - weight);
  const float qx = (weight * (beta1 + nu) - nu) / fdum;
  const float qt = (weight * (beta1 + nu) - beta1) / fdum;
  const float qxt = weight / (weight - 1.0f);
  fdum = (beta2 + nu) * (1.0f - weight);
  const float rx = (weight * (beta2 + nu) - nu) / fdum;
  const float rt = (weight * (beta2 + nu) - beta2) / fdum;
  const float rxt = weight / (weight - 1.0f);
  c[0 * stride] = qx + rx;
  c[1 * stride] = qx * rx;
  c[2 * stride] = qt + rt;
  c[3 * stride] = ((qx * rt + qt * rx) + qxt) + rxt;
  c[4 * stride] = qx * rxt + rx * qxt;
  c[5 * stride] = qt * rt;
  c[6 * stride] = qt * rxt + rt * qxt;
  c[7 * stride] = qxt * rxt;
}

// Higdon (libs/libwave/Boundary.f90:17-63).  Layouts: gz[c][k][j],
// gx[c][k][i], gy[c][j][i].
__global__ void k_higdon_coeffs(Geom g, const float *__restrict__ vel, float dt, float dxi,
                                float dyi, float dzi, float *gz, float *gx, float *gy) {
  const int n1 = g.nmax1 - g.nmin1 + 1, n2 = g.nmax2 - g.nmin2 + 1, n3 = g.nmax3 - g.nmin3 + 1;
  const long long nzc = (long long)n2 * n3, nxc = (long long)n1 * n3;
  const long long nyc = (g.nmax3 > 1) ? (long long)n1 * n2 : 0;
  const long long tot = nzc + nxc + nyc;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < tot;
       q += (long long)gridDim.x * blockDim.x) {
    if (q < nzc) {
      const int j = g.nmin2 + (int)(q % n2), k = g.nmin3 + (int)(q / n2);
      higdon_coeff((vel[g.idx(g.nmin1, j, k)] * dt) * dzi, gz + q, (int)nzc);
      higdon_coeff((vel[g.idx(g.nmax1, j, k)] * dt) * dzi, gz + q + 8 * nzc, (int)nzc);
    } else if (q < nzc + nxc) {
      const long long r = q - nzc;
      const int i = g.nmin1 + (int)(r % n1), k = g.nmin3 + (int)(r / n1);
      higdon_coeff((vel[g.idx(i, g.nmin2, k)] * dt) * dxi, gx + r, (int)nxc);
      higdon_coeff((vel[g.idx(i, g.nmax2, k)] * dt) * dxi, gx + r + 8 * nxc, (int)nxc);
    } else {
      const long long r = q - nzc - nxc;
      const int i = g.nmin1 + (int)(r % n1), j = g.nmin2 + (int)(r / n1);
      higdon_coeff((vel[g.idx(i, j, g.nmin3)] * dt) * dyi, gy + r, (int)nyc);
      higdon_coeff((vel[g.idx(i, j, g.nmax3)] * dt) * dyi, gy + r + 8 * nyc, (int)nyc);
    }
  }
}

// ---------------------------------------------------------------------------
// FWI helpers
// ---------------------------------------------------------------------------

// mod_window_pad(adj=.true.) (ExtractPadModel.f90:509-549).
__global__ void k_window_vel(int nz, int nx, int ny, float ox, float oy, float dx, float dy,
                             int nxw, int nyw, float oxw, float oyw, const float *__restrict__ big,
                             float *__restrict__ small) {
  const long long n = (long long)nz * nxw * nyw;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x) {
    const int l = (int)(q % nz);
    const long long r = q / nz;
    const int i = 1 + (int)(r % nxw), j = 1 + (int)(r / nxw);
    const float cy = (float)(j - 1) * dy + oyw;
    const int iy = (int)lroundf((cy - oy) / dy) + 1;
    const int iy1 = min(ny, max(1, iy));
    const float cx = (float)(i - 1) * dx + oxw;
    const int ix = (int)lroundf((cx - ox) / dx) + 1;
    const int ix1 = min(nx, max(1, ix));
    small[q] = 0.f + big[(long long)l + (long long)nz * ((ix1 - 1) + (long long)nx * (iy1 - 1))];
  }
}

// mod_copy_image (ExtractPadModel.f90:662-697); the window-to-model column
// map is injective, so threads never collide.
__global__ void k_copy_image(int nz, int nx, int ny, float ox, float oy, float dx, float dy,
                             int nxw, int nyw, float oxw, float oyw, const float *__restrict__ ims,
                             const float *__restrict__ ils, float *image, float *illum) {
  const long long n = (long long)nz * nxw * nyw;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x) {
    const int l = (int)(q % nz);
    const long long r = q / nz;
    const int i = 1 + (int)(r % nxw), j = 1 + (int)(r / nxw);
    const float cy = (float)(j - 1) * dy + oyw;
    const int iy = (int)lroundf((cy - oy) / dy) + 1;
    if (iy < 1 || iy > ny) continue;
    const float cx = (float)(i - 1) * dx + oxw;
    const int ix = (int)lroundf((cx - ox) / dx) + 1;
    if (ix < 1 || ix > nx) continue;
    const long long o = (long long)l + (long long)nz * ((ix - 1) + (long long)nx * (iy - 1));
    image[o] = image[o] + ims[q];
    illum[o] = illum[o] + ils[q];
  }
}

// Compute_OF_RES_ADJ (Objective_Function_Residual_Adjsource.f90:17-40) with
// the L2 norm (Norm.f90:26-28): every trace's misfit is one FP64 sum in
// sample order.  A block takes RES_T traces in chunks of RES_K samples: all
// threads form the residuals and adjoint sources (coalesced) and leave the
// squares in shared memory, where one thread per trace adds them while the
// others load the next chunk.  Bound by the chain of FP64 additions; one
// thread per trace reading its own row took 199 us for 451 traces of 1000
// samples.
constexpr int RES_T = 8, RES_K = 128;
__global__ void __launch_bounds__(256) k_residual(int nrec, int nt, const float *__restrict__ dobs,
                                                  const float *__restrict__ mute,
                                                  float *__restrict__ dmod,
                                                  float *__restrict__ resid, double *partial) {
  __shared__ double sq[2][RES_K][RES_T + 1];
  const int r0 = RES_T * blockIdx.x, tid = threadIdx.x;
  double ssum = 0.0;
  const int nchunk = (nt + RES_K - 1) / RES_K;
  for (int c = 0; c <= nchunk; ++c) {
    if (c < nchunk) {
#pragma unroll
      for (int q = tid; q < RES_T * RES_K; q += 256) {
        const int r = r0 + q / RES_K, k = q % RES_K, t = c * RES_K + k;
        if (r >= nrec || t >= nt) continue;
        const long long o = (long long)r * nt + t;
        const float m = mute ? mute[o] : 1.0f;
        const float d = m * (dobs[o] - dmod[o]);
        if (resid) resid[o] = d;
        dmod[o] = m * d;
        sq[c & 1][k][q / RES_K] = (double)d * (double)d;
      }
    }
    if (c > 0 && tid < RES_T) {
      const int len = min(RES_K, nt - (c - 1) * RES_K);
#pragma unroll 8
      for (int k = 0; k < len; ++k) ssum = ssum + sq[(c - 1) & 1][k][tid];
    }
    __syncthreads();
  }
  if (tid < RES_T && r0 + tid < nrec) partial[r0 + tid] = ssum / 2;
}

// max|m*(dobs - dmod)| of every trace: the threshold fct_compute takes when
// data_threshold is 0 (Norm.f90:37-40).
__global__ void k_trace_maxabs(int nrec, int nt, const float *__restrict__ dobs,
                               const float *__restrict__ mute, const float *__restrict__ dmod,
                               float *maxabs) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrec) return;
  const long long o = (long long)r * nt;
  float mx = 0.0f;
  for (int t = 0; t < nt; ++t) {
    const float m = mute ? mute[o + t] : 1.0f;
    mx = fmaxf(mx, fabsf(m * (dobs[o + t] - dmod[o + t])));
  }
  maxabs[r] = mx;
}

// Compute_OF_RES_ADJ for the L1, Huber, Cauchy and hyperbolic norms
// (Objective_Function_Residual_Adjsource.f90:32-38 with fct_compute and
// gdt_compute, libs/libinv/Norm.f90:12-141): one thread per trace, the
// trace's misfit summed in FP32 in sample order like the reference's
// sum() of a real array.  Trace r's threshold is thresh0, or, when that is
// 0, max|r| of the first trace k <= r whose maximum is not 0 (the caller's
// threshold is reset by the first such trace and kept by the following
// ones); with no such trace it stays 0, as in the reference.
__global__ void k_residual_nrm(int ntype, int nrec, int nt, const float *__restrict__ dobs,
                               const float *__restrict__ mute, float *dmod, float *resid,
                               double *partial, float thresh0, const float *__restrict__ maxabs) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrec) return;
  float g = thresh0;
  if (g == 0.0f && maxabs) {
    for (int k = 0; k <= r; ++k)
      if (maxabs[k] != 0.0f) {
        g = maxabs[k];
        break;
      }
  }
  const long long o = (long long)r * nt;
  float fs = 0.0f;
  for (int t = 0; t < nt; ++t) {
    const float m = mute ? mute[o + t] : 1.0f;
    const float d = m * (dobs[o + t] - dmod[o + t]);
    if (resid) resid[o + t] = d;
    fs = fs + nrm_term(ntype, d, g);
    dmod[o + t] = nrm_gdt(ntype, m * d, g);
  }
  partial[r] = (double)fs;
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
static inline int nblocks(long long n, int bs, int cap = 152 * 16) {
  long long b = (n + bs - 1) / bs;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}

cudaError_t launch_pad_velocity(const Geom &g, const float *vel_phys, float *vel_pad,
                                cudaStream_t s) {
  const long long n = (long long)g.n1p * g.n2p * g.n3p;
  k_pad_velocity<<<nblocks(n, 256), 256, 0, s>>>(g, vel_phys, vel_pad);
  return cudaGetLastError();
}

// One pass of Interpolate (Interpolate.f90:63-126) along `axis` (0 z, 1 x,
// 2 y): every line of the padded array is filtered by the 9-point half-cell
// sinc, its end values extended past both ends; one thread per line, taps
// added in order from -4 to +4.  recip stores 1/f (delp = 1/rho2,
// FDderivatives.f90:393,581) instead of f.
struct Sinc9 {
  float s[9];
};

__global__ void k_sinc9_lines(Geom g, int axis, Sinc9 w, const float *__restrict__ src,
                              float *__restrict__ dst, int recip) {
  const long long nl = axis == 0 ? (long long)g.n2p * g.n3p
                                 : axis == 1 ? (long long)g.n1p * g.n3p
                                             : (long long)g.n1p * g.n2p;
  for (long long L = blockIdx.x * (long long)blockDim.x + threadIdx.x; L < nl;
       L += (long long)gridDim.x * blockDim.x) {
    long long base, stride;
    int len;
    if (axis == 0) {
      base = g.idx(g.lo1, g.lo2 + (int)(L % g.n2p), g.lo3 + (int)(L / g.n2p));
      len = g.n1p;
      stride = 1;
    } else if (axis == 1) {
      base = g.idx(g.lo1 + (int)(L % g.n1p), g.lo2, g.lo3 + (int)(L / g.n1p));
      len = g.n2p;
      stride = g.ld1;
    } else {
      base = g.idx(g.lo1 + (int)(L % g.n1p), g.lo2 + (int)(L / g.n1p), g.lo3);
      len = g.n3p;
      stride = g.plane();
    }
    for (int q = 0; q < len; ++q) {
      float f = 0.f;
#pragma unroll
      for (int l = -4; l <= 4; ++l) {
        const int qq = min(max(q + l, 0), len - 1);
        f = f + w.s[4 + l] * src[base + (long long)qq * stride];
      }
      dst[base + (long long)q * stride] = recip ? 1.f / f : f;
    }
  }
}

cudaError_t launch_rho_delp(const Geom &g, const float *rho_pad, float *delp, float *tmp,
                            const float *sinc9, cudaStream_t s, int *nlaunch) {
  Sinc9 w;
  for (int q = 0; q < 9; ++q) w.s[q] = sinc9[q];
  auto go = [&](int axis, const float *a, float *b, int recip) {
    const long long nl = axis == 0 ? (long long)g.n2p * g.n3p
                                   : axis == 1 ? (long long)g.n1p * g.n3p
                                               : (long long)g.n1p * g.n2p;
    k_sinc9_lines<<<nblocks(nl, 128), 128, 0, s>>>(g, axis, w, a, b, recip);
    ++*nlaunch;
  };
  if (g.n3p > 1) {
    go(0, rho_pad, delp, 0);
    go(1, delp, tmp, 0);
    go(2, tmp, delp, 1);
  } else {
    go(0, rho_pad, tmp, 0);
    go(1, tmp, delp, 1);
  }
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Band-pass of traces (Bandpass.f90:89-149 with the filters of bandpass.c).
// The trace is padded by npad samples at each end with cosine-squared ramps
// from its end values, run through the low-cut and then the high-cut cascade
// of second-order sections (forward, and for a zero-phase filter again over
// the reversed samples 2..n-2), and its middle nt samples are returned.  The
// work array D is sample-major (sample i of trace t at i*ntr + t), so that a
// warp's accesses coalesce.
//
// The recursion is serial in time: one thread per trace, bound by its
// instruction issue.  A pass runs up to four sections at once, section q one
// sample behind section q-1, so that the sections' operations are
// independent within an iteration and a sample costs one load and one store
// for all of them; the inputs of the next eight samples are loaded ahead.
// One thread per trace running one section at a time through memory took
// 6.8 ms for 901 traces of 2223 samples (whole call, 14-pole zero phase).
// The first two outputs of every section stay zero, as the reference's
// never-written work samples do.
// ---------------------------------------------------------------------------
// A block of k_bp_pad and k_bp_cut takes 32 traces x 32 samples, trace blocks
// fastest in one grid dimension: the others hold 65535 blocks, fewer than
// long records or many traces need.
__global__ void __launch_bounds__(256) k_bp_pad(int ntr, int nt, int npad, const float *lead,
                                                const float *trail, const float *__restrict__ in,
                                                float *__restrict__ D) {
  __shared__ float tile[32][33];
  const int n = nt + 2 * npad, gx = (ntr + 31) / 32;
  const int t0 = 32 * (blockIdx.x % gx), i0 = 32 * (blockIdx.x / gx);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int r = w; r < 32; r += 8) {
    const int t = t0 + r, i = i0 + lane;
    if (t >= ntr || i >= n) continue;
    const float *tr = in + (size_t)t * nt;
    tile[r][lane] = i < npad ? tr[0] * lead[i]
                    : i < npad + nt ? tr[i - npad] : tr[nt - 1] * trail[i - npad - nt];
  }
  __syncthreads();
  for (int r = w; r < 32; r += 8)
    if (t0 + lane < ntr && i0 + r < n) D[(size_t)(i0 + r) * ntr + t0 + lane] = tile[lane][r];
}

__global__ void __launch_bounds__(256) k_bp_cut(int ntr, int nt, int npad,
                                                const float *__restrict__ D,
                                                float *__restrict__ out) {
  __shared__ float tile[32][33];
  const int gx = (ntr + 31) / 32, t0 = 32 * (blockIdx.x % gx), i0 = 32 * (blockIdx.x / gx);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int r = w; r < 32; r += 8)
    if (t0 + lane < ntr && i0 + r < nt)
      tile[r][lane] = D[(size_t)(npad + i0 + r) * ntr + t0 + lane];
  __syncthreads();
  for (int r = w; r < 32; r += 8)
    if (t0 + r < ntr && i0 + lane < nt) out[(size_t)(t0 + r) * nt + i0 + lane] = tile[lane][r];
}

// NS sections over samples 2..n-1 of every trace, in place; with rev over
// the reversed samples (sample i is D[n + 1 - i], before it zeros).
template <int NS>
__global__ void __launch_bounds__(32) k_bp_sections(int ntr, int n, int rev,
                                                    const float *__restrict__ c, float *D) {
  const int t = blockIdx.x * 32 + threadIdx.x;
  if (t >= ntr) return;
  float cf[NS][5], xm1[NS], xm2[NS], nm1[NS], nm2[NS], v[NS];
#pragma unroll
  for (int q = 0; q < NS; ++q) {
#pragma unroll
    for (int m = 0; m < 5; ++m) cf[q][m] = c[5 * q + m];
    xm1[q] = xm2[q] = nm1[q] = nm2[q] = v[q] = 0.f;
  }
  if (!rev) {
    xm2[0] = D[t];
    xm1[0] = D[(size_t)ntr + t];
  }
  float *const first = rev ? D + (size_t)(n - 1) * ntr + t : D + 2 * (size_t)ntr + t;   // sample 2
  const long long step = rev ? -(long long)ntr : (long long)ntr;
  const int m = n - 2;   // samples
  // Iteration k: section q takes sample k - q.
  auto iterate = [&](int k, float x, bool check) {
#pragma unroll
    for (int q = NS - 1; q >= 0; --q) {
      if (check && (k - q < 0 || k - q >= m)) continue;
      const float xc = q ? v[q - 1] : x;
      const float r = (((cf[q][0] * xc + cf[q][1] * xm1[q]) + cf[q][2] * xm2[q]) -
                       cf[q][3] * nm1[q]) - cf[q][4] * nm2[q];
      xm2[q] = xm1[q];
      xm1[q] = xc;
      nm2[q] = nm1[q];
      nm1[q] = r;
      v[q] = r;
    }
    if (k >= NS - 1) first[(k - (NS - 1)) * step] = v[NS - 1];
  };
  constexpr int U = 8;
  int k = 0;
  for (; k < NS - 1 && k < m; ++k) iterate(k, first[k * step], true);
  float x[U];
#pragma unroll
  for (int u = 0; u < U; ++u) x[u] = k + u < m ? first[(k + u) * step] : 0.f;
  for (; k + U <= m; k += U) {
    float y[U];
#pragma unroll
    for (int u = 0; u < U; ++u) y[u] = k + U + u < m ? first[(k + U + u) * step] : 0.f;
#pragma unroll
    for (int u = 0; u < U; ++u) iterate(k + u, x[u], false);
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = y[u];
  }
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (k + u < m) iterate(k + u, x[u], false);
  for (k = m; k < m + NS - 1; ++k) iterate(k, 0.f, true);
  if (!rev) D[t] = D[(size_t)ntr + t] = 0.f;
}

static void launch_bp_sections(int ntr, int n, int rev, int ns, const float *c, float *D,
                               cudaStream_t s, int *nlaunch) {
  const int g = (ntr + 31) / 32;
  for (int q = 0; q < ns; q += 4) {
    const float *cq = c + 5 * q;
    switch (ns - q < 4 ? ns - q : 4) {
      case 1: k_bp_sections<1><<<g, 32, 0, s>>>(ntr, n, rev, cq, D); break;
      case 2: k_bp_sections<2><<<g, 32, 0, s>>>(ntr, n, rev, cq, D); break;
      case 3: k_bp_sections<3><<<g, 32, 0, s>>>(ntr, n, rev, cq, D); break;
      default: k_bp_sections<4><<<g, 32, 0, s>>>(ntr, n, rev, cq, D);
    }
    ++*nlaunch;
  }
}

cudaError_t launch_bandpass(int ntr, int nt, int npad, int phase, int nlo, const float *clo,
                            int nhi, const float *chi, const float *lead, const float *trail,
                            const float *in, float *out, float *D, cudaStream_t s,
                            int *nlaunch) {
  const int n = nt + 2 * npad;
  const unsigned gx = (ntr + 31) / 32;
  k_bp_pad<<<gx * ((n + 31) / 32), 256, 0, s>>>(ntr, nt, npad, lead, trail, in, D);
  launch_bp_sections(ntr, n, 0, nlo, clo, D, s, nlaunch);
  if (phase == 0) launch_bp_sections(ntr, n, 1, nlo, clo, D, s, nlaunch);
  launch_bp_sections(ntr, n, 0, nhi, chi, D, s, nlaunch);
  if (phase == 0) launch_bp_sections(ntr, n, 1, nhi, chi, D, s, nlaunch);
  k_bp_cut<<<gx * ((nt + 31) / 32), 256, 0, s>>>(ntr, nt, npad, D, out);
  *nlaunch += 2;
  return cudaGetLastError();
}

cudaError_t launch_higdon_coeffs(const Geom &g, const float *vel_pad, float dt, float dxi,
                                 float dyi, float dzi, float *gz, float *gx, float *gy,
                                 cudaStream_t s) {
  const long long n1 = g.nmax1 - g.nmin1 + 1, n2 = g.nmax2 - g.nmin2 + 1,
                  n3 = g.nmax3 - g.nmin3 + 1;
  const long long tot = n2 * n3 + n1 * n3 + (g.nmax3 > 1 ? n1 * n2 : 0);
  k_higdon_coeffs<<<nblocks(tot, 256), 256, 0, s>>>(g, vel_pad, dt, dxi, dyi, dzi, gz, gx, gy);
  return cudaGetLastError();
}

cudaError_t launch_window_vel(int nz, int nx, int ny, float ox, float oy, float dx, float dy,
                              int nxw, int nyw, float oxw, float oyw, const float *big,
                              float *small, cudaStream_t s) {
  const long long n = (long long)nz * nxw * nyw;
  k_window_vel<<<nblocks(n, 256), 256, 0, s>>>(nz, nx, ny, ox, oy, dx, dy, nxw, nyw, oxw, oyw,
                                                big, small);
  return cudaGetLastError();
}

cudaError_t launch_copy_image(int nz, int nx, int ny, float ox, float oy, float dx, float dy,
                              int nxw, int nyw, float oxw, float oyw, const float *ims,
                              const float *ils, float *image, float *illum, cudaStream_t s) {
  const long long n = (long long)nz * nxw * nyw;
  k_copy_image<<<nblocks(n, 256), 256, 0, s>>>(nz, nx, ny, ox, oy, dx, dy, nxw, nyw, oxw, oyw,
                                                ims, ils, image, illum);
  return cudaGetLastError();
}

cudaError_t launch_residual(int nrec, int nt, const float *dobs, const float *mute, float *dmod,
                            float *resid, double *partial, cudaStream_t s) {
  k_residual<<<(nrec + RES_T - 1) / RES_T, 256, 0, s>>>(nrec, nt, dobs, mute, dmod, resid, partial);
  return cudaGetLastError();
}

cudaError_t launch_residual_nrm(int ntype, float thresh, int nrec, int nt, const float *dobs,
                                const float *mute, float *dmod, float *resid, double *partial,
                                float *maxabs, cudaStream_t s) {
  const bool need_max = ntype != SW_NRM_L1 && thresh == 0.0f;
  if (need_max)
    k_trace_maxabs<<<(nrec + 127) / 128, 128, 0, s>>>(nrec, nt, dobs, mute, dmod, maxabs);
  k_residual_nrm<<<(nrec + 127) / 128, 128, 0, s>>>(ntype, nrec, nt, dobs, mute, dmod, resid,
                                                    partial, thresh, need_max ? maxabs : nullptr);
  return cudaGetLastError();
}

}  // namespace swave
