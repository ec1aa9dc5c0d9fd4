// Green's-function kernels: the continued fraction of the Lanczos coefficients (new; the
// reference only has dense Lanczos helpers, cmpy/exactdiag.py:324-375), the thermal
// Lehmann pole sum of _accumulate_sum (cmpy/exactdiag.py:110-129), the real-time Green's
// function from Krylov spectral weights (gf_greater / gf_lesser, cmpy/exactdiag.py:248-302)
// and its Laplace transform to complex frequencies (fourier_t2z, cmpy/exactdiag.py:311-316).
// Complex numbers are interleaved (re, im) FP64 pairs.
#include <algorithm>
#include <cmath>

#include "ed_cf.cuh"
#include "ed_plan.cuh"

namespace ed {

// G(z) = sign * norm2 / (z' - a0 - b1^2 / (z' - a1 - ...)),  z' = sign * z + shift; one thread per
// frequency, blocks of one warp (a few thousand frequencies are spread over the SMs, whose FP64 pipes a
// single warp each already holds: 200 levels at 2048 frequencies 120 -> 87 us)
constexpr int CF_NT = 32;
__global__ void __launch_bounds__(CF_NT) k_cf(const double* __restrict__ a, const double* __restrict__ b, int n,
                                              double norm2, double shift, int sign, const double2* __restrict__ z,
                                              int64_t nz, double2* __restrict__ g, int accumulate) {
  __shared__ double2 st[CF_TILE];
  const int64_t i = blockIdx.x * (int64_t)CF_NT + threadIdx.x;
  const double2 zi = i < nz ? z[i] : make_double2(0.0, 1.0);
  double2 r = cf_value(a, b, n, sign * zi.x + shift, sign * zi.y, sign * norm2, st);
  if (i >= nz) return;
  if (accumulate) { r.x += g[i].x; r.y += g[i].y; }
  g[i] = r;
}

// coef[m*nd + n] = ov[m, n] * (w_n + w'_m),  pole = E'_m - E_n;  w = exp(-beta (E - emin))
// (all ones when beta is not finite, cmpy/exactdiag.py:114-119)
__global__ void k_lehmann_poles(const double* __restrict__ e, int64_t nd, const double* __restrict__ ep, int64_t ndp,
                                const double* __restrict__ ov, double beta, double emin, double* __restrict__ coef,
                                double* __restrict__ pole) {
  const int64_t tot = nd * ndp;
  const bool fin = isfinite(beta);
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < tot; k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = k / nd, n = k - m * nd;
    const double wn = fin ? exp(-beta * (e[n] - emin)) : 1.0;
    const double wm = fin ? exp(-beta * (ep[m] - emin)) : 1.0;
    coef[k] = ov[k] * (wn + wm);
    pole[k] = ep[m] - e[n];
  }
}

// part[q][z] = sum of coef_k / (z - pole_k) over the terms of chunk q (blockIdx.y), one thread
// per frequency, the terms staged in shared memory. Bound by the FP64 pipe (eight operations a
// term and frequency): the terms are split over as many blocks as fill the GPU, because the
// frequencies alone do not: 512 of them are four blocks, which took 8.4 ms for the mean sector
// pair of the 6-site chain. Split, its thermal G over all sectors went from 567 to 222 ms.
constexpr int LEH_NT = 128;  // frequencies per block
constexpr int LEH_T = 256;   // terms per tile
__global__ void __launch_bounds__(LEH_NT) k_lehmann_sum(const double* __restrict__ coef, const double* __restrict__ pole,
                                                        int64_t nt, int64_t chunk, const double2* __restrict__ z,
                                                        int64_t nz, double2* __restrict__ part) {
  __shared__ double2 st[LEH_T];
  const int64_t i = blockIdx.x * (int64_t)LEH_NT + threadIdx.x;
  const double2 zi = i < nz ? z[i] : make_double2(0.0, 1.0);
  const double zm2 = zi.y * zi.y;
  const int64_t k0 = blockIdx.y * chunk, k1 = min(nt, k0 + chunk);
  double gr = 0.0, gs = 0.0;
  for (int64_t t0 = k0; t0 < k1; t0 += LEH_T) {
    const int tn = (int)min((int64_t)LEH_T, k1 - t0);
    __syncthreads();
    for (int t = threadIdx.x; t < tn; t += LEH_NT) st[t] = make_double2(coef[t0 + t], pole[t0 + t]);
    __syncthreads();
#pragma unroll 4
    for (int t = 0; t < tn; ++t) {
      const double2 cp = st[t];
      if (cp.x == 0.0) continue;  // uniform over the block
      const double ar = zi.x - cp.y;
      const double inv = cp.x * rcp_f64(fma(ar, ar, zm2));
      gr = fma(ar, inv, gr);
      gs += inv;
    }
  }
  if (i < nz) part[blockIdx.y * nz + i] = make_double2(gr, -zi.y * gs);
}

// g[z] (+)= the chunk sums, one warp per frequency, in a fixed order
__global__ void __launch_bounds__(LEH_NT) k_chunk_reduce(const double2* __restrict__ part, int nq, int64_t nz,
                                                         double2* __restrict__ g, int accumulate) {
  const int64_t i = (blockIdx.x * (int64_t)LEH_NT + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= nz) return;
  double r = 0.0, m = 0.0;
  for (int q = lane; q < nq; q += 32) {
    const double2 v = part[q * nz + i];
    r += v.x;
    m += v.y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    r += __shfl_xor_sync(0xffffffffu, r, o);
    m += __shfl_xor_sync(0xffffffffu, m, o);
  }
  if (lane == 0) {
    if (accumulate) { r += g[i].x; m += g[i].y; }
    g[i] = make_double2(r, m);
  }
}


// out[n] (+)= -i*sign * sum_k w_k exp(-i sign (lam_k - e0) t_n)
// (sign = +1: greater function of c^dag|gs>; sign = -1: lesser function of c|gs>)
constexpr int TEVO_T = 1024;
__global__ void k_tevo_sum(const double* __restrict__ lam, const double* __restrict__ w, int64_t m, double e0, int sign,
                           const double* __restrict__ t, int64_t nt, double2* __restrict__ out, int accumulate) {
  __shared__ double sl[TEVO_T], sw[TEVO_T];
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const double tn = n < nt ? t[n] : 0.0;
  double sr = 0.0, si = 0.0;
  for (int64_t k0 = 0; k0 < m; k0 += TEVO_T) {
    __syncthreads();
    for (int k = threadIdx.x; k < TEVO_T; k += blockDim.x) {
      sl[k] = k0 + k < m ? lam[k0 + k] - e0 : 0.0;
      sw[k] = k0 + k < m ? w[k0 + k] : 0.0;
    }
    __syncthreads();
    const int kn = (int)((m - k0) < TEVO_T ? (m - k0) : TEVO_T);
    for (int k = 0; k < kn; ++k) {
      double sn, cs;
      sincos(sign * sl[k] * tn, &sn, &cs);
      sr = fma(sw[k], cs, sr);
      si = fma(-sw[k], sn, si);
    }
  }
  if (n < nt) {
    // -i*sign * (sr + i si) = sign*si - i sign*sr
    double2 r = make_double2(sign * si, -sign * sr);
    if (accumulate) { r.x += out[n].x; r.y += out[n].y; }
    out[n] = r;
  }
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ double2 cexp_(double2 x) {
  double sn, cs;
  sincos(x.y, &sn, &cs);
  const double r = exp(x.x);
  return make_double2(r * cs, r * sn);
}
__device__ __forceinline__ double2 cdiv(double2 a, double2 b) {
  const double d = b.x * b.x + b.y * b.y;
  return make_double2((a.x * b.x + a.y * b.y) / d, (a.y * b.x - a.x * b.y) / d);
}
// phi2(x) = (e^x - 1 - x)/x^2 and phi1 - phi2, phi1(x) = (e^x - 1)/x, of a complex x. |x| < 1/4: the Taylor series
// of phi2, sum x^k/(k+2)!, k < 13 (the first term left out is below 0.25^13/15! < 2e-20), and phi1 = 1 + x phi2,
// added in the order (1 - phi2) + x phi2. Elsewhere phi1 by its own quotient: 1 + x phi2 would keep the absolute
// rounding of 1 in a value of size 1/|x| (a relative error of 2^-53 |x|).
__constant__ double PHI2_C[13] = {1.0 / 2,         1.0 / 6,          1.0 / 24,          1.0 / 120,
                                  1.0 / 720,       1.0 / 5040,       1.0 / 40320,       1.0 / 362880,
                                  1.0 / 3628800,   1.0 / 39916800,   1.0 / 479001600,   1.0 / 6227020800.0,
                                  1.0 / 87178291200.0};
__device__ __forceinline__ void segment_weights(double2 x, double2* p2, double2* p12) {
  if (x.x * x.x + x.y * x.y < 0.0625) {
    double2 a = make_double2(PHI2_C[12], 0.0);
#pragma unroll
    for (int k = 11; k >= 0; --k) {
      a = cmul(a, x);
      a.x += PHI2_C[k];
    }
    const double2 xa = cmul(x, a);
    *p2 = a;
    *p12 = make_double2((1.0 - a.x) + xa.x, xa.y - a.y);
    return;
  }
  const double2 ex = cexp_(x);
  const double2 em1 = make_double2(ex.x - 1.0, ex.y);
  const double2 p1 = cdiv(em1, x);
  *p2 = cdiv(make_double2(em1.x - x.x, em1.y - x.y), cmul(x, x));
  *p12 = make_double2(p1.x - p2->x, p1.y - p2->y);
}

// Laplace transform G(z) = int_{t_0}^{t_{N-1}} e^{i z t} g(t) dt of samples g(t_j), the segments of
// chunk q = blockIdx.y, one thread per frequency:
//   method 0: exact integral of the piecewise-linear interpolant, segment by segment
//     int_{t_j}^{t_j+h} e^{u t} g dt = h e^{u t_j} [g_j phi2(u h) + g_{j+1} (phi1 - phi2)(u h)],  u = i z;
//   method 1: trapezoidal rule.
// Bound by the FP64 pipe (a complex exponential and the series per segment and frequency), so the
// segments are split over as many blocks as fill the GPU: one thread per frequency over all of 1000
// samples was eight blocks, with the series' factorials formed in the loop (36.1 ms for 1000
// samples and 1000 frequencies, 0.31 ms now).
__global__ void __launch_bounds__(LEH_NT) k_laplace_t2z(const double* __restrict__ t, const double2* __restrict__ g,
                                                        int64_t nt, int64_t chunk, const double2* __restrict__ z,
                                                        int64_t nz, int method, double2* __restrict__ part) {
  const int64_t i = blockIdx.x * (int64_t)LEH_NT + threadIdx.x;
  if (i >= nz) return;
  const double2 u = make_double2(-z[i].y, z[i].x);  // i z
  double2 acc = make_double2(0.0, 0.0);
  const int64_t j0 = blockIdx.y * chunk, j1 = min(nt - 1, j0 + chunk);
  for (int64_t j = j0; j < j1; ++j) {
    const double h = t[j + 1] - t[j];
    const double2 ej = cexp_(make_double2(u.x * t[j], u.y * t[j]));
    if (method == 0) {
      const double2 x = make_double2(u.x * h, u.y * h);
      double2 p2, p12;
      segment_weights(x, &p2, &p12);
      const double2 c0 = cmul(g[j], p2);
      const double2 c1 = cmul(g[j + 1], p12);
      const double2 seg = cmul(ej, make_double2(h * (c0.x + c1.x), h * (c0.y + c1.y)));
      acc.x += seg.x;
      acc.y += seg.y;
    } else {
      const double2 ej1 = cexp_(make_double2(u.x * t[j + 1], u.y * t[j + 1]));
      const double2 a = cmul(ej, g[j]), b = cmul(ej1, g[j + 1]);
      acc.x += 0.5 * h * (a.x + b.x);
      acc.y += 0.5 * h * (a.y + b.y);
    }
  }
  part[blockIdx.y * nz + i] = acc;
}

}  // namespace ed

using namespace ed;

extern "C" {

ED_API ed_status ed_gf_continued_fraction(const double* d_alpha, const double* d_beta, int n_lev, double norm2,
                                          double shift, int sign, const double* d_z, int64_t n_z, double* d_g,
                                          int accumulate, ed_stream_t stream) {
  if (n_lev < 1) return fail(ED_ERR_INVALID_ARG, "n_lev must be >= 1");
  if (sign != 1 && sign != -1) return fail(ED_ERR_INVALID_ARG, "sign must be +1 or -1");
  if (n_z < 0) return fail(ED_ERR_INVALID_ARG, "negative n_z");
  if (n_z == 0) return ED_OK;
  if (!d_alpha || !d_beta || !d_z || !d_g) return fail(ED_ERR_INVALID_ARG, "null argument");
  k_cf<<<(unsigned)((n_z + CF_NT - 1) / CF_NT), CF_NT, 0, as_stream(stream)>>>(
      d_alpha, d_beta, n_lev, norm2, shift, sign, (const double2*)d_z, n_z, (double2*)d_g, accumulate);
  ED_CHECK_LAUNCH("k_cf");
  return ED_OK;
}

ED_API ed_status ed_lehmann_accumulate(const double* d_e, int64_t nd, const double* d_ep, int64_t ndp,
                                       const double* d_ov, double beta, double emin, const double* d_z, int64_t nz,
                                       double* d_g, ed_stream_t stream) {
  if (nd < 0 || ndp < 0 || nz < 0) return fail(ED_ERR_INVALID_ARG, "negative size");
  if (nd == 0 || ndp == 0 || nz == 0) return ED_OK;
  if (!d_e || !d_ep || !d_ov || !d_z || !d_g) return fail(ED_ERR_INVALID_ARG, "null argument");
  if (std::isnan(beta)) return fail(ED_ERR_NONFINITE, "beta is NaN");
  DeviceContext* ctx;
  ED_TRY(device_context(&ctx));
  cudaStream_t s = as_stream(stream);
  const int64_t nt = nd * ndp;
  // chunks of terms: eight blocks per SM over all frequencies, at least one tile of terms each
  const int64_t zb = (nz + LEH_NT - 1) / LEH_NT;
  int64_t nq = std::min<int64_t>((nt + LEH_T - 1) / LEH_T, std::max<int64_t>(1, (int64_t)ctx->num_sms * 8 / zb));
  const int64_t chunk = ((nt + nq - 1) / nq + LEH_T - 1) / LEH_T * LEH_T;
  nq = (nt + chunk - 1) / chunk;
  double *coef = nullptr, *pole = nullptr;
  double2* part = nullptr;
  ED_CUDA(cudaMallocAsync(&coef, (2 * nt + 2 * nq * nz) * sizeof(double), s));
  pole = coef + nt;
  part = (double2*)(coef + 2 * nt);
  k_lehmann_poles<<<grid_for(nt, 256, ctx->num_sms * 8), 256, 0, s>>>(d_e, nd, d_ep, ndp, d_ov, beta, emin, coef, pole);
  k_lehmann_sum<<<dim3((unsigned)zb, (unsigned)nq), LEH_NT, 0, s>>>(coef, pole, nt, chunk, (const double2*)d_z, nz, part);
  k_chunk_reduce<<<(unsigned)((nz * 32 + LEH_NT - 1) / LEH_NT), LEH_NT, 0, s>>>(part, (int)nq, nz, (double2*)d_g, 1);
  ED_CHECK_LAUNCH_N("ed_lehmann_accumulate", 3);
  ED_CUDA(cudaFreeAsync(coef, s));
  return ED_OK;
}

ED_API ed_status ed_tevo_sum(const double* d_lam, const double* d_w, int64_t m, double e0, int sign, const double* d_t,
                             int64_t n_t, double* d_out, int accumulate, ed_stream_t stream) {
  if (m < 0 || n_t < 0) return fail(ED_ERR_INVALID_ARG, "negative size");
  if (sign != 1 && sign != -1) return fail(ED_ERR_INVALID_ARG, "sign must be +1 or -1");
  if (n_t == 0) return ED_OK;
  if ((m > 0 && (!d_lam || !d_w)) || !d_t || !d_out) return fail(ED_ERR_INVALID_ARG, "null argument");
  if (!std::isfinite(e0)) return fail(ED_ERR_NONFINITE, "e0 is not finite");
  k_tevo_sum<<<(unsigned)((n_t + 127) / 128), 128, 0, as_stream(stream)>>>(d_lam, d_w, m, e0, sign, d_t, n_t,
                                                                           (double2*)d_out, accumulate);
  ED_CHECK_LAUNCH("k_tevo_sum");
  return ED_OK;
}

ED_API ed_status ed_laplace_t2z(const double* d_t, const double* d_gt, int64_t n_t, const double* d_z, int64_t n_z,
                                int method, double* d_out, ed_stream_t stream) {
  if (n_t < 0 || n_z < 0) return fail(ED_ERR_INVALID_ARG, "negative size");
  if (method != 0 && method != 1) return fail(ED_ERR_INVALID_ARG, "method must be 0 (linear) or 1 (trapezoid)");
  if (n_z == 0) return ED_OK;
  if (!d_t || !d_gt || !d_z || !d_out) return fail(ED_ERR_INVALID_ARG, "null argument");
  DeviceContext* ctx;
  ED_TRY(device_context(&ctx));
  cudaStream_t s = as_stream(stream);
  // chunks of segments: eight blocks per SM over all frequencies
  const int64_t seg = std::max<int64_t>(1, n_t - 1), zb = (n_z + LEH_NT - 1) / LEH_NT;
  int64_t nq = std::min<int64_t>(seg, std::max<int64_t>(1, (int64_t)ctx->num_sms * 8 / zb));
  const int64_t chunk = (seg + nq - 1) / nq;
  nq = (seg + chunk - 1) / chunk;
  double2* part = nullptr;
  ED_CUDA(cudaMallocAsync(&part, nq * n_z * sizeof(double2), s));
  k_laplace_t2z<<<dim3((unsigned)zb, (unsigned)nq), LEH_NT, 0, s>>>(d_t, (const double2*)d_gt, n_t, chunk,
                                                                   (const double2*)d_z, n_z, method, part);
  k_chunk_reduce<<<(unsigned)((n_z * 32 + LEH_NT - 1) / LEH_NT), LEH_NT, 0, s>>>(part, (int)nq, n_z, (double2*)d_out, 0);
  ED_CHECK_LAUNCH_N("k_laplace_t2z", 2);
  ED_CUDA(cudaFreeAsync(part, s));
  return ED_OK;
}

}  // extern "C"
