// Real-time Green's function straight from a Lanczos tridiagonal T (gf_greater / gf_lesser,
// cmpy/exactdiag.py:248-302): <e1| exp(-i s (T - e0) t) |e1> for many times by the Chebyshev
// expansion of the exponential (Tal-Ezer and Kosloff, J. Chem. Phys. 81, 3967 (1984)), instead of
// the eigenpairs of T (at m = 2000 of the 8-site chain, t <= 50 and 1000 times: 0.8 ms against 96). With the spectrum of T inside [b - a, b + a] and x = (T - b) / a,
//   exp(-i s a t x) = sum_n (2 - delta_n0) (-i)^n J_n(s a t) T_n(x),
// so G(t) needs the moments mu_n = <e1|T_n(x)|e1>, n <= N, once, and per time the Bessel
// functions J_n(a t). J_n falls off beyond n = a t like the Airy function of (n - a t)
// (2 / (a t))^(1/3): N = a t + 14 (a t)^(1/3) + 40 leaves terms below 1e-21 out.
#include <algorithm>
#include <atomic>
#include <cmath>

#include "ed_common.cuh"

namespace ed {

constexpr int CHB_NT = 512;
constexpr int CHB_MMAX = 4096;   // four arrays of m doubles in one CTA's shared memory
constexpr int CHB_NMAX = 16384;  // largest order of the expansion

__host__ __device__ inline double cheb_order(double tau) { return tau + 14.0 * cbrt(tau) + 40.0; }

// Gershgorin interval of T = (alpha, beta): res = (b, a)
__global__ void __launch_bounds__(256) k_cheb_bounds(const double* __restrict__ alpha, const double* __restrict__ beta,
                                                     int m, double* __restrict__ res) {
  __shared__ double slo[8], shi[8];
  double lo = alpha[0], hi = alpha[0];
  bool bad = false;
  for (int i = threadIdx.x; i < m; i += 256) {
    const double r = (i > 0 ? fabs(beta[i]) : 0.0) + (i + 1 < m ? fabs(beta[i + 1]) : 0.0);
    bad |= !isfinite(alpha[i]) || !isfinite(r);
    lo = fmin(lo, alpha[i] - r);
    hi = fmax(hi, alpha[i] + r);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((threadIdx.x & 31) == 0) {
    slo[threadIdx.x >> 5] = lo;
    shi[threadIdx.x >> 5] = hi;
  }
  bad = __syncthreads_or(bad);
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      lo = fmin(lo, slo[w]);
      hi = fmax(hi, shi[w]);
    }
    const double b = 0.5 * (lo + hi);
    const double a = fmax(0.5 * (hi - lo) * (1.0 + 1e-14), fmax(1e-8 * fmax(fabs(lo), fabs(hi)), 1e-300));
    res[0] = bad ? nan("") : b;
    res[1] = bad ? nan("") : a;
  }
}

// mu[n] = (T_n(x) e1)_0, n = 0..N, by the three-term recurrence on vectors in shared memory, one
// block barrier a step. Element i of step n matters only for i <= min(n, N - n) (it takes i steps
// to get there and i to come back), so the work is a triangle of at most N/2 rows. Bound by the
// latency of a step (barrier, shared-memory loads, three dependent FP64 operations).
__global__ void __launch_bounds__(CHB_NT) k_cheb_moments(const double* __restrict__ alpha,
                                                         const double* __restrict__ beta, int m,
                                                         const double* __restrict__ ba, int N, double* __restrict__ mu) {
  extern __shared__ double sh[];
  double* d2 = sh;          // 2 (alpha - b) / a
  double* o2 = sh + m;      // 2 beta / a: o2[i] couples i - 1 and i; o2[0] = 0
  double* cur = sh + 2 * m;
  double* prv = sh + 3 * m;
  const double b = ba[0], ia = 1.0 / ba[1];
  for (int i = threadIdx.x; i < m; i += CHB_NT) {
    d2[i] = 2.0 * ((alpha[i] - b) * ia);
    o2[i] = i > 0 ? 2.0 * (beta[i] * ia) : 0.0;
    cur[i] = i == 0 ? 1.0 : 0.0;
    prv[i] = 0.0;
  }
  __syncthreads();
  // T_1 = x: the recurrence from T_{-1} = T_1, i.e. half of 2 x e1
  if (threadIdx.x == 0) {
    mu[0] = 1.0;
    prv[0] = 0.5 * d2[0];
    if (m > 1) prv[1] = 0.5 * o2[1];
    if (N >= 1) mu[1] = prv[0];
  }
  __syncthreads();
  {
    double* t = cur;
    cur = prv;
    prv = t;
  }
  for (int n = 2; n <= N; ++n) {
    const int top = min(min(n, N - n), m - 1);
    for (int i = threadIdx.x; i <= top; i += CHB_NT) {
      double v = fma(d2[i], cur[i], -prv[i]);
      if (i > 0) v = fma(o2[i], cur[i - 1], v);
      if (i + 1 < m) v = fma(o2[i + 1], cur[i + 1], v);
      prv[i] = v;
      if (i == 0) mu[n] = v;
    }
    __syncthreads();
    double* t = cur;
    cur = prv;
    prv = t;
  }
}

// out[k] (+)= -i s norm2 e^{-i s (b - e0) t_k} sum_n (2 - delta_n0) (-i)^n J_n(s a t_k) mu_n, one
// thread per time. The Bessel functions come from Miller's downward recurrence
// J_{n-1} = (2 n / tau) J_n - J_{n+1}, normalised by J_0^2 + 2 sum J_n^2 = 1 (no cancellation;
// J_n > 0 at the start), in the same loop as the two sums.
__global__ void __launch_bounds__(32) k_cheb_sum(const double* __restrict__ mu, int N, const double* __restrict__ ba,
                                                 double norm2, double e0, int sign, const double* __restrict__ t,
                                                 int64_t nt, double2* __restrict__ out, int accumulate) {
  const int64_t k = blockIdx.x * (int64_t)32 + threadIdx.x;
  if (k >= nt) return;
  const double b = ba[0], a = ba[1], tk = t[k];
  const double y = sign * a * tk, tau = fabs(y);
  double re, im;
  if (tau < 1e-9) {  // 1 - i y x: the next term is below 1e-18
    re = 1.0;
    im = N >= 1 ? -y * mu[1] : 0.0;
  } else {
    const int M = min(N, (int)ceil(cheb_order(tau)));
    const double r = 2.0 / tau;
    double jp = 0.0, j = 0x1p-80, even = 0.0, odd = 0.0, sq = 0.0;  // J_{n+1}, J_n
    for (int n = M; n >= 1; --n) {
      const double c = (n & 2) ? -mu[n] : mu[n];  // (-1)^(n/2) and (-1)^((n-1)/2)
      if (n & 1) odd = fma(c, j, odd);
      else even = fma(c, j, even);
      sq = fma(j, j, sq);
      const double jm = fma((double)n * r, j, -jp);
      jp = j;
      j = jm;
      if (((unsigned)__double2hiint(j) & 0x7fffffffu) > 0x5a000000u) {  // |j| > 2^416: keep in range
        const double sc = 0x1.0p-832;
        j *= sc;
        jp *= sc;
        even *= sc;
        odd *= sc;
        sq *= sc;
        sq *= sc;
      }
    }
    const double inv = 1.0 / sqrt(fma(2.0, sq, j * j));
    re = fma(2.0, even, j * mu[0]) * inv;
    im = -copysign(2.0, y) * odd * inv;
  }
  double sn, cs;
  sincos(-sign * (b - e0) * tk, &sn, &cs);
  const double fr = norm2 * (re * cs - im * sn), fi = norm2 * (re * sn + im * cs);
  double2 v = make_double2(sign * fi, -sign * fr);
  if (accumulate) { v.x += out[k].x; v.y += out[k].y; }
  out[k] = v;
}

}  // namespace ed

using namespace ed;

extern "C" {

ED_API ed_status ed_tevo_krylov(const double* d_alpha, const double* d_beta, int m, double norm2, double e0, int sign,
                                const double* d_t, int64_t n_t, double t_abs_max, double* d_out, int accumulate,
                                int* h_done, ed_stream_t stream) {
  if (!h_done) return fail(ED_ERR_INVALID_ARG, "null argument");
  *h_done = 0;
  if (m < 1 || n_t < 0) return fail(ED_ERR_INVALID_ARG, "m must be >= 1 and n_t >= 0");
  if (sign != 1 && sign != -1) return fail(ED_ERR_INVALID_ARG, "sign must be +1 or -1");
  if (n_t == 0) { *h_done = 1; return ED_OK; }
  if (!d_alpha || !d_beta || !d_t || !d_out) return fail(ED_ERR_INVALID_ARG, "null argument");
  if (!std::isfinite(e0)) return fail(ED_ERR_NONFINITE, "e0 is not finite");
  if (m > CHB_MMAX || !std::isfinite(t_abs_max) || t_abs_max < 0.0) return ED_OK;
  DeviceContext* ctx;
  ED_TRY(device_context(&ctx));
  const size_t smem = (size_t)4 * m * sizeof(double);
  if (smem > (size_t)ctx->smem_optin) return ED_OK;
  if (smem > 48 * 1024) {
    static std::atomic<uint64_t> set{0};
    const uint64_t bit = 1ull << (ctx->device & 63);
    if (!(set.load() & bit)) {
      ED_CUDA(cudaFuncSetAttribute(k_cheb_moments, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->smem_optin));
      set.fetch_or(bit);
    }
  }
  cudaStream_t s = as_stream(stream);
  double* buf = nullptr;
  ED_CUDA(cudaMallocAsync((void**)&buf, (2 + CHB_NMAX + 1) * sizeof(double), s));
  auto run = [&]() -> ed_status {
    k_cheb_bounds<<<1, 256, 0, s>>>(d_alpha, d_beta, m, buf);
    ED_CHECK_LAUNCH("k_cheb_bounds");
    double ba[2];
    ED_CUDA(cudaMemcpyAsync(ba, buf, sizeof(ba), cudaMemcpyDeviceToHost, s));
    ED_CUDA(cudaStreamSynchronize(s));
    const double order = std::ceil(cheb_order(ba[1] * t_abs_max));
    // The expansion's time grows with its order N, the eigenpairs' with m; at 1000 times (us,
    // expansion / eigenpairs): m = 32: N = 250: 403 / 533, N = 1000: 863; m = 400: N = 1000: 1026 /
    // 2863, N = 4000: 3681; m = 2000: N = 4000: 5821 / 29549, N = 16000: 33961.
    if (!(order <= std::min<double>(CHB_NMAX, std::max(400.0, 7.0 * m)))) return ED_OK;
    const int N = (int)order;
    k_cheb_moments<<<1, CHB_NT, smem, s>>>(d_alpha, d_beta, m, buf, N, buf + 2);
    k_cheb_sum<<<(unsigned)((n_t + 31) / 32), 32, 0, s>>>(buf + 2, N, buf, norm2, e0, sign, d_t, n_t, (double2*)d_out,
                                                          accumulate);
    ED_CHECK_LAUNCH_N("ed_tevo_krylov", 2);
    *h_done = 1;
    return ED_OK;
  };
  const ed_status st = run();
  cudaFreeAsync(buf, s);
  return st;
}

}  // extern "C"
