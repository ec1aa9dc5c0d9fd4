// Thermal sums of one sector over its eigenpairs: the partition function, the occupation of a site and
// its double occupation (occupation / double_occupation and the bookkeeping of
// GreensFunctionMeasurement.accumulate, cmpy/exactdiag.py:60-107, 137-212) in one pass over the
// eigenvectors. What bounds it is launches and waits, not the pass: 42 sectors of the 6-site chain took
// 42 x (36 tensor operations, 4 waits for a scalar), 40 of the 86 ms of its thermal G; here two launches
// and one wait each.
#include <cmath>

#include "ed_plan.cuh"

namespace ed {

constexpr int TH_NT = 256;

struct ThermalArgs {
  const double* e;        // [n]
  int64_t n;
  const double* v;        // element i of eigenvector k at v[i * si + k * sk]
  int64_t si, sk;
  const int64_t* states;  // [nu] up, then [nd] dn
  int64_t nu, nd;
  int site, dn;           // the occupation's species
  int occ;                // 0: energies alone
  double beta, emin;
};

// the smallest energy (the block's threads together) and e0 = min(emin, it)
__device__ __forceinline__ double2 thermal_min(const ThermalArgs& a, double* sm) {
  double m = INFINITY;
  for (int64_t k = threadIdx.x; k < a.n; k += TH_NT) m = fmin(m, a.e[k]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmin(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
  __syncthreads();
  for (int w = 0; w < TH_NT / 32; ++w) m = fmin(m, sm[w]);
  __syncthreads();
  return make_double2(m, m < a.emin ? m : a.emin);
}

// block b: the weights and occupations of its eigenvectors -> part[3 b ..]. ROWS: the vectors' elements are
// closest together (a warp per vector), else the vectors are (a thread per vector).
template <bool ROWS>
__global__ void __launch_bounds__(TH_NT) k_thermal_sums(const ThermalArgs a, double* part) {
  __shared__ double sm[TH_NT / 32][3];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double e0 = thermal_min(a, &sm[0][0]).y;
  double z = 0.0, occ = 0.0, dbl = 0.0;
  const int64_t first = blockIdx.x * (int64_t)(ROWS ? TH_NT / 32 : TH_NT) + (ROWS ? warp : (int)threadIdx.x);
  const int64_t step = gridDim.x * (int64_t)(ROWS ? TH_NT / 32 : TH_NT);
  for (int64_t k = first; k < a.n; k += step) {
    const double w = exp(-a.beta * (a.e[k] - e0));
    double o = 0.0, b = 0.0;
    if (a.occ) {
      const double* v = a.v + k * a.sk;
      for (int64_t i = ROWS ? lane : 0; i < a.nu * a.nd; i += ROWS ? 32 : 1) {
        const int64_t u = i / a.nd, d = i - u * a.nd;
        const int bu = (int)(a.states[u] >> a.site) & 1, bd = (int)(a.states[a.nu + d] >> a.site) & 1;
        if (!(a.dn ? bd : bu)) continue;
        const double x = v[i * a.si];
        o = fma(x, x, o);
        if (bu & bd) b = fma(x, x, b);
      }
    }
    if (!ROWS || lane == 0) z += w;
    occ = fma(w, o, occ);
    dbl = fma(w, b, dbl);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    z += __shfl_xor_sync(0xffffffffu, z, o);
    occ += __shfl_xor_sync(0xffffffffu, occ, o);
    dbl += __shfl_xor_sync(0xffffffffu, dbl, o);
  }
  if (lane == 0) {
    sm[warp][0] = z;
    sm[warp][1] = occ;
    sm[warp][2] = dbl;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = 0.0;
    for (int w = 0; w < TH_NT / 32; ++w) t += sm[w][threadIdx.x];
    part[3 * blockIdx.x + threadIdx.x] = t;
  }
}

// out = {smallest energy, partition function, occupation, double occupation}
__global__ void __launch_bounds__(TH_NT) k_thermal_final(const ThermalArgs a, const double* part, int blocks,
                                                         double* out) {
  __shared__ double sm[TH_NT / 32];
  const double m = thermal_min(a, sm).x;
  if (threadIdx.x == 0) out[0] = m;
  if (threadIdx.x >= 96) return;
  const int q = threadIdx.x >> 5;
  double t = 0.0;
  for (int b = threadIdx.x & 31; b < blocks; b += 32) t += part[3 * b + q];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) out[1 + q] = t;
}

}  // namespace ed

using namespace ed;

extern "C" {

ED_API ed_status ed_thermal_sums(const double* d_evals, int64_t n, const double* d_evecs, int64_t row_stride,
                                 int64_t col_stride, const int64_t* d_states, int64_t n_up_states,
                                 int64_t n_dn_states, int site, int dn, int occ, double beta, double emin,
                                 double* h_out, ed_stream_t stream) {
  if (n < 1 || !d_evals || !h_out) return fail(ED_ERR_INVALID_ARG, "need eigenvalues and an output");
  if (occ && (!d_evecs || !d_states || n_up_states < 1 || n_dn_states < 1))
    return fail(ED_ERR_INVALID_ARG, "the occupations need eigenvectors and states");
  if (site < 0 || site > 62) return fail(ED_ERR_INVALID_ARG, "site must be in [0, 62]");
  DeviceContext* ctx;
  ED_TRY(device_context(&ctx));
  cudaStream_t s = as_stream(stream);
  const ThermalArgs a{d_evals, n,    d_evecs, row_stride, col_stride, d_states, n_up_states,
                      n_dn_states, site, dn,   occ,     beta,       emin};
  const bool rows = std::llabs(row_stride) <= std::llabs(col_stride);
  const int64_t per = rows ? TH_NT / 32 : TH_NT;
  const int blocks = (int)std::min<int64_t>((n + per - 1) / per, ctx->num_sms * 4);
  double* buf = nullptr;
  ED_CUDA(cudaMallocAsync((void**)&buf, (3 * (size_t)blocks + 4) * sizeof(double), s));
  if (rows) k_thermal_sums<true><<<blocks, TH_NT, 0, s>>>(a, buf + 4);
  else k_thermal_sums<false><<<blocks, TH_NT, 0, s>>>(a, buf + 4);
  k_thermal_final<<<1, TH_NT, 0, s>>>(a, buf + 4, blocks, buf);
  const cudaError_t e = cudaGetLastError();
  count_launches(2);
  cudaError_t c = cudaMemcpyAsync(h_out, buf, 4 * sizeof(double), cudaMemcpyDeviceToHost, s);
  cudaFreeAsync(buf, s);
  if (e != cudaSuccess) return cuda_fail(e, "k_thermal_sums");
  if (c == cudaSuccess) c = cudaStreamSynchronize(s);
  if (c != cudaSuccess) return cuda_fail(c, "ed_thermal_sums");
  return ED_OK;
}

}  // extern "C"
