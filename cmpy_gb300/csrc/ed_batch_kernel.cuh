// The batched Lanczos kernel and its launch (included by the files that instantiate them).
#pragma once

#include "ed_batch.cuh"

namespace ed {

// (CTAs of 288 and 544 threads: three and two to an SM)
template <int NT, int CS>
__global__ void __launch_bounds__(NT, NT == 288 ? 3 : (NT <= 544 ? 2 : 1)) k_batch_lanczos(const BatchProblem* __restrict__ probs,
                                                      const int* __restrict__ order, int n, int K, double tol,
                                                      int check_every, uint64_t seed,
                                                      const double* const* __restrict__ starts, int want_vector,
                                                      size_t smem_budget, BatchOut out, BatchWork wk) {
  extern __shared__ __align__(16) unsigned char res_sm[];
  __shared__ int sh_p;
  __shared__ ResShared s;
  __shared__ BatchProblem P;
  const int rk = CS > 1 ? (int)(blockIdx.x % CS) : 0;
  const int64_t cid = blockIdx.x / CS;  // the cluster's vector slots
  ResIo io;
  io.run.K = K;
  io.run.tol = tol;
  io.run.check_every = check_every;
  io.run.rk = rk;
  io.run.R = wk.slots + cid * 5 * wk.dmax;
  io.run.Rp = io.run.R + wk.dmax;
  io.run.W = io.run.Rp + wk.dmax;
  io.run.store = nullptr;
  io.acc_lo = (uint64_t*)(io.run.W + wk.dmax);
  io.acc_hi = (int64_t*)(io.acc_lo + wk.dmax);
  // this CTA's tridiagonal work, eigenvector, copies of alpha, beta, and exponents
  io.run.work = wk.tri + (int64_t)blockIdx.x * 8 * (K + 2);
  io.run.c = io.run.work + 5 * (K + 2);
  io.run.alpha = io.run.c + (K + 2);
  io.run.beta = io.run.alpha + (K + 2);
  io.run.exps = wk.exps + (int64_t)blockIdx.x * (K + 2);
  io.Ck = wk.coefs + (int64_t)blockIdx.x * (K + 2);
  while (true) {
    // rank 0 pulls the next problem; every CTA of the cluster reads it from rank 0
    if (threadIdx.x == 0 && rk == 0) sh_p = atomicAdd(wk.queue, 1);
    csync<CS>();
    int q;
    if constexpr (CS > 1) q = *cg::this_cluster().map_shared_rank(&sh_p, 0);
    else q = sh_p;
    csync<CS>();
    if (q >= n) break;
    const int p = order[q];
    for (int i = threadIdx.x; i < (int)(sizeof(BatchProblem) / 4); i += NT) ((int*)&P)[i] = ((const int*)(probs + p))[i];
    __syncthreads();
    io.run.start = starts ? starts[p] : nullptr;
    io.run.seed = seed + 0x9E37ull * (uint64_t)p;
    io.alpha = out.alpha + (int64_t)p * K;
    io.beta = out.beta + (int64_t)p * (K + 1);
    io.energy = out.energy ? out.energy + p : nullptr;
    io.residual = out.energy ? out.residual + p : nullptr;
    io.steps = out.steps + p;
    io.vec = want_vector && out.vec ? out.vec + out.vec_off[p] : nullptr;
    const ResLayout L = res_layout(P.nu, P.nd, P.quads, NT, CS, smem_budget);
    if (P.diag64) res_dispatch<NT, CS, true>(P, L, res_sm, io, s);
    else res_dispatch<NT, CS, false>(P, L, res_sm, io, s);
    csync<CS>();  // the cluster's slots and P are free for the next problem
  }
  csync<CS>();  // no CTA leaves while another may still read its shared memory
}

template <int NT, int CS>
ed_status launch_batch(const ed_batch_s* b, int grid, int per_sm, int K, double tol, int check_every, uint64_t seed,
                              const double* const* starts, int want_vector, const BatchOut& out, const BatchWork& wk,
                              cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(NT);
  const size_t budget = batch_smem(b, NT, CS, per_sm);
  cfg.dynamicSmemBytes = budget;
  cfg.stream = s;
  if (budget > 0) {
    static std::atomic<uint64_t> done{0};
    const uint64_t bit = 1ull << (b->ctx->device & 63);
    if (!(done.load() & bit)) {
      cudaFuncAttributes fa;
      ED_CUDA(cudaFuncGetAttributes(&fa, k_batch_lanczos<NT, CS>));
      if (fa.sharedSizeBytes > RES_STATIC) return fail(ED_ERR_CUDA, "k_batch_lanczos: static shared memory above its bound");
      ED_CUDA(cudaFuncSetAttribute(k_batch_lanczos<NT, CS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   b->ctx->smem_optin - (int)fa.sharedSizeBytes));
      done.fetch_or(bit);
    }
  }
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CS > 1 ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_batch_lanczos<NT, CS>, (const BatchProblem*)b->d_probs,
                                           (const int*)b->d_order, b->n, K, tol, check_every, seed, starts, want_vector,
                                           budget, out, wk);
  if (e != cudaSuccess) return cuda_fail(e, "k_batch_lanczos");
  ED_CHECK_LAUNCH("k_batch_lanczos");
  return ED_OK;
}

template <int NT, int CS>
int clusters_for() {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CS * 16);
  cfg.blockDim = dim3(NT);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, k_batch_lanczos<NT, CS>, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return n;
}

}  // namespace ed
