// One Lanczos run of a small fixed-point sector as a single launch of one thread-block cluster
// (ed_resident.cuh) in place of two launches a step.
//
// What bounds it: the launched steps cost 23-26 us whatever the sector's size below ~20,000 states (two
// launches, their reductions through global memory, a grid that is mostly idle); a cluster's
// step costs its three cluster barriers, two chains of scalars and its eighth of the elements. Measured,
// us a step, launched / one CTA / 8 CTAs of 512 threads: 36 states 26.4 / 6.2 / 7.1, 400 states 23.2 / 5.4 /
// 5.8, 1225 states 24.2 / 7.5 / 6.1, 3920 states 26.4 / 13.3 / 6.9, 10584 states 26.0 / 29.3 / 9.6, 15876
// states 26.1 / 42.3 / 13.7. Hence always the cluster of 8, and always when the vectors fit.
#include <atomic>

#include "ed_lzcheck.cuh"
#include "ed_resident.cuh"

namespace ed {

namespace {
constexpr int RUN_NT = 512, RUN_CS = 8;
constexpr size_t RUN_STATIC = 5 * 1024;  // bound of the kernel's static shared memory
}  // namespace

struct ResSingle {
  const double* start;
  int K;
  double tol;
  int check_every;
  double *alpha, *beta, *c, *work, *norm;
  int zero_beta0;
  int32_t* exps;
  int64_t* store;
  int *stop, *steps, *status;
  TriResult* tri;
};

__global__ void __launch_bounds__(RUN_NT, 1) k_res_run(const __grid_constant__ BatchProblem prob, const ResLayout L,
                                                       const ResSingle a) {
  extern __shared__ __align__(16) unsigned char res_sm[];
  __shared__ ResShared s;
  __shared__ BatchProblem P;
  const int rk = (int)blockIdx.x;
  for (int i = threadIdx.x; i < (int)(sizeof(BatchProblem) / 4); i += RUN_NT) ((int*)&P)[i] = ((const int*)&prob)[i];
  __syncthreads();
  res_tables(P, L, res_sm);
  const ResTables T = res_offsets(L);
  ResRun io = {};
  io.start = a.start;
  io.K = a.K;
  io.tol = a.tol;
  io.check_every = a.check_every;
  io.rk = rk;
  if (rk == 0) {
    io.alpha = a.alpha;
    io.beta = a.beta;
    io.c = a.c;
    io.work = a.work;
    io.exps = a.exps;
  }
  io.store = a.store;
  const int m = P.diag64 ? res_recurrence<RUN_NT, RUN_CS, RES_ALL, true>(P, T, io, s)
                         : res_recurrence<RUN_NT, RUN_CS, RES_ALL, false>(P, T, io, s);
  if (threadIdx.x == 0 && rk == 0) {
    if (m == 0) {
      *a.status = a.beta[0] == 0.0 ? RES_ZERO_START : (int)DEV_NONFINITE;
      a.beta[0] = 0.0;
      *a.stop = 3;  // no eigenpair
      *a.steps = 0;
    } else {
      *a.stop = s.stop;
      *a.steps = m;
      if (a.tri && s.me == m) {  // the eigenpair that stopped the run
        a.tri->m_checked = m;
        a.tri->e_checked = s.e;
      }
    }
    *a.norm = a.beta[0];
    if (a.zero_beta0) a.beta[0] = 0.0;
  }
  cg::this_cluster().sync();  // no CTA leaves while another may still read its shared memory
}

static ResLayout run_layout(const ed_plan_s* p) {
  return res_layout(p->num_up, p->num_dn, p->bfp.quads, RUN_NT, RUN_CS, (size_t)p->ctx->smem_optin - RUN_STATIC);
}

// the device can hold such a cluster (asked once per device; also sets the kernel's attributes)
static bool cluster_ok(const ed_plan_s* p) {
  static std::atomic<uint64_t> yes{0}, asked{0};
  const uint64_t bit = 1ull << (p->ctx->device & 63);
  if (asked.load() & bit) return yes.load() & bit;
  cudaFuncAttributes fa;
  int n = 0;
  if (cudaFuncGetAttributes(&fa, k_res_run) == cudaSuccess && fa.sharedSizeBytes <= RUN_STATIC &&
      cudaFuncSetAttribute(k_res_run, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           p->ctx->smem_optin - (int)RUN_STATIC) == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(RUN_CS);
    cfg.blockDim = dim3(RUN_NT);
    cfg.dynamicSmemBytes = (size_t)p->ctx->smem_optin - RUN_STATIC;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = RUN_CS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, k_res_run, &cfg) != cudaSuccess) n = 0;
  }
  (void)cudaGetLastError();
  if (n >= 1) yes.fetch_or(bit);
  asked.fetch_or(bit);
  return n >= 1;
}

// (a matvec kernel or a wait limit asked for by name is a request for the launched steps)
bool resident_fits(const ed_plan_s* p) {
  return p->bfp.eligible && forced_variant(p) <= 0 && p->bfp.wait_limit == 0 && run_layout(p).ws && cluster_ok(p);
}

ed_status resident_run(const ed_plan_s* p, int K, double tol, int check_every, const double* start, double* alpha,
                       double* beta, double* norm, int zero_beta0, int32_t* exps, int64_t* store, double* c,
                       double* work, int* stop, int* steps, int* status, TriResult* tri, cudaStream_t s) {
  BatchProblem prob;
  describe_problem(p, &prob);
  const ResLayout L = run_layout(p);
  ResSingle a{start, K, tol, check_every, alpha, beta, c, work, norm, zero_beta0, exps, store, stop, steps, status, tri};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(RUN_CS);
  cfg.blockDim = dim3(RUN_NT);
  cfg.dynamicSmemBytes = L.total;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = RUN_CS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_res_run, prob, L, a);
  if (e != cudaSuccess) return cuda_fail(e, "k_res_run");
  ED_CHECK_LAUNCH("k_res_run");
  return ED_OK;
}

}  // namespace ed
