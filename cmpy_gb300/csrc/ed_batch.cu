// Batched Lanczos (the kernel: ed_batch.cuh, ed_resident.cuh): batch handles, the choice of the launch
// configuration, and the batched continued fraction.
#include "ed_batch.cuh"
#include "ed_cf.cuh"

namespace ed {

// G_p(z) += sign * norm_p^2 / (z' - a0 - b1^2 / (z' - a1 - ...)),  z' = sign*z + e0_p,
// norm_p = beta[p][0] (start norm), m_p = steps[p]; one thread per frequency, one problem per
// blockIdx.y. Bound by the FP64 pipe: 512 problems x 1280 frequencies x 2000 levels 32.9 -> 26.4 ms.
constexpr int BCF_NT = 128;
__global__ void __launch_bounds__(BCF_NT) k_batch_cf(int n, int K, const double* __restrict__ alpha,
                                                     const double* __restrict__ beta, const int32_t* __restrict__ steps,
                                                     const double* __restrict__ e0, int sign,
                                                     const double2* __restrict__ z, int64_t nz, double2* __restrict__ g) {
  __shared__ double2 st[CF_TILE];
  const int64_t j = blockIdx.x * (int64_t)BCF_NT + threadIdx.x;
  const double2 zi = j < nz ? z[j] : make_double2(0.0, 1.0);
  for (int p = blockIdx.y; p < n; p += gridDim.y) {
    const int m = steps[p];
    if (m < 1) continue;
    const double* b = beta + (int64_t)p * (K + 1);
    const double2 r = cf_value(alpha + (int64_t)p * K, b, m, sign * zi.x + e0[p], sign * zi.y, sign * b[0] * b[0], st);
    if (j < nz) {
      double2& o = g[(int64_t)p * nz + j];
      o = make_double2(o.x + r.x, o.y + r.y);
    }
  }
}

}  // namespace ed

// ---- host side ---------------------------------------------------------------------------------

namespace ed {

// the grid: clusters of cs CTAs, at most one cluster per problem and per_sm CTAs per SM
static int batch_grid(const ed_batch_s* b, int per_sm, int cs) {
  const int clusters = std::max(1, std::min(b->n, b->ctx->num_sms * per_sm / cs));
  return clusters * cs;
}

struct BatchLayout {
  size_t off_queue, off_slots, off_tri, off_exps, off_coefs, total;
};

static size_t al256b(size_t x) { return (x + 255) & ~(size_t)255; }

// vector slots per cluster; tridiagonal work, eigenvector, alpha/beta copies, exponents and
// Ritz coefficients per CTA
static BatchLayout batch_layout(const ed_batch_s* b, int K, int grid, int cs) {
  BatchLayout L;
  size_t o = 0;
  L.off_queue = o; o = al256b(o + 256);
  L.off_slots = o; o = al256b(o + (size_t)(grid / cs) * 5 * b->dmax * 8);
  L.off_tri = o; o = al256b(o + (size_t)grid * 8 * (K + 2) * 8);
  L.off_exps = o; o = al256b(o + (size_t)grid * (K + 2) * 4);
  L.off_coefs = o; o = al256b(o + (size_t)grid * (K + 2) * 8);
  L.total = o;
  return L;
}

static bool valid_config(int threads, int per_sm, int cs) {
  const bool t_ok = threads == 128 || threads == 256 || threads == 512 || threads == 1024;
  const bool c_ok = cs == 1 || ((cs == 2 || cs == 4 || cs == 8) && threads >= 512);
  return t_ok && c_ok && per_sm >= 1 && per_sm <= 16;
}

// threads of the kernel that a request for `threads` takes: with one CTA per problem whole columns of the sums
// (RES_COLS) and a warp for the scalars
static int kernel_threads(int threads, int cs) {
  return cs > 1 ? threads : (threads <= 256 ? 288 : (threads == 512 ? 544 : 800));
}

static ed_status run_batch(const ed_batch_s* b, int threads, int per_sm, int cs, int K, double tol, int check_every,
                           uint64_t seed, const double* const* starts, int want_vector, void* work, size_t bytes,
                           const BatchOut& out, cudaStream_t s) {
  if (!valid_config(threads, per_sm, cs))
    return fail(ED_ERR_INVALID_ARG, "threads 128/256/512/1024; clusters of 2, 4 or 8 CTAs need 512 or 1024 threads");
  const int grid = batch_grid(b, per_sm, cs);
  const BatchLayout L = batch_layout(b, K, grid, cs);
  if (!work || bytes < L.total) return fail(ED_ERR_INVALID_ARG, "batch workspace too small (see ed_batch_workspace)");
  char* base = (char*)work;
  BatchWork wk;
  wk.queue = (int*)(base + L.off_queue);
  wk.slots = (int64_t*)(base + L.off_slots);
  wk.dmax = b->dmax;
  wk.tri = (double*)(base + L.off_tri);
  wk.exps = (int32_t*)(base + L.off_exps);
  wk.coefs = (int64_t*)(base + L.off_coefs);
  ED_CUDA(cudaMemsetAsync(wk.queue, 0, sizeof(int), s));
#define ED_BATCH_CASE(NT, CS) \
  if (threads == NT && cs == CS) return launch_batch<NT, CS>(b, grid, per_sm, K, tol, check_every, seed, starts, want_vector, out, wk, s);
  if (cs == 1) {
    const int nt = kernel_threads(threads, 1);
    if (nt == 288) return launch_batch<288, 1>(b, grid, per_sm, K, tol, check_every, seed, starts, want_vector, out, wk, s);
    if (nt == 544) return launch_batch<544, 1>(b, grid, per_sm, K, tol, check_every, seed, starts, want_vector, out, wk, s);
    return launch_batch<800, 1>(b, grid, per_sm, K, tol, check_every, seed, starts, want_vector, out, wk, s);
  }
  ED_BATCH_CASE(512, 2)
  ED_BATCH_CASE(512, 4)
  ED_BATCH_CASE(512, 8)
  ED_BATCH_CASE(1024, 2)
  ED_BATCH_CASE(1024, 4)
  ED_BATCH_CASE(1024, 8)
#undef ED_BATCH_CASE
  return fail(ED_ERR_INVALID_ARG, "unsupported launch configuration");
}

static int cluster_schedulable(int threads, int cs) {
  if (threads == 512 && cs == 2) return clusters_for<512, 2>();
  if (threads == 512 && cs == 4) return clusters_for<512, 4>();
  if (threads == 512 && cs == 8) return clusters_for<512, 8>();
  if (threads == 1024 && cs == 2) return clusters_for<1024, 2>();
  if (threads == 1024 && cs == 4) return clusters_for<1024, 4>();
  if (threads == 1024 && cs == 8) return clusters_for<1024, 8>();
  return 0;
}

static void default_config(const ed_batch_s* b, int* threads, int* per_sm, int* cs) {
  if (b->tuned_threads) {
    *threads = b->tuned_threads;
    *per_sm = b->tuned_per_sm;
    *cs = b->tuned_cluster;
    return;
  }
  *threads = 512;
  *per_sm = 2;
  *cs = 1;
}

}  // namespace ed

using namespace ed;

extern "C" {

ED_API ed_status ed_batch_create(const ed_plan* plans, int n, ed_batch* out) {
  if (!out) return fail(ED_ERR_INVALID_ARG, "null output");
  *out = nullptr;
  if (n < 1 || !plans) return fail(ED_ERR_INVALID_ARG, "need at least one plan");
  ed_batch_s* b = new ed_batch_s();
  ED_CUDA(cudaGetDevice(&b->device));
  ed_status st = device_context(&b->ctx);
  if (st != ED_OK) { delete b; return st; }
  std::vector<BatchProblem> hp(n);
  for (int i = 0; i < n; ++i) {
    const ed_plan_s* p = plans[i];
    if (!p || p->device != b->device) { delete b; return fail(ED_ERR_INVALID_ARG, "plans must be on the current device"); }
    if (p->kind != 0 || !p->bfp.eligible) {
      delete b;
      return fail(ED_ERR_INVALID_ARG, "batched Lanczos needs fixed-point sectors (ed_plan_fixed_point > 0)");
    }
    describe_problem(p, &hp[i]);
    ed_batch_s::Shape sh{p->num_up, p->num_dn, {}};
    memcpy(sh.quads, p->bfp.quads, sizeof(sh.quads));
    bool seen = false;
    for (const auto& q : b->shapes)
      seen |= q.nu == sh.nu && q.nd == sh.nd && memcmp(q.quads, sh.quads, sizeof(sh.quads)) == 0;
    if (!seen) b->shapes.push_back(sh);
    b->dims.push_back(p->dim);
    b->dmax = std::max(b->dmax, p->dim);
  }
  b->n = n;
  // largest problems first (longest-processing-time order for the work queue)
  std::vector<int> order(n);
  for (int i = 0; i < n; ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int a, int c) { return b->dims[a] > b->dims[c]; });
  cudaError_t e = cudaMalloc(&b->d_probs, n * sizeof(BatchProblem));
  if (e == cudaSuccess) e = cudaMemcpy(b->d_probs, hp.data(), n * sizeof(BatchProblem), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMalloc(&b->d_order, n * sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpy(b->d_order, order.data(), n * sizeof(int), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(b->d_probs);
    cudaFree(b->d_order);
    delete b;
    return cuda_fail(e, "ed_batch_create");
  }
  b->n = n;
  *out = b;
  return ED_OK;
}

ED_API ed_status ed_batch_destroy(ed_batch b) {
  if (!b) return ED_OK;
  cudaFree(b->d_probs);
  cudaFree(b->d_order);
  delete b;
  return ED_OK;
}

ED_API int ed_batch_resident(ed_batch b, int threads, int ctas_per_sm, int cluster_size) {
  if (!b || !valid_config(threads, ctas_per_sm, cluster_size)) return 0;
  const int nt = kernel_threads(threads, cluster_size);
  const size_t budget = batch_smem(b, nt, cluster_size, ctas_per_sm);
  for (const auto& q : b->shapes)
    if (!res_layout(q.nu, q.nd, q.quads, nt, cluster_size, budget).ws) return 0;
  return 1;
}

ED_API ed_status ed_batch_workspace(ed_batch b, int max_steps, int threads, int ctas_per_sm, int cluster_size,
                                    size_t* bytes) {
  if (!b || !bytes) return fail(ED_ERR_INVALID_ARG, "null argument");
  if (max_steps < 1 || max_steps > 4096) return fail(ED_ERR_INVALID_ARG, "max_steps must be in [1, 4096]");
  int t = threads, ps = ctas_per_sm, cs = cluster_size;
  if (t <= 0 || ps <= 0) default_config(b, &t, &ps, &cs);
  if (cs <= 0) cs = 1;
  if (!valid_config(t, ps, cs)) return fail(ED_ERR_INVALID_ARG, "unsupported launch configuration");
  *bytes = batch_layout(b, max_steps, batch_grid(b, ps, cs), cs).total;
  return ED_OK;
}

ED_API ed_status ed_batch_lanczos(ed_batch b, int max_steps, double tol, int check_every, uint64_t seed,
                                  const double* const* d_starts, int want_vector, void* d_work, size_t work_bytes,
                                  double* d_alpha, double* d_beta, double* d_energy, double* d_residual,
                                  int32_t* d_steps, double* d_vecs, const int64_t* d_vec_offsets, int threads,
                                  int ctas_per_sm, int cluster_size, ed_stream_t stream) {
  if (!b) return fail(ED_ERR_INVALID_ARG, "null batch");
  if (max_steps < 1 || max_steps > 4096) return fail(ED_ERR_INVALID_ARG, "max_steps must be in [1, 4096]");
  if (!d_alpha || !d_beta || !d_energy || !d_residual || !d_steps)
    return fail(ED_ERR_INVALID_ARG, "null output array");
  if (want_vector && (!d_vecs || !d_vec_offsets)) return fail(ED_ERR_INVALID_ARG, "want_vector needs vectors");
  int dev = -1;
  ED_CUDA(cudaGetDevice(&dev));
  if (dev != b->device) return fail(ED_ERR_INVALID_ARG, "batch belongs to another device");
  int t = threads, ps = ctas_per_sm, cs = cluster_size;
  if (t <= 0 || ps <= 0) default_config(b, &t, &ps, &cs);
  if (cs <= 0) cs = 1;
  BatchOut out{d_alpha, d_beta, d_energy, d_residual, d_steps, d_vecs, d_vec_offsets};
  return run_batch(b, t, ps, cs, max_steps, tol, check_every, seed, d_starts, want_vector, d_work, work_bytes, out,
                   as_stream(stream));
}

ED_API ed_status ed_batch_lanczos_coeffs(ed_batch b, int max_steps, uint64_t seed, const double* const* d_starts,
                                         void* d_work, size_t work_bytes, double* d_alpha, double* d_beta,
                                         int32_t* d_steps, int threads, int ctas_per_sm, int cluster_size,
                                         ed_stream_t stream) {
  if (!b) return fail(ED_ERR_INVALID_ARG, "null batch");
  if (max_steps < 1 || max_steps > 4096) return fail(ED_ERR_INVALID_ARG, "max_steps must be in [1, 4096]");
  if (!d_alpha || !d_beta || !d_steps) return fail(ED_ERR_INVALID_ARG, "null output array");
  int dev = -1;
  ED_CUDA(cudaGetDevice(&dev));
  if (dev != b->device) return fail(ED_ERR_INVALID_ARG, "batch belongs to another device");
  int t = threads, ps = ctas_per_sm, cs = cluster_size;
  if (t <= 0 || ps <= 0) default_config(b, &t, &ps, &cs);
  if (cs <= 0) cs = 1;
  BatchOut out{d_alpha, d_beta, nullptr, nullptr, d_steps, nullptr, nullptr};
  return run_batch(b, t, ps, cs, max_steps, 0.0, 0, seed, d_starts, 0, d_work, work_bytes, out, as_stream(stream));
}

// Autotuner: times the candidate (threads, CTAs per SM, cluster size) configurations on a short
// run (tune_steps Lanczos steps, no vector) and keeps the fastest for this batch. Cluster
// candidates the device cannot schedule (no active cluster) are skipped.
ED_API ed_status ed_batch_tune(ed_batch b, int tune_steps, void* d_work, size_t work_bytes, double* d_alpha,
                               double* d_beta, double* d_energy, double* d_residual, int32_t* d_steps,
                               int* h_threads, int* h_ctas_per_sm, int* h_cluster_size, float* h_ms,
                               ed_stream_t stream) {
  if (!b) return fail(ED_ERR_INVALID_ARG, "null batch");
  cudaStream_t s = as_stream(stream);
  const int cand[][3] = {{256, 2, 1}, {256, 3, 1},  {256, 4, 1},  {512, 1, 1},  {512, 2, 1},  {1024, 1, 1},
                         {512, 2, 2}, {1024, 1, 2}, {512, 2, 4},  {1024, 1, 4}, {512, 2, 8},  {1024, 1, 8}};
  float best = 1e30f;
  int bt = 0, bp = 0, bc = 0;
  cudaEvent_t e0, e1;
  ED_CUDA(cudaEventCreate(&e0));
  ED_CUDA(cudaEventCreate(&e1));
  (void)d_energy;
  (void)d_residual;
  BatchOut out{d_alpha, d_beta, nullptr, nullptr, d_steps, nullptr, nullptr};
  for (auto& c : cand) {
    const int grid = batch_grid(b, c[1], c[2]);
    const size_t need = batch_layout(b, tune_steps, grid, c[2]).total;
    if (need > work_bytes) continue;
    if (c[2] > 1 && cluster_schedulable(c[0], c[2]) < 1) continue;
    // warm once, then time
    ED_TRY(run_batch(b, c[0], c[1], c[2], tune_steps, 0.0, 0, 1, nullptr, 0, d_work, work_bytes, out, s));
    ED_CUDA(cudaEventRecord(e0, s));
    ED_TRY(run_batch(b, c[0], c[1], c[2], tune_steps, 0.0, 0, 1, nullptr, 0, d_work, work_bytes, out, s));
    ED_CUDA(cudaEventRecord(e1, s));
    ED_CUDA(cudaEventSynchronize(e1));
    float ms = 0.f;
    ED_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    if (ms < best) { best = ms; bt = c[0]; bp = c[1]; bc = c[2]; }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (!bt) return fail(ED_ERR_INVALID_ARG, "workspace too small for every tuning candidate");
  b->tuned_threads = bt;
  b->tuned_per_sm = bp;
  b->tuned_cluster = bc;
  if (h_threads) *h_threads = bt;
  if (h_ctas_per_sm) *h_ctas_per_sm = bp;
  if (h_cluster_size) *h_cluster_size = bc;
  if (h_ms) *h_ms = best;
  return ED_OK;
}

ED_API ed_status ed_batch_gf_continued_fraction(int n, int max_steps, const double* d_alpha, const double* d_beta,
                                                const int32_t* d_steps, const double* d_e0, int sign,
                                                const double* d_z, int64_t n_z, double* d_g, ed_stream_t stream) {
  if (n < 1 || n_z < 0) return fail(ED_ERR_INVALID_ARG, "bad sizes");
  if (sign != 1 && sign != -1) return fail(ED_ERR_INVALID_ARG, "sign must be +1 or -1");
  if (n_z == 0) return ED_OK;
  if (!d_alpha || !d_beta || !d_steps || !d_e0 || !d_z || !d_g) return fail(ED_ERR_INVALID_ARG, "null argument");
  const dim3 grid((unsigned)((n_z + BCF_NT - 1) / BCF_NT), (unsigned)std::min(n, 65535));
  k_batch_cf<<<grid, BCF_NT, 0, as_stream(stream)>>>(n, max_steps, d_alpha, d_beta, d_steps, d_e0, sign,
                                                     (const double2*)d_z, n_z, (double2*)d_g);
  ED_CHECK_LAUNCH("k_batch_cf");
  return ED_OK;
}

}  // extern "C"
