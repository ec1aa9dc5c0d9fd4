// Batched Lanczos: many independent sectors (all (n_up, n_dn) sectors of a model, or many
// disorder realisations) in ONE persistent launch. No reference counterpart — the reference
// loops over sectors on the host (cmpy/exactdiag.py:24-43, one ARPACK solve each).
//
// Each CTA pulls problems from a device work queue (largest dimension first) and runs the
// whole fixed-point Lanczos of that problem with block-level synchronisation only (scalars in
// shared memory, vectors in the CTA's own workspace slot); CTAs never wait on each other, so
// there is no grid-wide barrier. With want_vector the CTA replays the recurrence once — the
// integer arithmetic and the fixed-order reductions make the replay bit-identical — and
// accumulates the ground-state vector in 128-bit fixed point. The launch is asynchronous and
// allocation-free, so host sequences of batched launches can be captured in a CUDA graph.
//
// Vector arithmetic is the block-fixed-point scheme of ed_bfp.cu (int64 mantissas, one
// exponent per vector, exact integer matvec, 128-bit dot products).
//
// With a thread-block cluster of CS > 1 CTAs per problem, the cluster's CTAs split the
// elements of every vector loop (CTA rank r takes the r-th stripe of the CS * (NT - 32) that own
// elements) and exchange their block totals through distributed shared memory at the hardware cluster
// barrier; every CTA then holds the same totals and computes the same scalars, an invariant subspace
// among them. The convergence tests are CTA 0's alone: the others wait for it at a cluster barrier and
// take its stop flag. So all CTAs of a cluster take the same branches and reach the same barriers. The
// largest sectors, which bound the makespan of the work queue, thus run on CS SMs.
//
// This header holds the kernel and its launch; ed_batch_one.cu and ed_batch_c{2,4,8}.cu instantiate them (one
// translation unit each, compiled in parallel), ed_batch.cu has the entry points.
#pragma once

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <vector>

#include "ed_plan.cuh"
#include "ed_resident.cuh"

namespace ed {
struct BatchOut {
  double* alpha;     // [n][K]
  double* beta;      // [n][K+1]; beta[p][0] = start norm, beta[p][k>0] couplings
  double* energy;    // [n]
  double* residual;  // [n]
  int32_t* steps;    // [n]
  double* vec;       // optional ground-state vectors: problem p at vec + vec_off[p]
  const int64_t* vec_off;
};

struct BatchWork {
  int64_t* slots;     // per CTA: Ra, Rb, W, acc_lo, acc_hi (each dmax)
  int64_t dmax;
  double* tri;        // per CTA: 8*(K+2) doubles (tridiagonal work 5, eigenvector, alpha, beta)
  int32_t* exps;      // per CTA: K+2 exponents of R_k
  int64_t* coefs;     // per CTA: K+2 Ritz coefficients
  int* queue;
};

}  // namespace ed

struct ed_batch_s {
  int device = -1;
  int n = 0;
  int64_t dmax = 0;
  ed::BatchProblem* d_probs = nullptr;
  int* d_order = nullptr;
  std::vector<int64_t> dims;
  struct Shape {
    int64_t nu, nd;
    int quads[4];
  };
  std::vector<Shape> shapes;  // the distinct ones
  ed::DeviceContext* ctx = nullptr;
  int tuned_threads = 0;
  int tuned_per_sm = 0;
  int tuned_cluster = 0;
};

namespace ed {

template <int NT, int CS>
ed_status launch_batch(const ed_batch_s* b, int grid, int per_sm, int K, double tol, int check_every, uint64_t seed,
                       const double* const* starts, int want_vector, const BatchOut& out, const BatchWork& wk,
                       cudaStream_t s);
// Dynamic shared memory of a CTA when per_sm of them share an SM: as much as that leaves, but no more
// than the batch's largest need (a problem that does not fit keeps R or all its vectors in its
// global slots).
constexpr size_t RES_STATIC = 5 * 1024;  // bound of the kernel's static shared memory
static inline size_t batch_smem(const ed_batch_s* b, int NT, int CS, int per_sm) {
  const size_t sm = (size_t)b->ctx->smem_optin + 1024;  // one CTA's limit plus the system's share
  const size_t per = sm / per_sm;
  if (per <= RES_STATIC + 1024) return 0;
  const size_t budget = (per - RES_STATIC - 1024) / 1024 * 1024;
  size_t need = 0;
  for (const auto& q : b->shapes) need = std::max(need, res_layout(q.nu, q.nd, q.quads, NT, CS, budget).total);
  return need;
}

// how many clusters of cs CTAs of the NT-thread kernel the device can hold at once (0: none)
template <int NT, int CS>
int clusters_for();

}  // namespace ed
