// One fixed-point Lanczos recurrence per CTA (or per thread-block cluster), run from start to end
// without leaving the kernel: the batched launches of ed_batch.cu and the runs of small sectors.
//
// Vector arithmetic is the block-fixed-point scheme of ed_bfp.cu (int64 mantissas, one exponent per
// vector, exact integer matvec). Layout: the vector R_k that the matvec gathers from is updated in
// place; W = H R_k and R_{k-1} are only touched by the thread that owns the element. R_k lives in shared
// memory when it fits (in a cluster every CTA holds a copy of it, and an element's owner writes the
// new value to all of them), and so do the thread-owned vectors; the hop lists, states and energies
// of the sector are always in shared memory when they fit.
//
// What bounds a step: its instruction stream for the larger sectors, and for the small ones the chain
// of scalars between its two phases. A warp's FP64 instruction holds the pipe for 64 cycles on
// this GPU, dependent or not, and the four sub-partitions share one of 19 cycles a warp (measured),
// so FP64 operations are counted one by one here: the last warp of the CTA owns no elements and
// forms the step's scalars, the norm of R_{k+1} while the other warps already run the next matvec; the
// dot products are 128-bit integers per thread.
//
// Sums. One CTA: the elements go to 256 columns (i mod 256) whose exact sums are rounded to FP64 and
// added in one fixed order, whatever the number of threads, so every configuration gives the same
// bits. A cluster: the exact total (a warp adds the 128-bit values as 26-bit limbs with the integer
// reduction instruction), converted to FP64 from its high and low words, each rounded, and their sum.
#pragma once

#include <cooperative_groups.h>

#include "ed_plan.cuh"
#include "ed_tridiag.cuh"

namespace ed {

namespace cg = cooperative_groups;

namespace {

struct I128 {
  uint64_t lo;
  int64_t hi;
};
// unsigned 64 x 64 -> 128 bits from four 32 x 32 + 64 -> 64 multiply-adds
__device__ __forceinline__ I128 mul_u64(uint64_t a, uint64_t b) {
  const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32), bl = (uint32_t)b, bh = (uint32_t)(b >> 32);
  const uint64_t p = (uint64_t)al * bl;
  const uint64_t q = (uint64_t)ah * bl + (p >> 32);
  const uint64_t r = (uint64_t)al * bh + (uint32_t)q;
  I128 v;
  v.lo = (r << 32) | (uint32_t)p;
  v.hi = (int64_t)((uint64_t)ah * bh + (q >> 32) + (r >> 32));
  return v;
}
__device__ __forceinline__ I128 mul_s64(int64_t a, int64_t b) {
  I128 v = mul_u64((uint64_t)a, (uint64_t)b);
  v.hi -= ((a >> 63) & b) + ((b >> 63) & a);
  return v;
}
__device__ __forceinline__ void add128(I128& acc, const I128& v) {
  asm("add.cc.u64 %0, %0, %2;\n\taddc.u64 %1, %1, %3;" : "+l"(acc.lo), "+l"(acc.hi) : "l"(v.lo), "l"(v.hi));
}
__device__ __forceinline__ double i128_to_double(const I128& v) { return fma((double)v.hi, 0x1.0p64, (double)v.lo); }
__device__ __forceinline__ int64_t shr128_round(I128 v, int s) {
  I128 h;
  h.lo = 1ull << (s - 1);
  h.hi = 0;
  add128(v, h);
  return (int64_t)((v.lo >> s) | ((uint64_t)v.hi << (64 - s)));
}
__device__ __forceinline__ unsigned long long uabs64(int64_t v) {
  return v < 0 ? (unsigned long long)(-v) : (unsigned long long)v;
}
// x^2 as 128 bits for |x| < 2^63: the unsigned square needs no sign corrections
__device__ __forceinline__ I128 sqr_s64(int64_t x) {
  const uint64_t u = uabs64(x);
  const uint32_t l = (uint32_t)u, h = (uint32_t)(u >> 32);
  const uint64_t p = (uint64_t)l * l, q = (uint64_t)l * h;
  const uint64_t t = q + q + (p >> 32);  // q < 2^63: no overflow of 2 q beyond 64 bits
  I128 v;
  v.lo = (t << 32) | (uint32_t)p;
  v.hi = (int64_t)((uint64_t)h * h + (t >> 32));
  return v;
}
__device__ __forceinline__ uint64_t bsplitmix(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}
// A sum of many 128-bit values: lo + 2^64 (hi + 2^40 top). (The products of a long flat vector can
// add up to more than 127 bits.)
struct Wide {
  uint64_t lo, hi;
  int top;
};
// sum over the warp (all lanes get it): four 26-bit limbs and the rest, each by one integer reduction
__device__ __forceinline__ Wide warp_sum_wide(uint64_t lo, uint64_t hi, int rest) {
  const unsigned F = 0xffffffffu, M = (1u << 26) - 1u;
  const unsigned s0 = __reduce_add_sync(F, (unsigned)lo & M);
  const unsigned s1 = __reduce_add_sync(F, (unsigned)(lo >> 26) & M);
  const unsigned s2 = __reduce_add_sync(F, (unsigned)((lo >> 52) | (hi << 12)) & M);
  const unsigned s3 = __reduce_add_sync(F, (unsigned)(hi >> 14) & M);
  Wide w;
  w.top = __reduce_add_sync(F, rest);
  w.lo = (uint64_t)s0 + ((uint64_t)s1 << 26);
  const uint64_t add = (uint64_t)s2 << 52;
  w.lo += add;
  w.hi = ((uint64_t)s3 << 14) + (uint64_t)(s2 >> 12) + (w.lo < add ? 1u : 0u);
  return w;
}
__device__ __forceinline__ Wide warp_sum_wide(const I128& v) {
  return warp_sum_wide(v.lo, (uint64_t)v.hi, (int)(v.hi >> 40));
}
__device__ __forceinline__ Wide warp_sum_wide(const Wide& v) {
  return warp_sum_wide(v.lo, v.hi, v.top + (int)(v.hi >> 40));
}
// (the magnitude is converted: no cancellation between the words)
__device__ __forceinline__ double wide_to_double(const Wide& v) {
  const int64_t t = (int64_t)v.top + (int64_t)(v.hi >> 40);
  const uint64_t h = v.hi & ((1ull << 40) - 1);
  if (t >= ((int64_t)1 << 22) || t < -((int64_t)1 << 22))  // beyond 127 bits
    return fma((double)t, 0x1.0p104, fma((double)h, 0x1.0p64, (double)v.lo));
  I128 x{v.lo, (int64_t)(((uint64_t)t << 40) + h)};
  const bool neg = x.hi < 0;
  if (neg) {
    x.lo = ~x.lo + 1;
    x.hi = ~x.hi + (x.lo == 0 ? 1 : 0);
  }
  const double d = i128_to_double(x);
  return neg ? -d : d;
}
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
  const unsigned F = 0xffffffffu, h = (unsigned)(v >> 32), mh = __reduce_max_sync(F, h);
  const unsigned ml = __reduce_max_sync(F, h == mh ? (unsigned)v : 0u);
  return ((unsigned long long)mh << 32) | ml;
}
// x * 2^n, and the exponent e of x = f 2^e, 0.5 <= f < 1, on the bits (x finite; x != 0 for exp2_of)
__device__ __forceinline__ double scale2(double x, int n) {
  const int hi = __double2hiint(x), e = ((hi >> 20) & 0x7ff), ne = e + n;
  if (e == 0 || ne < 1 || ne > 2046) return ldexp(x, n);
  return __hiloint2double(hi + (n << 20), __double2loint(x));
}
__device__ __forceinline__ int exp2_of(double x) {
  const int e = (__double2hiint(x) >> 20) & 0x7ff;
  if (e != 0) return e - 1022;
  int r = 0;
  frexp(x, &r);
  return r;
}

}  // namespace

// one problem = one fixed-point sector (device pointers owned by its plan)
struct BatchProblem {
  int64_t nu, nd, D;
  const int32_t* up_off;
  const int32_t* up_npos;
  const int32_t* up_idx;
  const uint16_t* dn_tab;
  const uint64_t* up_states;
  const uint64_t* dn_states;
  const int32_t* e_up;
  const int32_t* e_dn;
  const int64_t* e_up_fx;
  const int64_t* e_dn_fx;
  int max_up, max_dn, diag64, dshift, F, m_in, u_uniform;
  int quads[4];  // largest numbers of up +, up -, dn +, dn - partners of a state, in fours
  int32_t t_int, u0;
  int64_t u0_fx;
  int32_t u[ED_MAX_SITES + 2];
  int64_t u_fx[ED_MAX_SITES + 2];
};

static void describe_problem(const ed_plan_s* p, BatchProblem* q) {
  const BfpTables& B = p->bfp;
  memset(q, 0, sizeof(*q));
  q->nu = p->num_up; q->nd = p->num_dn; q->D = p->dim;
  q->up_off = B.up_off; q->up_npos = B.up_npos; q->up_idx = B.up_idx; q->dn_tab = B.dn_tab;
  q->up_states = p->up.states; q->dn_states = p->dn.states;
  q->e_up = B.e_up_int; q->e_dn = B.e_dn_int; q->e_up_fx = B.e_up_fx; q->e_dn_fx = B.e_dn_fx;
  q->max_up = B.max_up; q->max_dn = B.max_dn;
  for (int k = 0; k < 4; ++k) q->quads[k] = B.quads[k];
  q->diag64 = B.diag64; q->dshift = B.Fd - B.F; q->F = B.F; q->m_in = B.m_in;
  q->u_uniform = B.u_uniform; q->t_int = B.t_int; q->u0 = B.u0_int; q->u0_fx = B.u0_fx;
  for (int k = 0; k < ED_MAX_SITES + 2; ++k) { q->u[k] = B.u_int[k]; q->u_fx[k] = B.u_fx[k]; }
}

// Dynamic shared memory of a CTA: the sector's tables, R, then W and R_{k-1} of the CTA's own elements,
// as far as they fit. ts / rs / ws: tables / R / W and R_{k-1} in shared memory.
struct ResLayout {
  int ts, rs, ws;
  int up_quads, dn_quads;  // list words per state
  int own;                 // elements of a CTA (padded to whole rounds of its threads)
  size_t ex, vec, wvec, uplist, dnlist, uprec, dnrec, total;
};
__host__ __device__ inline ResLayout res_layout(int64_t nu, int64_t nd, const int (&quads)[4], int nt, int cs,
                                                size_t budget) {
  ResLayout L;
  auto al = [](size_t v) { return (v + 15) & ~(size_t)15; };
  L.up_quads = quads[0] + quads[1];
  L.dn_quads = quads[2] + quads[3];
  size_t o = 0;
  L.ex = o; o = al(o + (cs == 1 && nt > 288 ? (size_t)(nt - 288) * 16 : 0));
  L.uprec = o; o = al(o + (size_t)nu * 16);
  L.dnrec = o; o = al(o + (size_t)nd * 16);
  L.uplist = o; o = al(o + (size_t)nu * L.up_quads * 16);
  L.dnlist = o; o = al(o + (size_t)nd * L.dn_quads * 8);
  L.vec = o;
  const int64_t D = nu * nd, per = (int64_t)cs * (nt - 32);
  const size_t v8 = al((size_t)D * 8);
  L.ts = nd < 65536 && D < ((int64_t)1 << 31) && o <= budget;
  L.rs = L.ts && o + v8 <= budget;
  L.own = L.rs ? (int)((D + per - 1) / per) * (nt - 32) : 0;
  L.wvec = o + v8;
  const size_t w8 = al((size_t)L.own * 8);
  L.ws = L.rs && o + v8 + 2 * w8 <= budget;
  L.total = !L.ts ? L.uprec : (L.ws ? o + v8 + 2 * w8 : (L.rs ? o + v8 : o));
  return L;
}

// where a problem's data live: vectors and tables in global memory; tables in shared memory; R too
// (in RES_ALL also W and R_{k-1}). RES_GLOBAL reads the diagonal's mode from the problem, the others
// are compiled for it.
enum ResMode : int { RES_GLOBAL = 0, RES_TABLES = 1, RES_SHARED = 2, RES_ALL = 3 };

// byte offsets in the dynamic shared memory. Every state has the sector's largest numbers of + and of -
// partners, in fours, padded with itself: the loops over them have one length for the whole launch (no
// divergence), and the surplus t x of the padding is taken off the diagonal (integer diagonals: in
// the energies; fixed-point ones: by ResRec.pad).
struct ResTables {
  unsigned uplist;         // uint4 [nu][up_quads]: element offsets u' * nd
  unsigned dnlist;         // uint2 [dn_quads][nd]: partner columns, 16 bits each
  unsigned uprec, dnrec;   // ResRec per state
  unsigned r, rp, w;       // R, R_{k-1}, W
  unsigned ex;             // exchange buffer of res_put
};
struct __align__(16) ResRec {
  int32_t pad;     // padding: + entries minus - entries
  uint32_t state;
  int64_t e;       // on-site energy, integer or fixed point
};

// the sector's tables into shared memory (every thread of the CTA; a barrier follows)
static __device__ void res_tables(const BatchProblem& P, const ResLayout& L, unsigned char* sm) {
  uint32_t* uplist = (uint32_t*)(sm + L.uplist);
  uint16_t* dnlist = (uint16_t*)(sm + L.dnlist);
  const int nu = (int)P.nu, nd = (int)P.nd;
  for (int u = threadIdx.x; u < nu; u += blockDim.x) {
    const int o0 = P.up_off[u], np = P.up_npos[u], nm = P.up_off[u + 1] - o0 - np;
    uint32_t* l = uplist + (size_t)u * L.up_quads * 4;
    for (int e = 0; e < 4 * L.up_quads; ++e) {
      const int m = e - 4 * P.quads[0];
      const int j = m < 0 ? (e < np ? e : -1) : (m < nm ? np + m : -1);
      l[e] = (uint32_t)(j >= 0 ? P.up_idx[o0 + j] : u) * (uint32_t)nd;
    }
    const int pad = (4 * P.quads[0] - np) - (4 * P.quads[1] - nm);
    ((ResRec*)(sm + L.uprec))[u] =
        ResRec{pad, (uint32_t)P.up_states[u], P.diag64 ? P.e_up_fx[u] : (int64_t)P.e_up[u] - (int64_t)pad * P.t_int};
  }
  for (int d = threadIdx.x; d < nd; d += blockDim.x) {
    for (int q = 0; q < 4 * L.dn_quads; ++q) dnlist[4 * ((q >> 2) * nd + d) + (q & 3)] = (uint16_t)d;
    int np = 0, nm = 0;
    for (int e = 0; e < P.max_dn; ++e) {
      const int sl = P.dn_tab[(int64_t)e * nd + d];
      if (sl >= 2 * nd) continue;
      const int q = sl < nd ? np++ : 4 * P.quads[2] + nm++;
      dnlist[4 * ((q >> 2) * nd + d) + (q & 3)] = (uint16_t)(sl < nd ? sl : sl - nd);
    }
    const int pad = (4 * P.quads[2] - np) - (4 * P.quads[3] - nm);
    ((ResRec*)(sm + L.dnrec))[d] =
        ResRec{pad, (uint32_t)P.dn_states[d], P.diag64 ? P.e_dn_fx[d] : (int64_t)P.e_dn[d] - (int64_t)pad * P.t_int};
  }
}
static __device__ ResTables res_offsets(const ResLayout& L) {
  const unsigned w8 = (unsigned)(((size_t)L.own * 8 + 15) & ~(size_t)15), v = (unsigned)L.wvec;
  return ResTables{(unsigned)L.uplist, (unsigned)L.dnlist, (unsigned)L.uprec, (unsigned)L.dnrec, (unsigned)L.vec, v,
                   v + w8, (unsigned)L.ex};
}

static __device__ __forceinline__ double start_value(const double* start, int64_t i, uint64_t seed) {
  if (start) return start[i];
  return (double)(bsplitmix(seed * 0x100000001B3ull + (uint64_t)i) >> 11) * 0x1.0p-53 + 0x1.0p-54;
}

// shared state of one recurrence; index 0: the matvec's totals, 1: the norm's
struct ResShared {
  Wide part[2][32];                // the warps' totals
  unsigned long long pmax[2][32];
  Wide xch[2];                     // the CTA's totals, read by the cluster
  unsigned long long xmax[2];
  double xd;
  uint64_t A[3];                   // |update coefficients| of W, R_k, R_{k-1}
  int64_t sgn[3];                  // 0 or -1: their signs
  I128 cst;                        // the constant of the biased products, and half a unit for the rounding
  int SA, stop, m;
  double red[2][32];               // the warps' FP64 sums
  // the scalar warp's state between steps: the norms b_k and b_{k-1}, the scale of row k - 1 of T, the
  // exponents and largest mantissas of R_k and R_{k-1}
  double bk, bkm1, row;
  unsigned long long mk, mp;
  int ek, ep;
  double lo, hi;                   // bracket of the lowest eigenvalue (res_test)
  double e;                        // the last careful solution: lowest eigenvalue of T_me, its vector in c
  int me;
  int cnt[128];
};

// The elements of a CTA of NT threads belong to NT - 32 threads; RES_COLS of them (or all, in a cluster)
// are the columns of the sums.
constexpr int RES_COLS = 256;

// a warp's total into its slot (ex: exchange buffer of the threads beyond the columns)
template <int NT, int CS>
static __device__ __forceinline__ void res_put(ResShared& s, I128* ex, int ph, I128 v, unsigned long long mx) {
  const unsigned long long m = warp_max_u64(mx);
  const int w = threadIdx.x >> 5;
  if constexpr (CS > 1) {
    const Wide t = warp_sum_wide(v);
    if ((threadIdx.x & 31) == 0) s.part[ph][w] = t;
  } else {
    constexpr int NC = NT - 32;
    static_assert(NC % RES_COLS == 0, "whole columns");
    if constexpr (NC > RES_COLS) {
      if (threadIdx.x >= RES_COLS) ex[threadIdx.x - RES_COLS] = v;
      asm volatile("bar.sync 1, %0;" ::"n"(NC) : "memory");  // the element-owning warps
      if (threadIdx.x < RES_COLS)
#pragma unroll
        for (int q = 0; q < NC / RES_COLS - 1; ++q) add128(v, ex[threadIdx.x + q * RES_COLS]);
    }
    if (threadIdx.x < RES_COLS) {
      double d = i128_to_double(v);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      if ((threadIdx.x & 31) == 0) s.red[ph][w] = d;
    }
  }
  if ((threadIdx.x & 31) == 0) s.pmax[ph][w] = m;
}
// the CTA's total from the warps' slots (the scalar warp); in a cluster it goes to the exchange slot
template <int NT, int CS>
static __device__ __forceinline__ void res_get(ResShared& s, int ph, double* v, unsigned long long* mx) {
  const int lane = threadIdx.x & 31;
  const bool on = lane < NT / 32 - 1;
  *mx = warp_max_u64(on ? s.pmax[ph][lane] : 0ull);
  if constexpr (CS > 1) {
    const Wide t = warp_sum_wide(on ? s.part[ph][lane] : Wide{0, 0, 0});
    if (lane == 0) {
      s.xch[ph] = t;
      s.xmax[ph] = *mx;
    }
    *v = 0.0;
  } else {
    double r = s.red[ph][0];
#pragma unroll
    for (int i = 1; i < RES_COLS / 32; ++i) r += s.red[ph][i];
    *v = r;
  }
}
// the cluster's total (one warp, after a cluster barrier): lane q reads rank q's
template <int CS>
static __device__ __forceinline__ void res_collect(ResShared& s, int ph, double* v, unsigned long long* mx) {
  const int lane = threadIdx.x & 31;
  Wide t{0, 0, 0};
  unsigned long long m = 0;
  if (lane < CS) {
    const ResShared* r = cg::this_cluster().map_shared_rank(&s, lane);
    t = r->xch[ph];
    m = r->xmax[ph];
  }
  *v = wide_to_double(warp_sum_wide(t));
  *mx = warp_max_u64(m);
}
template <int CS>
static __device__ __forceinline__ void csync() {
  if constexpr (CS > 1) cg::this_cluster().sync();
  else __syncthreads();
}

// W = H R on this thread's elements (i = i0, i0 + st, ...); its exact <R, W> and max |W|
template <int NT, int MODE, bool DIAG64>
static __device__ __forceinline__ void res_matvec(const BatchProblem& P, const ResTables& T, const int64_t* Rg, int64_t* Wg,
                                                  int64_t i0, int64_t st, I128* dot_out,
                                                  unsigned long long* max_out) {
  extern __shared__ __align__(16) unsigned char res_sm[];
  I128 dot{0, 0};
  unsigned long long mx = 0;
  if constexpr (MODE != RES_GLOBAL) {
    // everything indexed from the shared array itself, so that the loads are shared loads; the
    // sector's constants in registers (a store to W could alias them where they are)
    const int64_t* R = MODE >= RES_SHARED ? (const int64_t*)(res_sm + T.r) : Rg;
    int64_t* W = MODE == RES_ALL ? (int64_t*)(res_sm + T.w) : Wg;
    const uint4* const uplist = (const uint4*)(res_sm + T.uplist);
    const uint2* const dnlist = (const uint2*)(res_sm + T.dnlist);
    const ResRec* const urec = (const ResRec*)(res_sm + T.uprec);
    const ResRec* const drec = (const ResRec*)(res_sm + T.dnrec);
    const int nd = (int)P.nd, D = (int)P.D, step = (int)st, dshift = P.dshift;
    const int uqp = P.quads[0], uq = uqp + P.quads[1], dqp = P.quads[2], dq = dqp + P.quads[3];
    const bool uni = P.u_uniform != 0;
    const int64_t u0 = DIAG64 ? P.u0_fx : (int64_t)P.u0, t_int = P.t_int;
    // (u, d) advance by the stride without a division
    const int us = step / nd, ds = step - us * nd;
    int u = (int)i0 / nd, d = (int)i0 - u * nd, l = threadIdx.x;
    for (int i = (int)i0; i < D; i += step, l += NT - 32) {
      const ResRec ru = urec[u], rd = drec[d];
      const uint4* ul = uplist + u * uq;
      const uint2* dl = dnlist + d;
      const int64_t* col = R + d;
      const int64_t* row = R + (i - d);
      const int64_t x = R[i];
      int64_t h = 0;
      int q = 0;
      for (; q < uqp; ++q) {
        const uint4 o = ul[q];
        h += (col[o.x] + col[o.y]) + (col[o.z] + col[o.w]);
      }
      for (; q < uq; ++q) {
        const uint4 o = ul[q];
        h -= (col[o.x] + col[o.y]) + (col[o.z] + col[o.w]);
      }
      q = 0;
      for (; q < dqp; ++q, dl += nd) {
        const uint2 o = *dl;
        h += (row[o.x & 0xffffu] + row[o.x >> 16]) + (row[o.y & 0xffffu] + row[o.y >> 16]);
      }
      for (; q < dq; ++q, dl += nd) {
        const uint2 o = *dl;
        h -= (row[o.x & 0xffffu] + row[o.x >> 16]) + (row[o.y & 0xffffu] + row[o.y >> 16]);
      }
      const uint32_t both = ru.state & rd.state;
      int64_t w;
      if (!DIAG64) {
        int32_t dg = (int32_t)ru.e + (int32_t)rd.e;
        if (uni) dg += (int32_t)u0 * __popc(both);
        else
          for (uint32_t b = both; b; b &= b - 1) dg += P.u[__ffs((int)b) - 1];
        w = t_int * h + (int64_t)dg * x;
      } else {
        h -= (int64_t)(ru.pad + rd.pad) * x;
        int64_t dg = ru.e + rd.e;
        if (uni) dg += u0 * (int64_t)__popc(both);
        else
          for (uint32_t b = both; b; b &= b - 1) dg += P.u_fx[__ffs((int)b) - 1];
        w = t_int * h + shr128_round(mul_s64(dg, x), dshift);
      }
      W[MODE == RES_ALL ? l : i] = w;
      add128(dot, mul_s64(x, w));
      mx = max(mx, uabs64(w));
      u += us;
      d += ds;
      if (d >= nd) {
        d -= nd;
        ++u;
      }
    }
  } else {
    const int64_t nd = P.nd;
    for (int64_t i = i0; i < P.D; i += st) {
      const int64_t u = i / nd, d = i - u * nd;
      const int64_t* xrow = Rg + u * nd;
      int64_t h = 0;
      const int32_t o0 = __ldg(P.up_off + u), o1 = __ldg(P.up_off + u + 1), op = o0 + __ldg(P.up_npos + u);
      for (int32_t e = o0; e < op; ++e) h += Rg[(int64_t)__ldg(P.up_idx + e) * nd + d];
      for (int32_t e = op; e < o1; ++e) h -= Rg[(int64_t)__ldg(P.up_idx + e) * nd + d];
      for (int e = 0; e < P.max_dn; ++e) {
        const int sl = __ldg(P.dn_tab + (int64_t)e * nd + d);
        if (sl < nd) h += xrow[sl];
        else if (sl < 2 * nd) h -= xrow[sl - nd];
      }
      const int64_t x = xrow[d];
      const uint64_t both = __ldg(P.up_states + u) & __ldg(P.dn_states + d);
      int64_t dterm;
      if (!P.diag64) {
        int32_t dg = __ldg(P.e_up + u) + __ldg(P.e_dn + d);
        if (P.u_uniform) dg += P.u0 * __popcll(both);
        else
          for (uint64_t b = both; b; b &= b - 1) dg += P.u[__ffsll((long long)b) - 1];
        dterm = (int64_t)dg * x;
      } else {
        int64_t dg = __ldg(P.e_up_fx + u) + __ldg(P.e_dn_fx + d);
        if (P.u_uniform) dg += P.u0_fx * (int64_t)__popcll(both);
        else
          for (uint64_t b = both; b; b &= b - 1) dg += P.u_fx[__ffsll((long long)b) - 1];
        dterm = shr128_round(mul_s64(dg, x), P.dshift);
      }
      const int64_t w = (int64_t)P.t_int * h + dterm;
      Wg[i] = w;
      add128(dot, mul_s64(x, w));
      mx = max(mx, uabs64(w));
    }
  }
  *dot_out = dot;
  *max_out = mx;
}

// The lowest eigenpair of T_m by the careful solver (the convergence's confirmation, the result)
static __device__ __noinline__ double res_tridiag(const double* al, const double* be, int m, double* c, double* work,
                                                  double lo, double hi) {
  return tridiag_lowest_block(al, be, m, c, work, lo, hi);
}

// Quick estimate of the residual |beta_m c_{m-1}| of T_m's lowest eigenvector, relative to max(1, |E|),
// for a convergence test: two rounds of 128 Sturm counts in the bracket that the previous test left
// (s.lo, s.hi: E can only have fallen, by less than the earlier residual says; lo >= hi: none yet, the
// Gershgorin interval), then the eigenvector's components upward from the last one, v_{i-1} =
// -((a_i - E) v_i + b_{i+1} v_{i+1}) / b_i, the direction in which they grow. Three FP64 operations a
// row and pass where the careful solver takes some hundred. Every thread of the CTA calls it; work:
// 5 m doubles.
static __device__ double res_test(const double* al, const double* be, int m, double* work, ResShared& s) {
  double* bb = work;          // b_i^2
  double* ra = work + m;      // -a_i / b_i, then -(a_i - E) / b_i
  double* rc = work + 2 * m;  // -b_{i+1} / b_i
  double glo = al[0], ghi = al[0];
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    bb[i] = be[i] * be[i];
    const double r = (i > 0 ? fabs(be[i]) : 0.0) + (i + 1 < m ? fabs(be[i + 1]) : 0.0);
    glo = fmin(glo, al[i] - r);
    ghi = fmax(ghi, al[i] + r);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    glo = fmin(glo, __shfl_xor_sync(0xffffffffu, glo, o));
    ghi = fmax(ghi, __shfl_xor_sync(0xffffffffu, ghi, o));
  }
  double* rl = (double*)&s.part[0][0];  // the totals' slots are free here
  if ((threadIdx.x & 31) == 0) {
    rl[threadIdx.x >> 5] = glo;
    s.red[0][threadIdx.x >> 5] = ghi;
  }
  __syncthreads();
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
    glo = fmin(glo, rl[w]);
    ghi = fmax(ghi, s.red[0][w]);
  }
  double lo = s.lo, hi = s.hi;
  if (!(lo < hi)) {
    lo = glo;
    hi = ghi;
  }
  for (int round = 0; round < 2; ++round) {
    const double h = (hi - lo) * (1.0 / 127.0);
    __syncthreads();
    if (threadIdx.x < 128) s.cnt[threadIdx.x] = sturm_count(al, be, bb, m, lo + h * threadIdx.x) > 0;
    __syncthreads();
    int t = 0;
    while (t < 128 && !s.cnt[t]) ++t;  // the first point with an eigenvalue below
    if (t == 0) {                      // the bracket's lower end was too high
      hi = lo;
      lo = glo;
    } else if (t == 128) {
      lo = hi;
      hi = ghi;
    } else {
      hi = lo + h * t;
      lo = lo + h * (t - 1);
    }
  }
  for (int i = threadIdx.x; i < m; i += blockDim.x)
    if (i > 0) {
      const double r = -1.0 / be[i];
      ra[i] = (al[i] - lo) * r;
      rc[i] = i + 1 < m ? be[i + 1] * r : 0.0;
    }
  __syncthreads();
  if (threadIdx.x == 0) {
    double v = 1.0, vn = 0.0, q = 1.0;
    for (int i = m - 1; i > 0; --i) {
      const double p = fma(ra[i], v, rc[i] * vn);
      vn = v;
      v = p;
      q = fma(v, v, q);
      if (((unsigned)__double2hiint(q) & 0x7fffffffu) > 0x70000000u) {  // q > 2^769: only the ratio matters
        v *= 0x1.0p-300;
        vn *= 0x1.0p-300;
        q *= 0x1.0p-600;
      }
    }
    const double sc = fmax(1.0, fabs(lo)), res = fabs(be[m]) / sqrt(q);
    // (rescaled: q lost the factor; the true residual is smaller still, which only matters below
    // any tolerance)
    s.xd = res / sc;
    s.lo = lo - fmax(16.0 * res, 1e-9 * sc);
    s.hi = hi;
  }
  __syncthreads();
  return s.xd;
}

// The Lanczos recurrence of one problem: R_{k+1} = W/b_k - (a_k/b_k) R_k - (b_k/b_{k-1}) R_{k-1}, the
// residuals r_k of norm b_k as mantissas R_k below 2^m_in with an exponent per step.
// Pass 1 (Ck == null) records alpha, beta and the exponents of the R_k (and every R_k in `store` when
// given) and stops on convergence / invariant subspace; pass 2 replays exactly `m_replay` steps (the
// same bits) and accumulates acc += Ck[k] * R_k. alpha / beta / exps are this CTA's copies (global
// memory). Every thread of the CTA calls it; returns m (0: zero or non-finite start vector, beta[0] = 0
// or NaN in pass 1).
struct ResRun {
  const double* start;
  uint64_t seed;
  int K;
  double tol;
  int check_every, rk;
  int64_t *R, *Rp, *W;  // global vectors, where they are not in shared memory
  double *alpha, *beta, *c, *work;
  int32_t* exps;
  int m_replay;
  const int64_t* Ck;
  uint64_t* acc_lo;
  int64_t* acc_hi;
  int64_t* store;       // [K][D] or null
};  // (alpha null: this CTA of a cluster records nothing)
template <int NT, int CS, int MODE, bool DIAG64>
static __device__ __noinline__ int res_recurrence(const BatchProblem& P, const ResTables T, const ResRun& io, ResShared& s) {
  extern __shared__ __align__(16) unsigned char res_sm[];
  int64_t* const R = MODE >= RES_SHARED ? (int64_t*)(res_sm + T.r) : io.R;
  int64_t* const Rp = MODE == RES_ALL ? (int64_t*)(res_sm + T.rp) : io.Rp;
  int64_t* const W = MODE == RES_ALL ? (int64_t*)(res_sm + T.w) : io.W;
  constexpr int NC = NT - 32;  // threads that own elements; the last warp does the scalars
  const bool pass2 = io.Ck != nullptr, rec = !pass2 && io.alpha != nullptr;
  const bool rk0 = CS == 1 || io.rk == 0;
  const int lane = threadIdx.x & 31;
  const bool scalar = (int)(threadIdx.x >> 5) == NT / 32 - 1;
  const int64_t D = P.D, i0 = scalar ? D : (int64_t)io.rk * NC + threadIdx.x, st = (int64_t)CS * NC;
  double* const alpha = io.alpha;
  double* const beta = io.beta;
  I128* const ex = (I128*)(res_sm + T.ex);
  double tot = 0.0;
  unsigned long long tmax = 0;
  // an element of R, in every CTA's copy
  auto put_r = [&](int64_t i, int64_t r) {
    if constexpr (CS > 1 && MODE >= RES_SHARED) {
#pragma unroll
      for (int q = 0; q < CS; ++q) *cg::this_cluster().map_shared_rank(R + i, q) = r;
    } else {
      R[i] = r;
    }
  };
  // the start vector: R_0 = round(v0 2^-e), max |R_0| < 2^m_in
  unsigned long long mb = 0;
  for (int64_t i = i0; i < D; i += st) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(fabs(start_value(io.start, i, io.seed)));
    mb = max(mb, min(b, 0x7FF0000000000000ull));  // any non-finite value: infinity
  }
  __syncthreads();  // s is free
  if (!scalar) res_put<NT, CS>(s, ex, 0, I128{0, 0}, mb);
  __syncthreads();
  res_get<NT, CS>(s, 0, &tot, &tmax);  // by every warp (the same values)
  csync<CS>();
  if constexpr (CS > 1) res_collect<CS>(s, 0, &tot, &tmax);
  const double mx0 = __longlong_as_double((long long)tmax);
  if (tmax == 0 || tmax >= 0x7FF0000000000000ull) {  // the same in every thread of the cluster
    if (threadIdx.x == 0 && rec) beta[0] = tmax == 0 ? 0.0 : nan("");
    csync<CS>();
    return 0;
  }
  const int e_start = exp2_of(mx0) - P.m_in;
  I128 nn{0, 0};
  unsigned long long mm = 0;
  int l = threadIdx.x;
  for (int64_t i = i0; i < D; i += st, l += NC) {
    const int64_t r = llrint(ldexp(start_value(io.start, i, io.seed), -e_start));
    put_r(i, r);
    Rp[MODE == RES_ALL ? l : i] = 0;
    if (io.store) io.store[i] = r;
    add128(nn, sqr_s64(r));
    mm = max(mm, uabs64(r));
    if (pass2) {
      io.acc_lo[i] = 0;
      io.acc_hi[i] = 0;
    }
  }
  if (!scalar) res_put<NT, CS>(s, ex, 1, nn, mm);
  if (threadIdx.x == 0) {
    s.stop = 0;
    s.m = 0;
    s.me = 0;
    s.lo = 0.0;
    s.hi = 0.0;
    s.bk = 0.0;
    s.ek = e_start;
    s.mk = 0;
  }
  const int Km = (int)min((int64_t)io.K, D);
  const int mlim = pass2 ? io.m_replay : Km;
  // b_k from the posted totals of R_k, and the invariant-subspace test (the scalar warp)
  auto norm_finish = [&](int k) {
    if constexpr (CS > 1) res_collect<CS>(s, 1, &tot, &tmax);
    else res_get<NT, CS>(s, 1, &tot, &tmax);
    const double bk = scale2(sqrt(tot), s.ek);
    __syncwarp();
    if (lane == 0) {
      s.bkm1 = s.bk;
      s.bk = bk;
      s.mp = s.mk;
      s.mk = tmax;
      if (rec) {
        beta[k] = bk;
        io.exps[k] = s.ek;
      }
      if (!pass2) {
        // the new residual vanishes relative to the scale of T (beta[0] holds the start-vector norm,
        // not an entry of T)
        if (k > 0 && (!(bk > 1e-13 * s.row) || tmax == 0)) {
          s.stop = 2;
          s.m = k;
        }
      }
    }
    __syncwarp();
  };
  __syncthreads();
  if constexpr (CS > 1) {
    if (scalar) res_get<NT, CS>(s, 1, &tot, &tmax);
    csync<CS>();  // also orders the cluster's R_0 before the first gathers
  }
  bool pending = true;  // the norm of R_k has been posted, not finished
  for (int k = 0; k < mlim; ++k) {
    if (pass2) {
      const int64_t C = io.Ck[k];
      for (int64_t i = i0; i < D; i += st) {
        I128 v{io.acc_lo[i], io.acc_hi[i]};
        add128(v, mul_s64(C, R[i]));
        io.acc_lo[i] = v.lo;
        io.acc_hi[i] = v.hi;
      }
      if (k + 1 == mlim) break;
    }
    // W = H R_k; meanwhile the scalar warp finishes the norm of R_k
    if (scalar) {
      if (pending) norm_finish(k);
    } else {
      I128 dot;
      unsigned long long mxw;
      res_matvec<NT, MODE, DIAG64>(P, T, R, W, i0, st, &dot, &mxw);
      res_put<NT, CS>(s, ex, 0, dot, mxw);
    }
    __syncthreads();
    if (CS == 1 && s.stop) break;  // R_k spans no new direction: m = k
    if (scalar) res_get<NT, CS>(s, 0, &tot, &tmax);
    if constexpr (CS > 1) {
      csync<CS>();  // every CTA has gathered from R_k
      if (s.stop) break;  // (the same in every CTA)
      if (scalar) res_collect<CS>(s, 0, &tot, &tmax);
    }
    double a_k = 0.0;
    if (scalar) {
      const double bk = s.bk;
      const int ek = s.ek, ep = s.ep, ew = ek - P.F;
      const double a = scale2(tot, ek + ew) / (bk * bk);
      // R_{k+1} on a grid with max |R_{k+1}| < 2^m_in; lanes 0, 1, 2: the three terms
      double cc = (lane == 0 ? 1.0 : (lane == 1 ? -a : -bk)) / (lane == 2 ? s.bkm1 : bk);
      if (lane > 2 || (lane == 2 && k == 0)) cc = 0.0;
      const int ex2 = lane == 0 ? ew : (lane == 1 || k == 0 ? ek : ep);
      const unsigned long long ml = lane == 0 ? tmax : (lane == 1 ? s.mk : s.mp);
      const double term = cc != 0.0 ? fabs(cc) * scale2((double)ml, ex2) : 0.0;
      const double B = (__shfl_sync(0xffffffffu, term, 0) + __shfl_sync(0xffffffffu, term, 1)) +
                       __shfl_sync(0xffffffffu, term, 2);
      const int er = (B > 0.0 ? exp2_of(B) : 1) - P.m_in;
      const double g = cc != 0.0 ? scale2(cc, ex2 - er) : 0.0;
      const int eg = __reduce_max_sync(0xffffffffu, g != 0.0 ? exp2_of(g) : -100000);
      const int SA = min(60, 60 - (eg == -100000 ? 1 : eg));
      const int64_t A = g != 0.0 ? llrint(scale2(g, SA)) : 0;
      const uint64_t mag = uabs64(A);
      // A x = |A| z - |A| (2^63 - [A < 0]) with z = (x ^ sign) + 2^63 >= 0: unsigned products, one constant
      const I128 cl = mul_u64(mag, 0x8000000000000000ull - (A < 0 ? 1 : 0));
      I128 c1{0, 0};
#pragma unroll
      for (int q = 0; q < 3; ++q)
        add128(c1, I128{__shfl_sync(0xffffffffu, cl.lo, q), __shfl_sync(0xffffffffu, cl.hi, q)});
      I128 c2{0ull - c1.lo, -c1.hi - (c1.lo != 0 ? 1 : 0)};
      add128(c2, I128{1ull << (SA - 1), 0});
      __syncwarp();
      if (lane < 3) {
        s.A[lane] = mag;
        s.sgn[lane] = A >> 63;
      }
      if (lane == 0) {
        s.cst = c2;
        s.SA = SA;
        s.ep = ek;
        s.ek = er;
      }
      a_k = a;
    }
    __syncthreads();
    if (scalar) {
      if (lane == 0) {
        if (rec) alpha[k] = a_k;
        s.row = fabs(a_k) + (k > 0 ? s.bk : 0.0) + 1e-300;
      }
      __syncwarp();
    } else {
      const uint64_t Aw = s.A[0], Aq = s.A[1], Ap = s.A[2];  // (Ap = 0 at k = 0)
      const int64_t top = (int64_t)0x8000000000000000ll;
      const int64_t gw = s.sgn[0] ^ top, gq = s.sgn[1] ^ top, gp = s.sgn[2] ^ top;
      const I128 cst = s.cst;
      const int SA = s.SA;
      int64_t* const out = io.store && k + 1 < Km ? io.store + (int64_t)(k + 1) * D : nullptr;
      nn = I128{0, 0};
      mm = 0;
      l = threadIdx.x;
      for (int64_t i = i0; i < D; i += st, l += NC) {
        const int64_t li = MODE == RES_ALL ? (int64_t)l : i;
        const int64_t x = R[i], y = Rp[li], w = W[li];
        I128 t = cst;
        add128(t, mul_u64(Aw, (uint64_t)(w ^ gw)));
        add128(t, mul_u64(Aq, (uint64_t)(x ^ gq)));
        add128(t, mul_u64(Ap, (uint64_t)(y ^ gp)));
        const int64_t r = (int64_t)((t.lo >> SA) | ((uint64_t)t.hi << (64 - SA)));
        Rp[li] = x;
        put_r(i, r);
        if (out) out[i] = r;
        add128(nn, sqr_s64(r));
        mm = max(mm, uabs64(r));
      }
      res_put<NT, CS>(s, ex, 1, nn, mm);
    }
    __syncthreads();
    if constexpr (CS > 1) {
      if (scalar) res_get<NT, CS>(s, 1, &tot, &tmax);
      csync<CS>();  // orders every CTA's part of R_{k+1} before the next gathers
    }
    pending = true;
    if (!pass2 && io.check_every > 0 && (k + 1) % io.check_every == 0 && k + 1 < Km) {
      if (scalar) norm_finish(k + 1);
      pending = false;
      __syncthreads();
      if (s.stop) break;
      // the first CTA of a cluster tests; a pass is confirmed by the careful solver
      if (rk0 && res_test(alpha, beta, k + 1, io.work, s) <= 2.0 * io.tol) {
        const double e = res_tridiag(alpha, beta, k + 1, io.c, io.work, s.lo, s.hi);
        if (threadIdx.x == 0) {
          s.e = e;
          s.me = k + 1;
          if (fabs(beta[k + 1] * io.c[k]) <= io.tol * fmax(1.0, fabs(e))) {
            s.stop = 1;
            s.m = k + 1;
          }
        }
        __syncthreads();
      }
      if constexpr (CS > 1) {
        csync<CS>();  // (s.stop of the first CTA does not change again before the next cluster barrier)
        const int stop0 = *cg::this_cluster().map_shared_rank(&s.stop, 0);
        if (threadIdx.x == 0 && !rk0) {
          s.stop = stop0;
          s.m = k + 1;
        }
        __syncthreads();
      }
      if (s.stop) break;
    }
  }
  __syncthreads();
  if (!pass2 && !s.stop) {  // (uniform) the run took all its steps
    if (pending && scalar) norm_finish(Km);
    __syncthreads();
  }
  const int m = pass2 ? io.m_replay : (s.stop ? s.m : Km);
  csync<CS>();  // the pass's last vector writes and exchange reads, ordered before what follows
  return m;
}

// sum of the threads' FP64 values over the cluster, warp by warp in order (every thread gets it)
template <int NT, int CS>
static __device__ double res_sum_f64(double v, ResShared& s) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s.red[0][threadIdx.x >> 5] = v;
  __syncthreads();
  double r = 0.0;
  for (int i = 0; i < NT / 32; ++i) r += s.red[0][i];
  if constexpr (CS > 1) {
    if (threadIdx.x == 0) s.xd = r;
    csync<CS>();
    r = 0.0;
    for (int q = 0; q < CS; ++q) r += cg::this_cluster().map_shared_rank(&s, q)->xd;
    csync<CS>();
  }
  return r;
}

// One problem from its start vector to its outputs by one CTA or cluster
struct ResIo {
  ResRun run;                     // work: 5 (K + 2) doubles, alpha / beta / c / exps: K + 2
  int64_t* Ck;                    // K + 2
  uint64_t* acc_lo;
  int64_t* acc_hi;
  double *alpha, *beta;           // outputs [K], [K + 1]
  double *energy, *residual;      // null: the coefficients alone
  int32_t* steps;
  double* vec;                    // the ground-state vector or null
};

template <int NT, int CS, int MODE, bool DIAG64>
static __device__ void res_problem(const BatchProblem& P, const ResLayout& L, unsigned char* sm, ResIo& io,
                                   ResShared& s) {
  __shared__ int sh_sc;
  if (MODE != RES_GLOBAL) res_tables(P, L, sm);
  const ResTables T = res_offsets(L);
  const int rk = io.run.rk;
  io.run.m_replay = 0;
  io.run.Ck = nullptr;
  const int m = res_recurrence<NT, CS, MODE, DIAG64>(P, T, io.run, s);
  const double* be = io.run.beta;
  double* c = io.run.c;
  if (rk == 0) {
    for (int k = threadIdx.x; k < m; k += NT) io.alpha[k] = io.run.alpha[k];
    for (int k = threadIdx.x; k <= m; k += NT) io.beta[k] = be[k];
  }
  if (m == 0) {
    if (threadIdx.x == 0 && rk == 0) {
      if (io.energy) {
        *io.energy = nan("");
        *io.residual = 0.0;
      }
      *io.steps = 0;
    }
    return;
  }
  if (threadIdx.x == 0 && rk == 0) *io.steps = m;
  if (!io.energy) return;
  const double e = res_tridiag(io.run.alpha, be, m, c, io.run.work, 0.0, 0.0);
  if (threadIdx.x == 0 && rk == 0) {
    *io.energy = e;
    *io.residual = fabs(be[m] * c[m - 1]);
  }
  if (!io.vec) return;
  // psi = sum_k (c_k / beta_k) R_k,  R_k = Rm_k 2^e_k:  C_k = round(c_k/beta_k 2^(e_k + SC))
  if (threadIdx.x < 32) {
    int eg = -100000;
    for (int k = threadIdx.x; k < m; k += 32) {
      const double v = ldexp(c[k] / be[k], io.run.exps[k]);
      // (a zero matrix leaves NaN in c; its coefficient below still makes a unit vector)
      if (v != 0.0 && isfinite(v)) eg = max(eg, exp2_of(v));
    }
    eg = __reduce_max_sync(0xffffffffu, eg);
    const int sc = 52 - (eg == -100000 ? 1 : eg);
    for (int k = threadIdx.x; k < m; k += 32) io.Ck[k] = llrint(ldexp(c[k] / be[k], io.run.exps[k] + sc));
    if (threadIdx.x == 0) sh_sc = sc;
  }
  __syncthreads();
  io.run.m_replay = m;
  io.run.Ck = io.Ck;
  io.run.acc_lo = io.acc_lo;
  io.run.acc_hi = io.acc_hi;
  res_recurrence<NT, CS, MODE, DIAG64>(P, T, io.run, s);
  // normalise (one CTA: 256 threads, the columns of its sums) and write FP64
  __syncthreads();
  csync<CS>();
  constexpr int NC = NT - 32, NS = CS > 1 ? NC : RES_COLS;
  const int64_t st = (int64_t)CS * NS, i0 = threadIdx.x < NS ? (int64_t)rk * NS + threadIdx.x : P.D;
  double sq = 0.0;
  const int sc = sh_sc;
  for (int64_t i = i0; i < P.D; i += st) {
    const double v = ldexp(i128_to_double(I128{io.acc_lo[i], io.acc_hi[i]}), -sc);
    sq = fma(v, v, sq);
  }
  const double nrm = 1.0 / sqrt(res_sum_f64<NT, CS>(sq, s));
  for (int64_t i = i0; i < P.D; i += st) io.vec[i] = ldexp(i128_to_double(I128{io.acc_lo[i], io.acc_hi[i]}), -sc) * nrm;
}

// res_problem in the mode that L allows (a cluster takes R into shared memory only together with the
// rest, one CTA the tables only together with R)
template <int NT, int CS, bool DIAG64>
static __device__ __forceinline__ void res_dispatch(const BatchProblem& P, const ResLayout& L, unsigned char* sm, ResIo& io,
                                                    ResShared& s) {
  constexpr int SECOND = CS > 1 ? RES_TABLES : RES_SHARED;
  if (L.ws) res_problem<NT, CS, RES_ALL, DIAG64>(P, L, sm, io, s);
  else if (CS > 1 ? L.ts : L.rs) res_problem<NT, CS, SECOND, DIAG64>(P, L, sm, io, s);
  else res_problem<NT, CS, RES_GLOBAL, false>(P, L, sm, io, s);
}

}  // namespace ed
