// The Lanczos continued fraction at one complex frequency,
//   1 / (z - a_0 - b_1^2 / (z - a_1 - ... b_{n-1}^2 / (z - a_{n-1}))),
// by the three-term recurrence of its tails t_l = p_l / p_{l+1} (Wallis; from the last level up):
//   p_l = (z - a_l) p_{l+1} - b_{l+1}^2 p_{l+2},
// seven FP64 operations a level and no division, where t_l = z - a_l - b_{l+1}^2 / t_{l+1} takes
// some fifteen. The pipe of this GPU (64 cycles a warp instruction alone, 19 for each when it is full)
// bounds both. p is brought back to size one by its own exponent, an exact power of two, whenever it leaves
// 2^-320 .. 2^320: whatever one level grows by, the next starts in range.
#pragma once

#include "ed_common.cuh"

namespace ed {

constexpr int CF_TILE = 256;  // levels staged in shared memory at a time
// The levels nearest to the value are taken as tails: their roundings are the ones that the value keeps (a
// deeper level's is damped by every b^2 / t^2 above it). Root mean square error against extended precision, 400
// coefficient sets, relative to tails throughout: no such level 1.09 (Matsubara), 1.10 and 1.06 (0.05 and 0.2
// above the real axis); four 1.00, 1.02, 1.02; eight 1.00, 1.00, 1.01.
constexpr int CF_LAST = 8;

// 2^-e of a number of exponent e, from its exponent bits (clamped to the normal powers of two)
__device__ __forceinline__ double cf_unit(int e) { return __hiloint2double(max(0x7fe00000 - e, 0x00100000), 0); }
__device__ __forceinline__ int cf_exponent(double x, double y) {
  return max(__double2hiint(x) & 0x7ff00000, __double2hiint(y) & 0x7ff00000);
}

// value * norm at (zr, zi); every thread of the block calls it (barriers).
// a[0..n), b[1..n) of one problem; st: CF_TILE double2 of shared memory
__device__ __forceinline__ double2 cf_value(const double* __restrict__ a, const double* __restrict__ b, int n, double zr,
                                            double zi, double norm, double2* st) {
  const int last = min(CF_LAST, n - 1);
  double pr = 1.0, pi = 0.0, qr = 0.0, qi = 0.0;  // p_{l+1}, p_{l+2}
  for (int top = n, l0; top > 0; top = l0) {
    l0 = (top - 1) / CF_TILE * CF_TILE;
    __syncthreads();
    for (int l = l0 + threadIdx.x; l < top; l += blockDim.x) {
      const double bl = l + 1 < n ? b[l + 1] : 0.0;
      st[l - l0] = make_double2(a[l], bl * bl);
    }
    __syncthreads();
    for (int l = top - 1; l >= max(l0, last); --l) {
      const double2 ab = st[l - l0];
      const double ar = zr - ab.x;
      const double nr = fma(-zi, pi, fma(ar, pr, -(ab.y * qr)));
      const double ni = fma(zi, pr, fma(ar, pi, -(ab.y * qi)));
      qr = pr;
      qi = pi;
      pr = nr;
      pi = ni;
      const int e = cf_exponent(pr, pi);
      if ((unsigned)(e - 0x2bf00000) > 0x28000000u && e != 0) {  // outside 2^-320 .. 2^320
        const double sc = cf_unit(e);
        pr *= sc;
        pi *= sc;
        qr *= sc;
        qi *= sc;
      }
    }
  }
  // t = p_last / p_{last+1}, and the levels above it (in the last tile, which starts at level 0)
  const double su = cf_unit(cf_exponent(qr, qi));
  qr *= su;
  qi *= su;
  const double iq = 1.0 / fma(qr, qr, qi * qi);
  double tr = fma(pr, qr, pi * qi) * iq * su, tm = fma(pi, qr, -(pr * qi)) * iq * su;
  for (int l = last - 1; l >= 0; --l) {
    const double2 ab = st[l];
    const double inv = ab.y / fma(tr, tr, tm * tm);
    tr = fma(-tr, inv, zr - ab.x);
    tm = fma(tm, inv, zi);
  }
  const double inv = norm / fma(tr, tr, tm * tm);
  return make_double2(tr * inv, -tm * inv);
}

}  // namespace ed
