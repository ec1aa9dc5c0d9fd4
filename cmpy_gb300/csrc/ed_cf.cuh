// The Lanczos continued fraction at one complex frequency,
//   1 / (z - a_0 - b_1^2 / (z - a_1 - ... b_{n-1}^2 / (z - a_{n-1}))),
// by the three-term recurrence of its tails t_l = p_l / p_{l+1} (Wallis; from the last level up):
//   p_l = (z - a_l) p_{l+1} - b_{l+1}^2 p_{l+2},  value p_1 / p_0,
// seven FP64 operations a level and no division, where t_l = z - a_l - b_{l+1}^2 / t_{l+1} takes
// some fifteen. The pipe of this GPU (64 cycles a warp instruction alone, 19 for each when it is full)
// bounds both. p is brought back to size one by its own exponent, an exact power of two, whenever it leaves
// 2^-320 .. 2^320: whatever one level grows by, the next starts in range.
#pragma once

#include "ed_common.cuh"

namespace ed {

constexpr int CF_TILE = 256;  // levels staged in shared memory at a time

// value * norm at (zr, zi); every thread of the block calls it (barriers), `on` = this thread has a
// frequency. a[0..n), b[1..n) of one problem; st: CF_TILE double2 of shared memory
__device__ __forceinline__ double2 cf_value(const double* __restrict__ a, const double* __restrict__ b, int n, double zr,
                                            double zi, double norm, double2* st) {
  double pr = 1.0, pi = 0.0, qr = 0.0, qi = 0.0;  // p_{l+1}, p_{l+2}
  for (int top = n; top > 0; top -= CF_TILE) {
    const int l0 = max(0, top - CF_TILE);
    __syncthreads();
    for (int l = l0 + threadIdx.x; l < top; l += blockDim.x) {
      const double bl = l + 1 < n ? b[l + 1] : 0.0;
      st[l - l0] = make_double2(a[l], bl * bl);
    }
    __syncthreads();
    for (int l = top - 1; l >= l0; --l) {
      const double2 ab = st[l - l0];
      const double ar = zr - ab.x;
      const double nr = fma(-zi, pi, fma(ar, pr, -(ab.y * qr)));
      const double ni = fma(zi, pr, fma(ar, pi, -(ab.y * qi)));
      qr = pr;
      qi = pi;
      pr = nr;
      pi = ni;
      const int e = max(__double2hiint(pr) & 0x7ff00000, __double2hiint(pi) & 0x7ff00000);
      if ((unsigned)(e - 0x2bf00000) > 0x28000000u && e != 0) {  // outside 2^-320 .. 2^320
        const double sc = __hiloint2double(max(0x7fe00000 - e, 0x00100000), 0);  // 2^-e
        pr *= sc;
        pi *= sc;
        qr *= sc;
        qi *= sc;
      }
    }
  }
  const double inv = norm / fma(pr, pr, pi * pi);
  return make_double2((qr * pr + qi * pi) * inv, (qi * pr - qr * pi) * inv);
}

}  // namespace ed
