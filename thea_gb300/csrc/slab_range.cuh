// The value of n . v for a slab's range (host and device; compiles with nvcc and with a plain C++ compiler): an interval of
// two floats that holds it, as tight as the exact value rounded outwards to float (one ulp more where that value lies within
// 2^-44 of the products' magnitudes from a float). Each product is a float and its exact error (fused multiply-add), the sums
// carry theirs along (Knuth's two-sum), so the arithmetic runs on the FP32 pipe and keeps about 45 bits; the same values in
// FP64 took most of the range pass's time on the FP64 pipe, and plain FP32 sums widened by their own rounding lose three
// bits of the range's 24 and more where the products cancel (a mesh far from the origin).
#pragma once

#include <cmath>

#if defined(__CUDACC__)
#define THEA_SLAB_HD __host__ __device__ __forceinline__
#else
#define THEA_SLAB_HD inline
#endif

namespace thea {

// s + e = a + b exactly (short of overflow)
THEA_SLAB_HD float slab_two_sum(float a, float b, float & e) {
  float s = a + b;
  float t = s - a;
  e = (a - (s - t)) + (b - t);
  return s;
}

// The largest float <= a + b, and the smallest >= a + b
THEA_SLAB_HD float slab_add_down(float a, float b) {
#if defined(__CUDA_ARCH__)
  return __fadd_rd(a, b);
#else
  float e, s = slab_two_sum(a, b, e);
  return e < 0.f ? nextafterf(s, -INFINITY) : s;
#endif
}
THEA_SLAB_HD float slab_add_up(float a, float b) { return -slab_add_down(-a, -b); }

// [lo, hi] around nx vx + ny vy + nz vz; [-inf, inf] where a product is not finite
THEA_SLAB_HD void slab_project(float nx, float ny, float nz, float vx, float vy, float vz, float & lo, float & hi) {
  float x = nx * vx, y = ny * vy, z = nz * vz;
  float mag = fabsf(x) + fabsf(y) + fabsf(z);
  if (!(mag < INFINITY)) {
    lo = -INFINITY;
    hi = INFINITY;
    return;
  }
  float xe = fmaf(nx, vx, -x), ye = fmaf(ny, vy, -y), ze = fmaf(nz, vz, -z);
  float e1, e2;
  float s = slab_two_sum(slab_two_sum(x, y, e1), z, e2);
  float e = (e1 + e2) + (xe + ye + ze);
  // the sum of the errors, each at most 2^-24 of `mag`, is rounded four times: within 2^-45 of it in all. (The constant:
  // products below the normal range, whose errors are not floats.)
  float w = mag * (1.0f / 17592186044416.0f) + 1e-44f;  // 2^-44
  lo = slab_add_down(s, e - w);
  hi = slab_add_up(s, e + w);
}

}  // namespace thea
