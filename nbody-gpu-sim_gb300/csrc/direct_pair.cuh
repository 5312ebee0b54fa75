// direct_pair.cuh -- the direct-sum inner loop: one thread sums I targets
// against a shared-memory tile, two consecutive sources per packed FP32x2
// operation.
#pragma once

#include "common.cuh"

namespace nbgb {

// Adds t to a running sum: error-free into (s, e), or in plain FP32.
template <bool COMP>
__device__ __forceinline__ void fold(float t, float& s, float& e) {
  if constexpr (COMP) {
    float d;
    s = two_sum(s, t, d);
    e += d;
  } else {
    s += t;
  }
}

// One pair of sources added to one target (both halves of x, y, z the
// target's coordinate).  12 packed operations and 2 MUFU per 2 interactions.
template <bool ZERO_SOFT>
__device__ __forceinline__ void pair_step(f2 xj, f2 yj, f2 zj, f2 mj, f2 x, f2 y, f2 z, f2 e2,
                                          f2& ax, f2& ay, f2& az) {
  const f2 dx = f2_sub(xj, x);
  const f2 dy = f2_sub(yj, y);
  const f2 dz = f2_sub(zj, z);
  const f2 d2 = f2_fma(dx, dx, f2_fma(dy, dy, f2_fma(dz, dz, e2)));
  float d2l, d2h;
  f2_split(d2, d2l, d2h);
  float rl = rsqrt_approx(d2l), rh = rsqrt_approx(d2h);
  if constexpr (ZERO_SOFT) {  // coincident bodies (and the target itself) add nothing
    rl = (d2l > 0.f) ? rl : 0.f;
    rh = (d2h > 0.f) ? rh : 0.f;
  }
  const f2 r = f2_make(rl, rh);
  const f2 f = f2_mul(f2_mul(mj, r), f2_mul(r, r));
  ax = f2_fma(f, dx, ax);
  ay = f2_fma(f, dy, ay);
  az = f2_fma(f, dz, az);
}

// Tile rows x, y, z, m; sources [jb, je), both multiples of 4.  Four sources
// per step: one 16-byte broadcast load per row feeds 2 I pair steps.
template <int I, bool ZERO_SOFT, int ROW>
__device__ __forceinline__ void pair_sum(const float (&s)[4][ROW], int jb, int je,
                                         const f2 (&x)[I], const f2 (&y)[I], const f2 (&z)[I],
                                         f2 e2, f2 (&ax)[I], f2 (&ay)[I], f2 (&az)[I]) {
#pragma unroll 4
  for (int j = jb; j < je; j += 4) {
    const ulonglong2 X = *reinterpret_cast<const ulonglong2*>(&s[0][j]);
    const ulonglong2 Y = *reinterpret_cast<const ulonglong2*>(&s[1][j]);
    const ulonglong2 Z = *reinterpret_cast<const ulonglong2*>(&s[2][j]);
    const ulonglong2 M = *reinterpret_cast<const ulonglong2*>(&s[3][j]);
#pragma unroll
    for (int q = 0; q < I; ++q)
      pair_step<ZERO_SOFT>(f2{X.x}, f2{Y.x}, f2{Z.x}, f2{M.x}, x[q], y[q], z[q], e2, ax[q], ay[q],
                           az[q]);
#pragma unroll
    for (int q = 0; q < I; ++q)
      pair_step<ZERO_SOFT>(f2{X.y}, f2{Y.y}, f2{Z.y}, f2{M.y}, x[q], y[q], z[q], e2, ax[q], ay[q],
                           az[q]);
  }
}

}  // namespace nbgb
