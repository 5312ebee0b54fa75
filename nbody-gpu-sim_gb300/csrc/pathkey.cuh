// pathkey.cuh -- Morton keys and octant-path keys with the reference's float
// operations.
#pragma once

#include "bh_tree.cuh"
#include "geom.cuh"

namespace nbgb {

__device__ __forceinline__ uint32_t spread3(uint32_t v) {
  v &= 0x3FFu;
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

// computeMortonCode (force_barnes_hut.cu:42-50) on (p - min) * inv.
__device__ __forceinline__ uint32_t morton_of(float4 p, const BBox& b) {
  float nx = __fmul_rn(__fsub_rn(p.x, b.min[0]), b.inv[0]);
  float ny = __fmul_rn(__fsub_rn(p.y, b.min[1]), b.inv[1]);
  float nz = __fmul_rn(__fsub_rn(p.z, b.min[2]), b.inv[2]);
  uint32_t ix = (uint32_t)__fmul_rn(fminf(fmaxf(nx, 0.0f), 1.0f), 1023.0f);
  uint32_t iy = (uint32_t)__fmul_rn(fminf(fmaxf(ny, 0.0f), 1.0f), 1023.0f);
  uint32_t iz = (uint32_t)__fmul_rn(fminf(fmaxf(nz, 0.0f), 1.0f), 1023.0f);
  return (spread3(ix) << 2) | (spread3(iy) << 1) | spread3(iz);
}

// Octant path of a position through the reference's subdivision: the high
// key (levels 1..21, 3 bits each, level 1 most significant) and the low key
// (levels 22..32).
__device__ __forceinline__ void path_key(float4 p, const BBox& b, u64& hi, u64& lo) {
  float cx = b.center[0], cy = b.center[1], cz = b.center[2], h = b.half;
  u64 a = 0, c = 0;
#pragma unroll
  for (int lev = 1; lev <= kMaxDepth; ++lev) {
    const uint32_t o = (p.x >= cx ? 1u : 0u) | (p.y >= cy ? 2u : 0u) | (p.z >= cz ? 4u : 0u);
    const float hs = __fmul_rn(h, 0.5f);
    cx = __fadd_rn(cx, (o & 1u) ? hs : -hs);
    cy = __fadd_rn(cy, (o & 2u) ? hs : -hs);
    cz = __fadd_rn(cz, (o & 4u) ? hs : -hs);
    h = hs;
    if (lev <= kHiLevels)
      a = (a << 3) | o;
    else
      c = (c << 3) | o;
  }
  hi = a;
  lo = c;
}

}  // namespace nbgb
