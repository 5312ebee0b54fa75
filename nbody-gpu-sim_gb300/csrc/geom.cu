// geom.cu -- bounding box of the packed positions (K2 first half).
//
// Replaces computeBoundingBoxKernel + atomicMin/MaxFloat and the host wrapper
// that mallocs, copies and frees six scalars every step
// (src/cuda/force_barnes_hut.cu:53-122,266-306).  Min/max are exact, so the
// result equals the reference's whatever the reduction order.  One kernel that
// writes the box to mapped host memory: the caller sizes its grid from it
// after a stream synchronisation.  (A Barnes-Hut build has its own, per segment.)
#include "common.cuh"
#include "geom.cuh"
#include "kernels.cuh"

namespace nbgb {

constexpr int kBoxThreads = 256;

// Minima and maxima of one block's values, in thread 0's mn / mx.
__device__ __forceinline__ void block_min_max(float (&mn)[3], float (&mx)[3], float (*s)[6]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      mn[a] = fminf(mn[a], __shfl_down_sync(0xffffffffu, mn[a], o));
      mx[a] = fmaxf(mx[a], __shfl_down_sync(0xffffffffu, mx[a], o));
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      s[warp][a] = mn[a];
      s[warp][3 + a] = mx[a];
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kBoxThreads / 32; ++w)
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        mn[a] = fminf(mn[a], s[w][a]);
        mx[a] = fmaxf(mx[a], s[w][3 + a]);
      }
  }
  __syncthreads();
}

// Memory bound (16 bytes per body): four independent loads per thread and turn.
// The last block folds the blocks' partials (one thread that folded them took
// longer than the pass over 4M bodies) and leaves the counter zero.
__global__ void __launch_bounds__(kBoxThreads) bbox_kernel(const float4* pm, int64_t n,
                                                           float* part, uint32_t* counter,
                                                           HostBox* out, uint32_t* err) {
  chain_begin();
  __shared__ float s[kBoxThreads / 32][6];
  __shared__ bool s_last;
  float mn[3] = {1e30f, 1e30f, 1e30f}, mx[3] = {-1e30f, -1e30f, -1e30f};
  const int64_t step = (int64_t)gridDim.x * kBoxThreads;
#pragma unroll 4
  for (int64_t i = blockIdx.x * (int64_t)kBoxThreads + threadIdx.x; i < n; i += step) {
    const float4 p = pm[i];
    mn[0] = fminf(mn[0], p.x);
    mn[1] = fminf(mn[1], p.y);
    mn[2] = fminf(mn[2], p.z);
    mx[0] = fmaxf(mx[0], p.x);
    mx[1] = fmaxf(mx[1], p.y);
    mx[2] = fmaxf(mx[2], p.z);
  }
  block_min_max(mn, mx, s);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      __stcg(&part[(int64_t)blockIdx.x * 6 + a], mn[a]);
      __stcg(&part[(int64_t)blockIdx.x * 6 + 3 + a], mx[a]);
    }
    __threadfence();
    s_last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    mn[a] = 1e30f;
    mx[a] = -1e30f;
  }
  for (int b = threadIdx.x; b < (int)gridDim.x; b += kBoxThreads)
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      mn[a] = fminf(mn[a], __ldcg(&part[b * 6 + a]));
      mx[a] = fmaxf(mx[a], __ldcg(&part[b * 6 + 3 + a]));
    }
  block_min_max(mn, mx, s);
  if (threadIdx.x != 0) return;
  bool ok = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    out->min[a] = mn[a];
    out->max[a] = mx[a];
    ok = ok && isfinite(mn[a]) && isfinite(mx[a]);
  }
  out->valid = ok ? 1 : 0;
  if (!ok) raise_error(err, kErrBadInput);
  *counter = 0;
}

int bbox_blocks(int64_t n) {
  return (int)std::max<int64_t>(
      1, std::min<int64_t>(ceil_div(n, kBoxThreads * 4), (int64_t)num_sms() * 4));
}

void launch_bbox(const float4* pm, int64_t n, float* partials, uint32_t* counter, HostBox* out,
                 uint32_t* err, cudaStream_t st) {
  launch_chained(bbox_kernel, bbox_blocks(n), kBoxThreads, 0, st, pm, n, partials, counter, out, err);
}

}  // namespace nbgb
