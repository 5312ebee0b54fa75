// pathsort.cu -- sorts bodies by (segment, high path key, body index).
//
// That order is unique, so no step has to be stable: a sample sort.  Every
// segment has its own buckets (about kPsMean bodies each; PathSortBuckets).
//   1. a stratified sample of `over` keys per bucket is ranked by counting
//      (every sample against every other, over many CTAs); every `over`-th
//      becomes a splitter;
//   2. every body's key is computed and its bucket found by binary search in
//      shared memory; the last CTA turns the bucket counts into offsets;
//   3. bodies are scattered to their buckets (any order within);
//   4. one CTA per bucket splits it the same way into parts of about 32 bodies
//      in shared memory, ranks each body by counting within its part and writes
//      the sorted bodies with their keys, segments and positions.
// A bucket larger than the shared-memory capacity (rare, but any size may
// occur) takes the same steps on its stretch of the global arrays.
//
// What bounds it: latency of the launches below about 100,000 bodies, then
// the instructions of the key computation (21 levels) and of the counting.  The radix sort it replaces ran 8 passes (9 with
// several segments) of 16 ranking rounds each; the warp match instruction, at
// about 65 clocks per warp and SM, made a pass 11 us even for a few tiles.  A
// bitonic network in step 4 took 129 us at N = 1M (58 dependent steps).
#include "pathsort.cuh"

#include <algorithm>

#include "kernels.cuh"

namespace nbgb {

constexpr int kPsMaxSamples = 6 * kPsMaxBuckets;
constexpr int kPsMaxOver = 16;
constexpr int kPsChunk = 64;     // samples one CTA compares with
constexpr int kPsCap = 4096;     // bodies sorted in shared memory
constexpr int kPsPart = 32;      // bodies per part of a bucket
constexpr int kPsMaxParts = 64;
constexpr int kPsWhole = 256;    // buckets up to this size stay one part

struct __align__(16) SplitKey {
  u64 hi;
  uint32_t seg, idx;
};

struct PsWork {
  // zero before each sort (the bounds kernel clears it)
  uint32_t rank[kPsMaxSamples];
  uint32_t count[kPsMaxBuckets];
  uint32_t done[kPsMaxSamples / 256 + 4];  // CTAs done: per 256 samples; [last] counting
  // not zeroed
  uint32_t offset[kPsMaxBuckets + 4];
  uint32_t cursor[kPsMaxBuckets];
  SplitKey split[kPsMaxBuckets];
  SplitKey sample[kPsMaxSamples];
};

size_t path_sort_ws_bytes() { return sizeof(PsWork); }
size_t path_sort_zero_words() { return offsetof(PsWork, offset) / sizeof(uint32_t); }

int path_sort_buckets(const int64_t* n_per, int nseg, int32_t* first) {
  int64_t n = 0;
  for (int s = 0; s < nseg; ++s) n += n_per[s];
  // a bucket per kPsMean bodies, fewer where there would be too many
  const int64_t room = std::max<int64_t>(1, kPsMaxBuckets - nseg);
  const int64_t mean = std::max(kPsMean, ceil_div(n, room));
  int64_t nb = 0;
  for (int s = 0; s < nseg; ++s) {
    first[s] = (int32_t)nb;
    nb += std::max<int64_t>(1, n_per[s] / mean);
  }
  first[nseg] = (int32_t)nb;
  return nseg < kPsMaxBuckets && nb <= kPsMaxBuckets && n <= kPathSortMax ? (int)nb : 0;
}

struct PsArgs {
  const float4* pm;
  SegView sv;
  const int32_t* first;  // first bucket of each segment (nseg + 1)
  int nseg;
  int64_t n;
  int nb;       // buckets
  int over;     // samples per bucket
  PsWork* w;
  PathSortBuffers b;
};

__device__ __forceinline__ u64 hi_key(const PsArgs& a, int s, int64_t q) {
  u64 hi, lo;
  path_key(a.pm[a.sv.off[s] + (q - a.sv.base[s])], a.sv.box[s], hi, lo);
  return hi;
}

__device__ __forceinline__ int segment_of_bucket(const PsArgs& a, int bk) {
  int s = 0, e = a.nseg - 1;
  while (s < e) {  // last segment whose first bucket is not above bk
    const int mid = (s + e + 1) >> 1;
    if (a.first[mid] <= bk)
      s = mid;
    else
      e = mid - 1;
  }
  return s;
}

// Sample i belongs to bucket i / over of its segment's share: a body at a
// hashed place of one of the segment's equal stretches.
__device__ __forceinline__ SplitKey sample_key(const PsArgs& a, int i) {
  const int s = segment_of_bucket(a, i / a.over);
  const int i0 = a.first[s] * a.over, ns = (a.first[s + 1] - a.first[s]) * a.over;
  const int64_t b0 = a.sv.base[s];
  const uint32_t m = (uint32_t)(a.sv.base[s + 1] - b0), step = m / (uint32_t)ns;
  const uint32_t h = (((uint32_t)i * 2654435761u) ^ ((uint32_t)i >> 7)) >> 4;
  SplitKey k;
  const int64_t q = b0 + (step ? (uint32_t)(i - i0) * step + h % step : (uint32_t)(i - i0) % m);
  k.seg = (uint32_t)s;
  k.idx = (uint32_t)q;
  k.hi = hi_key(a, s, q);
  return k;
}

__global__ void ps_sample_kernel(PsArgs a) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < a.nb * a.over) a.w->sample[i] = sample_key(a, i);
}

// (segment, key, index) as one unsigned number.
using u128 = unsigned __int128;
__device__ __forceinline__ u128 wide(const SplitKey& k) {
  return ((u128)(((u64)k.seg << 32) | (k.hi >> 32)) << 64) | ((k.hi << 32) | k.idx);
}

// A segment with one bucket may draw a body twice; its splitter is not used.
__global__ void __launch_bounds__(256) ps_rank_kernel(PsArgs a) {
  chain_begin();
  __shared__ u128 s_k[kPsChunk];
  __shared__ bool s_last;
  const int ns = a.nb * a.over;
  const int i = blockIdx.x * 256 + threadIdx.x, j0 = blockIdx.y * kPsChunk;
  const int nj = min(kPsChunk, ns - j0);
  if ((int)threadIdx.x < nj) s_k[threadIdx.x] = wide(a.w->sample[j0 + threadIdx.x]);
  SplitKey me{};
  if (i < ns) me = a.w->sample[i];
  __syncthreads();
  if (i < ns) {
    const u128 k = wide(me);
    uint32_t r = 0;
#pragma unroll 8
    for (int j = 0; j < nj; ++j) r += s_k[j] < k ? 1u : 0u;
    if (r) atomicAdd(&a.w->rank[i], r);
  }
  // the last CTA of these 256 samples writes the splitters among them: bucket
  // b starts at the sample of rank b * over
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&a.w->done[blockIdx.x], 1u) == gridDim.y - 1;
  __syncthreads();
  if (!s_last || i >= ns) return;
  __threadfence();
  const uint32_t r = __ldcg(&a.w->rank[i]);
  if (r % a.over == 0) a.w->split[r / a.over] = me;
}

// Last of `left` entries from `at` on whose (key, index) is not above (k, q).
__device__ __forceinline__ int last_not_above(const u64* hi, const uint32_t* idx, int at, int left,
                                              u64 k, uint32_t q) {
  while (left > 1) {
    const int half = left >> 1;
    const u64 v = hi[at + half];
    const bool up = v < k || (v == k && idx[at + half] <= q);
    at = up ? at + half : at;
    left = up ? left - half : half;
  }
  return at;
}

// Keys, buckets and bucket counts; the last CTA scans the counts.
__global__ void __launch_bounds__(256) ps_count_kernel(PsArgs a) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char ps_smem[];
  u64* s_hi = reinterpret_cast<u64*>(ps_smem);                    // [nb]
  uint32_t* s_idx = reinterpret_cast<uint32_t*>(s_hi + a.nb);     // [nb]
  uint32_t* s_cnt = s_idx + a.nb;                                 // [nb]
  __shared__ bool s_last;
  __shared__ uint32_t s_w[8];
  for (int b = threadIdx.x; b < a.nb; b += 256) {
    const SplitKey k = a.w->split[b];
    s_hi[b] = k.hi;
    s_idx[b] = k.idx;
    s_cnt[b] = 0;
  }
  __syncthreads();
  for (int64_t q = blockIdx.x * 256ll + threadIdx.x; q < a.n; q += gridDim.x * 256ll) {
    const int s = a.nseg > 1 ? a.sv.seg_of[q] : 0;
    const u64 k = hi_key(a, s, q);
    const int b0 = a.first[s];
    const int at = last_not_above(s_hi, s_idx, b0, a.first[s + 1] - b0, k, (uint32_t)q);
    a.b.key[q] = k;
    a.b.bucket[q] = (uint32_t)at;
    atomicAdd(&s_cnt[at], 1u);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < a.nb; b += 256)
    if (s_cnt[b]) atomicAdd(&a.w->count[b], s_cnt[b]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0)
    s_last = atomicAdd(&a.w->done[kPsMaxSamples / 256], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  uint32_t c[kPsMaxBuckets / 256], sum = 0;
#pragma unroll
  for (int r = 0; r < kPsMaxBuckets / 256; ++r) {
    const int b = threadIdx.x * (kPsMaxBuckets / 256) + r;
    c[r] = b < a.nb ? __ldcg(&a.w->count[b]) : 0u;
    sum += c[r];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_w[warp] = x;
  __syncthreads();
  uint32_t at = x - sum;
  for (int w = 0; w < warp; ++w) at += s_w[w];
#pragma unroll
  for (int r = 0; r < kPsMaxBuckets / 256; ++r) {
    const int b = threadIdx.x * (kPsMaxBuckets / 256) + r;
    if (b < a.nb) {
      a.w->offset[b] = at;
      a.w->cursor[b] = at;
    }
    at += c[r];
  }
  if (threadIdx.x == 0) a.w->offset[a.nb] = (uint32_t)a.n;
}

// Bodies to their buckets: ranks within the CTA by shared-memory counters, one
// reservation per CTA and bucket.
template <int ITEMS>
__global__ void __launch_bounds__(256) ps_scatter_kernel(PsArgs a) {
  chain_begin();
  __shared__ uint32_t s_cnt[kPsMaxBuckets], s_base[kPsMaxBuckets];
  for (int b = threadIdx.x; b < a.nb; b += 256) s_cnt[b] = 0;
  __syncthreads();
  const int64_t q0 = (int64_t)blockIdx.x * (256 * ITEMS) + threadIdx.x;
  uint32_t bk[ITEMS], rk[ITEMS];
  u64 key[ITEMS];
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const int64_t q = q0 + r * 256;
    if (q < a.n) {
      bk[r] = a.b.bucket[q];
      key[r] = a.b.key[q];
    }
  }
#pragma unroll
  for (int r = 0; r < ITEMS; ++r)
    if (q0 + r * 256 < a.n) rk[r] = atomicAdd(&s_cnt[bk[r]], 1u);
  __syncthreads();
  for (int b = threadIdx.x; b < a.nb; b += 256)
    if (s_cnt[b]) s_base[b] = atomicAdd(&a.w->cursor[b], s_cnt[b]);
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const int64_t q = q0 + r * 256;
    if (q < a.n) {
      const uint32_t to = s_base[bk[r]] + rk[r];
      a.b.skey[to] = key[r];
      a.b.sidx[to] = (uint32_t)q;
    }
  }
}

// One bucket of m bodies (in: key, idx).  b_hi, b_idx, b_tmp: m entries of
// scratch, in shared memory or (m above the capacity) the bucket's stretch of
// global arrays; seen: m bits, zero.  Leaves the bodies by part in b_hi, b_idx
// and each one's sorted place in b_tmp.
__device__ __forceinline__ void sort_bucket(int m, const u64* key, const uint32_t* idx, u64* b_hi,
                                            uint32_t* b_idx, uint32_t* b_tmp, uint32_t* seen) {
  __shared__ u64 s_shi[4 * kPsMaxParts], s_phi[kPsMaxParts];
  __shared__ uint32_t s_sidx[4 * kPsMaxParts], s_pidx[kPsMaxParts];
  __shared__ uint32_t s_cnt[kPsMaxParts], s_off[kPsMaxParts + 1];
  __shared__ int s_tie;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int np = m <= kPsWhole ? 1 : min(kPsMaxParts, m / kPsPart);
  if (tid == 0) s_tie = 0;
  if (np == 1) {
    for (int i = tid; i < m; i += nt) {
      b_hi[i] = key[i];
      b_idx[i] = idx[i];
    }
    if (tid == 0) {
      s_off[0] = 0;
      s_off[1] = (uint32_t)m;
    }
  } else {
    // splitters: four samples per part at hashed places, ranked by counting
    const int ns = 4 * np, step = m / ns;
    if (tid < np) s_cnt[tid] = 0;
    if (tid < ns) {
      const int at = tid * step + (int)(((uint32_t)tid * 2654435761u >> 8) % (uint32_t)step);
      s_shi[tid] = key[at];
      s_sidx[tid] = idx[at];
    }
    __syncthreads();
    if (tid < ns) {
      const u64 h = s_shi[tid];
      const uint32_t q = s_sidx[tid];
      int r = 0;
      for (int j = 0; j < ns; ++j)
        r += (s_shi[j] < h || (s_shi[j] == h && s_sidx[j] < q)) ? 1 : 0;
      if ((r & 3) == 0) {
        s_phi[r >> 2] = h;
        s_pidx[r >> 2] = q;
      }
    }
    __syncthreads();
    for (int i = tid; i < m; i += nt) {
      const int p = last_not_above(s_phi, s_pidx, 0, np, key[i], idx[i]);
      b_tmp[i] = (uint32_t)p << 24;
      b_idx[i] = atomicAdd(&s_cnt[p], 1u);  // place within the part, for now
    }
    __syncthreads();
    if (tid < 32) {
      const uint32_t c0 = 2 * tid < np ? s_cnt[2 * tid] : 0u,
                     c1 = 2 * tid + 1 < np ? s_cnt[2 * tid + 1] : 0u;
      uint32_t x = c0 + c1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (tid >= o) x += y;
      }
      s_off[2 * tid] = x - c0 - c1;
      s_off[2 * tid + 1] = x - c1;
      if (tid == 31) s_off[kPsMaxParts] = x;
    }
    __syncthreads();
    for (int i = tid; i < m; i += nt) b_tmp[i] = s_off[b_tmp[i] >> 24] + b_idx[i];
    __syncthreads();
    for (int i = tid; i < m; i += nt) {
      b_hi[b_tmp[i]] = key[i];
      b_idx[b_tmp[i]] = idx[i];
    }
  }
  __syncthreads();
  // ranks by counting within the part, by key alone; two bodies of one rank
  // have equal keys, and then all ranks are taken again by (key, index)
  for (int pass = 0; pass < 2; ++pass) {
    for (int i = tid; i < m; i += nt) {
      int p = 0;
      for (int left = np; left > 1;) {
        const int half = left >> 1;
        const bool up = s_off[p + half] <= (uint32_t)i;
        p = up ? p + half : p;
        left = up ? left - half : half;
      }
      const int o = (int)s_off[p], e = p + 1 < np ? (int)s_off[p + 1] : m;
      const u64 h = b_hi[i];
      int r = o;
      if (pass == 0) {
#pragma unroll 4
        for (int j = o; j < e; ++j) r += b_hi[j] < h ? 1 : 0;
        const uint32_t bit = 1u << (r & 31);
        if (atomicOr(&seen[r >> 5], bit) & bit) s_tie = 1;
      } else {
        const uint32_t q = b_idx[i];
        for (int j = o; j < e; ++j) {
          const u64 v = b_hi[j];
          r += (v < h || (v == h && b_idx[j] < q)) ? 1 : 0;
        }
      }
      b_tmp[i] = (uint32_t)r;
    }
    __syncthreads();
    if (!s_tie) break;
  }
}

__global__ void __launch_bounds__(512) ps_local_kernel(PsArgs a) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char ps_smem[];
  u64* s_hi = reinterpret_cast<u64*>(ps_smem);                      // [kPsCap]
  uint32_t* s_idx = reinterpret_cast<uint32_t*>(s_hi + kPsCap);     // [kPsCap]
  uint32_t* s_tmp = s_idx + kPsCap;                                 // [kPsCap]
  uint32_t* s_seen = s_tmp + kPsCap;                                // [kPsCap / 32]
  const uint32_t o = a.w->offset[blockIdx.x];
  const int m = (int)(a.w->offset[blockIdx.x + 1] - o);
  const int s = segment_of_bucket(a, (int)blockIdx.x);
  const float4* pm = a.pm + (a.sv.off[s] - a.sv.base[s]);
  if (m <= kPsCap) {
    for (int i = threadIdx.x; i < (m + 31) / 32; i += blockDim.x) s_seen[i] = 0;
    __syncthreads();
    sort_bucket(m, a.b.skey + o, a.b.sidx + o, s_hi, s_idx, s_tmp, s_seen);
  } else {
    // global scratch: the bucket's stretch of arrays that are free by now (the
    // keys by body, the results it will write)
    u64* g_hi = a.b.key + o;
    uint32_t* g_idx = a.b.bucket + o;
    uint32_t* g_tmp = reinterpret_cast<uint32_t*>(a.b.kseg + o);
    uint32_t* g_seen = a.b.body + o;
    for (int i = threadIdx.x; i < (m + 31) / 32; i += blockDim.x) g_seen[i] = 0;
    __syncthreads();
    sort_bucket(m, a.b.skey + o, a.b.sidx + o, g_hi, g_idx, g_tmp, g_seen);
    // the sorted bodies over the scattered ones; the scratch is free again
    for (int i = threadIdx.x; i < m; i += blockDim.x) a.b.sidx[o + g_tmp[i]] = g_idx[i];
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
      const uint32_t k = o + i, q = a.b.sidx[k];
      const float4 p = pm[q];
      u64 h, l;
      path_key(p, a.sv.box[s], h, l);
      a.b.body[k] = q;
      a.b.kseg[k] = s;
      a.b.hi[k] = h;
      a.b.spm[k] = p;
    }
    return;
  }
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    const uint32_t k = o + s_tmp[i], q = s_idx[i];
    a.b.body[k] = q;
    a.b.kseg[k] = s;
    a.b.hi[k] = s_hi[i];
    a.b.spm[k] = pm[q];
  }
}

void path_sort(const float4* pm, const SegView& sv, const int32_t* first, int nb, int64_t n,
               int nseg, const PathSortBuffers& b, StageTimer* timer, cudaStream_t st) {
  stage_mark(timer, "barnes_hut.keys");
  PsArgs a;
  a.pm = pm;
  a.sv = sv;
  a.first = first;
  a.nseg = nseg;
  a.n = n;
  a.nb = nb;
  // more samples even out the buckets, and keep large ones (mean above 512)
  // within the capacity; the ranking grows with their square
  a.over = n / nb > 512 ? kPsMaxSamples / kPsMaxBuckets
                        : std::max(4, std::min(kPsMaxOver, 2048 / nb));
  a.w = reinterpret_cast<PsWork*>(b.ws);
  a.b = b;
  const int ns = nb * a.over;
  const dim3 g((unsigned)ceil_div(ns, 256), (unsigned)ceil_div(ns, kPsChunk));
  launch_chained(ps_sample_kernel, (unsigned)ceil_div(ns, 64), 64, 0, st, a);
  launch_chained(ps_rank_kernel, g, 256, 0, st, a);
  const unsigned gc =
      (unsigned)std::min<int64_t>(ceil_div(n, 256), (int64_t)num_sms() * 4);
  if (n < 262144) {
    launch_chained(ps_count_kernel, gc, 256, (size_t)nb * 16, st, a);
  } else {
    // (not chained: blocks placed beside the ranking's last ones share SMs to the end,
    // the keys of 1M bodies 85 us instead of 65)
    ps_count_kernel<<<gc, 256, (size_t)nb * 16, st>>>(a);
    NBGB_LAUNCH_CHECK();
  }
  stage_mark(timer, "barnes_hut.sort");
  if (n < 262144)
    launch_chained(ps_scatter_kernel<2>, (unsigned)ceil_div(n, 512), 256, 0, st, a);
  else
    launch_chained(ps_scatter_kernel<8>, (unsigned)ceil_div(n, 2048), 256, 0, st, a);
  constexpr size_t smem = (size_t)kPsCap * 16 + kPsCap / 8;
  NBGB_CUDA(cudaFuncSetAttribute(ps_local_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
  launch_chained(ps_local_kernel, (unsigned)nb, n / nb <= 512 ? 256 : 512, smem, st, a);
}

}  // namespace nbgb
