// hash.cu -- spatial hash: stable counting order by cell + 27-cell cutoff
// gather (K7).
//
// Replaces SpatialHashGrid::build / computeForces and
// SpatialHashCalculator::computeForces (src/cuda/force_spatial_hash.cu:241-388):
//  * bbox on the device (geom.cu), padded by 0.001f on the host with the
//    reference's float operations, dims = (int)ceilf((max-min)/cell) + 1,
//    1e8-cell cap (:232-260).  The kernel writes the box to mapped host memory,
//    one stream synchronisation per build (the reference does 12 allocations and 12 synchronous copies).
//  * cell id = clamp(floor((p - min) / cell)) with IEEE division, linear
//    x + y*gx + z*gx*gy (:29-50); the effective cell size is
//    max(cell_size, cutoff) (:382).
//  * count / scan / place (:53-81,292-308) with the same cell_start / cell_end,
//    and then each cell's bodies in ascending index (the reference's within-cell
//    order is whatever its atomics produced).
//  * positions+masses are gathered into cell order (two bodies per 32-byte
//    record), so the force kernel streams contiguous memory per neighbour row.
//  * force: targets in cell order; 27 neighbours dz, dy, dx; skip j == i;
//    accept d^2 < rc^2 on the unsoftened distance, then add
//    m_j d (d^2 + eps^2)^-3/2; scaled by G at the end (:84-158).  d^2 is
//    fma(dz,dz, fma(dy,dy, dx*dx)) with _rn intrinsics, the contraction nvcc
//    gives the reference's source, so neighbour counts match the oracle
//    bit-exactly.
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "geom.cuh"
#include "kernels.cuh"
#include "runtime.cuh"
#include "sort.cuh"

namespace nbgb {

struct HashState {
  DevBuf<float> bbox_part;
  DevBuf<uint32_t> box_ctr;  // zero between builds
  HostPinned<HostBox> h_box;
  DevBuf<uint32_t> placed;      // bodies by cell, in any order within it
  DevBuf<uint32_t> cells, idx;  // cell and index of the bodies in cell order
  DevBuf<uint32_t> scan_ws;
  DevBuf<int32_t> particle_cell;
  DevBuf<uint32_t> cell_start;  // total_cells + 1
  DevBuf<float4> sorted_pm;
  // last build
  int64_t n = 0;
  int dims[3] = {0, 0, 0};
  float bmin[3] = {0, 0, 0};
  float cell = 0.f;
  int64_t total = 0;
  bool built = false;  // the last build finished (the inspection calls read its buffers)
};

void hash_state_delete(HashState* p) { delete p; }

struct GridArgs {
  float bmin[3];
  float cell;
  int dims[3];
};

__device__ __forceinline__ int32_t cell_of(float4 p, const GridArgs& g) {
  int cx = (int)floorf(__fdiv_rn(__fsub_rn(p.x, g.bmin[0]), g.cell));
  int cy = (int)floorf(__fdiv_rn(__fsub_rn(p.y, g.bmin[1]), g.cell));
  int cz = (int)floorf(__fdiv_rn(__fsub_rn(p.z, g.bmin[2]), g.cell));
  cx = max(0, min(cx, g.dims[0] - 1));
  cy = max(0, min(cy, g.dims[1] - 1));
  cz = max(0, min(cz, g.dims[2] - 1));
  return cx + cy * g.dims[0] + cz * g.dims[0] * g.dims[1];
}

// Cell order by counting: count the bodies per cell with atomics, scan, place,
// and put each cell's bodies in ascending order.  Two random 4-byte accesses per
// body bound it (4M bodies 164 us; a radix sort of the cell ids, the cell starts
// by binary search and the records took 258).  The atomics hand out the places
// within a cell in any order, which the last kernel makes good.
__global__ void hash_count_kernel(const float4* __restrict__ pm, int64_t n, GridArgs g,
                                  int32_t* __restrict__ particle_cell,
                                  uint32_t* __restrict__ count, uint32_t* __restrict__ place) {
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
#pragma unroll 4
  for (int64_t w = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x - lane); w < n; w += step) {
    const int64_t i = w + lane;
    const bool on = i < n;
    const int32_t id = on ? cell_of(pm[i], g) : 0;
    const unsigned mask = __ballot_sync(0xffffffffu, on);
    const int32_t id0 = __shfl_sync(0xffffffffu, id, 0);
    uint32_t at = 0;
    if (__all_sync(0xffffffffu, !on || id == id0)) {
      // one cell: one atomic (a whole system in one cell would queue at it)
      if (lane == 0) at = atomicAdd(&count[id], (uint32_t)__popc(mask));
      at = __shfl_sync(0xffffffffu, at, 0) + lane;
    } else if (on) {
      at = atomicAdd(&count[id], 1u);
    }
    if (on) {
      particle_cell[i] = id;
      place[i] = at;
    }
  }
}

__global__ void hash_place_kernel(const int32_t* __restrict__ particle_cell,
                                  const uint32_t* __restrict__ place,
                                  const uint32_t* __restrict__ start, int64_t n,
                                  uint32_t* __restrict__ idx) {
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
#pragma unroll 4
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += step) {
    idx[start[particle_cell[i]] + place[i]] = (uint32_t)i;
  }
}

// Bodies in cell order, two per 32-byte record (x0 x1 y0 y1 z0 z1 m0 m1), so
// that two candidates arrive as packed FP32x2 operands.  A body with a NaN
// coordinate is put where its squared distance overflows to infinity, outside
// every cutoff (in the test d^2 < rc^2 a NaN never passes).  An odd last half
// is filled the same way, without mass.
__device__ __forceinline__ float4 gather_record(float4 q) {
  return q.x == q.x && q.y == q.y && q.z == q.z ? q : make_float4(3.0e38f, 0.f, 0.f, q.w);
}

// The bodies of each cell in ascending order, and their records: a body's place
// is the number of smaller indices in its cell.  In a cell of at most kHashCrowd
// bodies each thread compares its own.  A block meets at most two larger cells,
// its first and its last slot's; there every index of the cell is looked up among
// the block's sorted ones, so a cell of c bodies costs c * c / kHashCrowd lookups
// and not c * c compares (60 K bodies in one cell 74 us against 926).
constexpr int kHashCrowd = 256;  // threads (and slots) per block, too

__global__ void __launch_bounds__(kHashCrowd) hash_order_kernel(
    const float4* __restrict__ pm, GridArgs g, const uint32_t* __restrict__ idx,
    const uint32_t* __restrict__ start, int64_t n, uint32_t* __restrict__ cells,
    uint32_t* __restrict__ sorted_idx, float* __restrict__ out) {
  __shared__ uint32_t s_idx[kHashCrowd], s_sorted[kHashCrowd];
  __shared__ uint32_t s_hist[2][kHashCrowd + 1];
  __shared__ uint32_t s_cell[2][2];  // first and last slot's cell: start, end
  const int tid = threadIdx.x;
  const int64_t p0 = blockIdx.x * (int64_t)kHashCrowd, p = p0 + tid;
  const int64_t p1 = imin64(p0 + kHashCrowd, n);
  float4 b = make_float4(3.0e38f, 0.f, 0.f, 0.f);
  uint32_t i = 0, s = 0, e = 0, r = 0;
  if (p < n) {
    i = idx[p];
    b = pm[i];
    const int32_t id = cell_of(b, g);
    b = gather_record(b);
    cells[p] = (uint32_t)id;
    s = start[id];
    e = start[id + 1];
  }
  const bool crowd = e - s > (uint32_t)kHashCrowd;
  if (!crowd)
    for (uint32_t q = s; q < e; ++q) r += idx[q] < i ? 1u : 0u;
  if (__syncthreads_or(crowd)) {
    s_idx[tid] = i;
    if (p == p0 || p == p1 - 1) {
      const int w = p == p0 ? 0 : 1;
      s_cell[w][0] = s;
      s_cell[w][1] = e;
      if (p0 == p1 - 1) s_cell[1][0] = s_cell[1][1] = 0;
    }
    __syncthreads();
    for (int w = 0; w < 2; ++w) {
      const uint32_t cs = s_cell[w][0], ce = s_cell[w][1];
      if (ce - cs <= (uint32_t)kHashCrowd || (w == 1 && cs == s_cell[0][0])) continue;
      // the block's slots [a, z) of this cell, sorted
      const int a = cs > (uint32_t)p0 ? (int)(cs - (uint32_t)p0) : 0;
      const int z = (int)imin64((int64_t)ce, p1) - (int)p0;
      const bool mine = tid >= a && tid < z;
      int own = 0;
      if (mine) {
        for (int q = a; q < z; ++q) own += s_idx[q] < i ? 1 : 0;
        s_sorted[own] = i;
      } else {
        s_sorted[z - a + (tid < a ? tid : tid - (z - a))] = 0xffffffffu;
      }
      s_hist[0][tid] = 0;
      __syncthreads();
#pragma unroll 4
      for (uint32_t q = cs + tid; q < ce; q += kHashCrowd) {
        const uint32_t v = idx[q];
        int at = 0;  // sorted entries not above v
#pragma unroll
        for (int h = kHashCrowd / 2; h > 0; h >>= 1) at += s_sorted[at + h - 1] <= v ? h : 0;
        at += s_sorted[at] <= v ? 1 : 0;
        if (at < kHashCrowd) atomicAdd(&s_hist[0][at], 1u);
      }
      __syncthreads();
      int f = 0;
      for (int o = 1; o < kHashCrowd; o <<= 1) {
        s_hist[f ^ 1][tid] = s_hist[f][tid] + (tid >= o ? s_hist[f][tid - o] : 0u);
        f ^= 1;
        __syncthreads();
      }
      if (mine) r = s_hist[f][own];
      __syncthreads();
    }
  }
  if (p > n || (p == n && !(n & 1))) return;  // an odd last half is filled, too
  const int64_t at = p < n ? (int64_t)s + r : p;
  if (p < n) sorted_idx[at] = i;
  float* o = out + (at >> 1) * 8 + (at & 1);
  o[0] = b.x;
  o[2] = b.y;
  o[4] = b.z;
  o[6] = b.w;
}

// The 27-cell gather.  Cells cx-1 .. cx+1 of a neighbour row are consecutive
// in the sorted bodies, so a target walks 9 ranges, two candidates per packed
// step and without a branch on the cutoff: with 15 % of the candidates
// accepted almost every warp took both paths of a branch (24 to 31
// instructions per candidate, 21 of 32 lanes active).  A rejected candidate's
// force factor is zero.  The squared distance uses the reference's rounding
// (packed operations round each half like the scalar ones), so neighbour
// counts stay bit-exact.
//
// SUB threads share a target's rows (9 / SUB each) where the targets alone do
// not fill the GPU; their sums are added in row order.
template <bool COUNT, int SUB>
__global__ void __launch_bounds__(SUB == 1 ? 256 : 288) hash_force_kernel(
    const float4* __restrict__ spm, const uint32_t* __restrict__ sorted_cells,
    const uint32_t* __restrict__ sorted_idx, const uint32_t* __restrict__ start, int64_t n,
    GridArgs g, float cut2, float eps2, float G, float* __restrict__ ax, float* __restrict__ ay,
    float* __restrict__ az, int32_t* __restrict__ counts) {
  constexpr int T = SUB == 1 ? 256 : 32;  // targets per block
  const int t = threadIdx.x % T, sub = threadIdx.x / T;
  const int64_t k = (int64_t)blockIdx.x * T + t;
  const bool valid = k < n;
  const int64_t kk = valid ? k : n - 1;
  const float* sf = reinterpret_cast<const float*>(spm);
  const int64_t me = (kk >> 1) * 8 + (kk & 1);
  const float px = sf[me], py = sf[me + 2], pz = sf[me + 4];
  const f2 xi = f2_make(px, px), yi = f2_make(py, py), zi = f2_make(pz, pz);
  const f2 e2 = f2_make(eps2, eps2);
  const int id = (int)sorted_cells[kk];
  const int gxy = g.dims[0] * g.dims[1];
  const int cz = id / gxy;
  const int rem = id - cz * gxy;
  const int cy = rem / g.dims[0];
  const int cx = rem - cy * g.dims[0];
  const int x0 = max(cx - 1, 0), x1 = min(cx + 1, g.dims[0] - 1) + 1;
  f2 sx = f2_make(0.f, 0.f), sy = sx, sz = sx;
  int cnt = 0;
  // candidates [s, e) of one row; self: the row that holds the target
  auto row = [&](uint32_t s, uint32_t e, auto self) {
    for (uint32_t j = s & ~1u; j < e; j += 2) {
      const float4* rec = spm + j;  // record j / 2: two float4
      const ulonglong2 xy = __ldg(reinterpret_cast<const ulonglong2*>(rec));
      const ulonglong2 zm = __ldg(reinterpret_cast<const ulonglong2*>(rec + 1));
      const f2 dx = f2_sub(f2{xy.x}, xi), dy = f2_sub(f2{xy.y}, yi), dz = f2_sub(f2{zm.x}, zi);
      const f2 d2 = f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx)));
      float dl, dh;
      f2_split(d2, dl, dh);
      bool ol = dl < cut2 && j >= s, oh = dh < cut2 && j + 1 < e;
      if constexpr (decltype(self)::value) {
        ol = ol && (int64_t)j != kk;
        oh = oh && (int64_t)j + 1 != kk;
      }
      const f2 s2 = f2_add(d2, e2);
      f2_split(s2, dl, dh);
      const f2 r = f2_make(rsqrt_approx(dl), rsqrt_approx(dh));
      f2 f = f2_mul(f2_mul(f2{zm.y}, r), f2_mul(r, r));
      float fl, fh;
      f2_split(f, fl, fh);
      f = f2_make(ol ? fl : 0.f, oh ? fh : 0.f);
      sx = f2_fma(f, dx, sx);
      sy = f2_fma(f, dy, sy);
      sz = f2_fma(f, dz, sz);
      if (COUNT) cnt += (ol ? 1 : 0) + (oh ? 1 : 0);
    }
  };
#pragma unroll 1
  for (int r = sub * (9 / SUB); r < (sub + 1) * (9 / SUB); ++r) {
    const int nz = cz + r / 3 - 1, ny = cy + r % 3 - 1;
    if (nz < 0 || nz >= g.dims[2] || ny < 0 || ny >= g.dims[1]) continue;
    const int base = ny * g.dims[0] + nz * gxy;
    const uint32_t s = start[base + x0], e = start[base + x1];
    if (r == 4)
      row(s, e, std::true_type{});
    else
      row(s, e, std::false_type{});
  }
  float v[3], hi;
  f2_split(sx, v[0], hi);
  v[0] += hi;
  f2_split(sy, v[1], hi);
  v[1] += hi;
  f2_split(sz, v[2], hi);
  v[2] += hi;
  if constexpr (SUB > 1) {
    __shared__ float s_sum[SUB - 1][3][T];
    __shared__ int s_cnt[COUNT ? SUB - 1 : 1][T];
    if (sub > 0) {
#pragma unroll
      for (int c = 0; c < 3; ++c) s_sum[sub - 1][c][t] = v[c];
      if (COUNT) s_cnt[sub - 1][t] = cnt;
    }
    __syncthreads();
    if (sub > 0) return;
#pragma unroll
    for (int q = 0; q < SUB - 1; ++q) {
#pragma unroll
      for (int c = 0; c < 3; ++c) v[c] += s_sum[q][c][t];
      if (COUNT) cnt += s_cnt[q][t];
    }
  }
  if (!valid) return;
  const uint32_t i = sorted_idx[k];
  const bool nan = px == 3.0e38f;  // a NaN position has no neighbours
  ax[i] = nan ? 0.f : G * v[0];
  ay[i] = nan ? 0.f : G * v[1];
  az[i] = nan ? 0.f : G * v[2];
  if (COUNT) counts[i] = nan ? 0 : cnt;
}

static unsigned grid1d(int64_t n, int threads = 256) {
  return (unsigned)std::max<int64_t>(
      1, std::min<int64_t>(ceil_div(std::max<int64_t>(n, 1), threads), (int64_t)num_sms() * 32));
}

// One thread per target of the gather from this many bodies on, below it nine
// (one per neighbour row): N = 1M at 8 bodies per cell 209 against 226 us,
// N = 200 K 55 against 53, N = 60 K at 114 bodies per cell 343 against 126.
constexpr int64_t kHashOneThreadMin = 400000;

void hash_forces(nbgb_calculator* c, const float4* pm, int64_t n, float* ax, float* ay,
                 float* az) {
  if (!c->hash) c->hash.reset(new HashState());
  HashState& h = *c->hash;
  h.built = false;
  StageTimer* timer = stage_timer(c);
  stage_mark(timer, "spatial_hash.bounds");
  cudaStream_t st = c->stream;
  uint32_t* err = c->err.ensure(1);
  // 1. bounding box -> host (sizes the grid)
  float* part = h.bbox_part.ensure((size_t)bbox_blocks(n) * 6);
  if (!h.box_ctr.ptr) {
    h.box_ctr.ensure(1);
    NBGB_CUDA(cudaMemsetAsync(h.box_ctr.ptr, 0, sizeof(uint32_t), st));
  }
  HostBox* hb = h.h_box.ensure(1);
  launch_bbox(pm, n, part, h.box_ctr.ptr, hb, err, st);
  NBGB_CUDA(cudaStreamSynchronize(st));
  if (!hb->valid) fail(NBGB_ERR_INVALID_ARG, "Validation Error: non-finite particle position");
  const float cell = std::max(c->params.cell_size, c->params.cutoff);
  GridArgs g;
  int64_t total = 1;
  for (int a = 0; a < 3; ++a) {
    volatile float lo = hb->min[a] - 0.001f;  // force float rounding of each step
    volatile float hi = hb->max[a] + 0.001f;
    float ext = hi - lo;
    volatile float q = ext / cell;
    g.bmin[a] = lo;
    g.dims[a] = (int)std::ceil((float)q) + 1;
    total *= (int64_t)g.dims[a];
  }
  g.cell = cell;
  if (total > 100000000)
    fail(NBGB_ERR_OVERFLOW, "Spatial hash grid too large: reduce cell_size or bounding box");
  h.n = n;
  h.total = total;
  h.cell = cell;
  for (int a = 0; a < 3; ++a) {
    h.dims[a] = g.dims[a];
    h.bmin[a] = g.bmin[a];
  }
  // 2. assign cells
  stage_mark(timer, "spatial_hash.assign");
  int32_t* pc = h.particle_cell.ensure((size_t)n);
  uint32_t* placed = h.placed.ensure((size_t)n);
  uint32_t* cells = h.cells.ensure((size_t)n);
  uint32_t* idx = h.idx.ensure((size_t)n);
  uint32_t* place = idx;  // free until the last kernel fills it
  uint32_t* start = h.cell_start.ensure((size_t)total + 1);
  float4* spm = h.sorted_pm.ensure((size_t)n + 1);
  uint32_t* sws = h.scan_ws.ensure(scan_workspace_elems(total + 1));
  NBGB_CUDA(cudaMemsetAsync(start, 0, ((size_t)total + 1) * sizeof(uint32_t), st));
  hash_count_kernel<<<grid1d(n), 256, 0, st>>>(pm, n, g, pc, start, place);
  NBGB_LAUNCH_CHECK();
  // 3. cell starts and places
  stage_mark(timer, "spatial_hash.sort");
  scan_exclusive_u32(start, start, total + 1, sws, nullptr, st);
  hash_place_kernel<<<grid1d(n), 256, 0, st>>>(pc, place, start, n, placed);
  NBGB_LAUNCH_CHECK();
  // 4.-5. order within the cells, and records in that order
  stage_mark(timer, "spatial_hash.cells");
  hash_order_kernel<<<(unsigned)ceil_div(n + 1, kHashCrowd), kHashCrowd, 0, st>>>(
      pm, g, placed, start, n, cells, idx, reinterpret_cast<float*>(spm));
  NBGB_LAUNCH_CHECK();
  // 6. cutoff gather
  stage_mark(timer, "spatial_hash.forces");
  const float eps = c->params.softening, rc = c->params.cutoff;
  const bool count = (c->params.flags & NBGB_FLAG_COUNT_INTERACTIONS) != 0;
  int32_t* counts = count ? c->counts.ensure((size_t)n) : nullptr;
  const auto force = [&](auto cnt, auto sub) {
    constexpr int S = decltype(sub)::value, T = S == 1 ? 256 : 32;
    hash_force_kernel<decltype(cnt)::value, S>
        <<<(unsigned)ceil_div(n, T), T * S, 0, st>>>(spm, cells, idx, start,
                                                     n, g, rc * rc, eps * eps, c->params.G, ax,
                                                     ay, az, counts);
  };
  const auto pick = [&](auto cnt) {
    if (n >= kHashOneThreadMin)
      force(cnt, std::integral_constant<int, 1>{});
    else
      force(cnt, std::integral_constant<int, 9>{});
  };
  if (count)
    pick(std::true_type{});
  else
    pick(std::false_type{});
  NBGB_LAUNCH_CHECK();
  h.built = true;
}

}  // namespace nbgb

using namespace nbgb;

extern "C" {

nbgb_status nbgb_hash_grid_info(nbgb_calculator* c, int32_t dims[3], float bbox_min[3],
                                float* cell_size, int64_t* total_cells) {
  if (!c || !c->hash || c->method != NBGB_SPATIAL_HASH || !c->hash->built)
    return NBGB_ERR_INVALID_ARG;
  const HashState& h = *c->hash;
  for (int a = 0; a < 3; ++a) {
    if (dims) dims[a] = h.dims[a];
    if (bbox_min) bbox_min[a] = h.bmin[a];
  }
  if (cell_size) *cell_size = h.cell;
  if (total_cells) *total_cells = h.total;
  return NBGB_OK;
}

nbgb_status nbgb_hash_copy_cells(nbgb_calculator* c, int32_t* cell_start, int32_t* cell_end,
                                 int32_t* particle_cells, int32_t* sorted_indices) {
  if (!c || !c->hash || c->method != NBGB_SPATIAL_HASH || !c->hash->built)
    return NBGB_ERR_INVALID_ARG;
  HashState& h = *c->hash;
  if (cudaStreamSynchronize(c->stream) != cudaSuccess) return NBGB_ERR_CUDA;
  const size_t tot = (size_t)h.total, n = (size_t)h.n;
  cudaError_t e = cudaSuccess;
  if (cell_start && e == cudaSuccess)
    e = cudaMemcpy(cell_start, h.cell_start.ptr, tot * 4, cudaMemcpyDeviceToHost);
  if (cell_end && e == cudaSuccess)
    e = cudaMemcpy(cell_end, h.cell_start.ptr + 1, tot * 4, cudaMemcpyDeviceToHost);
  if (particle_cells && e == cudaSuccess)
    e = cudaMemcpy(particle_cells, h.particle_cell.ptr, n * 4, cudaMemcpyDeviceToHost);
  if (sorted_indices && e == cudaSuccess)
    e = cudaMemcpy(sorted_indices, h.idx.ptr, n * 4, cudaMemcpyDeviceToHost);
  return e == cudaSuccess ? NBGB_OK : NBGB_ERR_CUDA;
}

}  // extern "C"
