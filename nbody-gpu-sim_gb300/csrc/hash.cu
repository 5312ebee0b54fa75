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
#include <vector>

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
  DevBuf<int32_t> particle_cell;
  DevBuf<uint32_t> count;   // bodies per cell (total_cells + 1, the last 0)
  DevBuf<uint32_t> start;   // a cell's first slot (total_cells + 1): each cell has an
                            // even number of slots, a last odd one without a body
  DevBuf<uint32_t> placed;  // slots: bodies in any order within the cell
  DevBuf<uint32_t> idx;     // slots: bodies in ascending order within the cell
  DevBuf<uint32_t> cells;   // pairs of slots: their cell
  DevBuf<float4> pairs;     // pairs of slots: their bodies
  DevBuf<uint32_t> scan_ws;
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
__global__ void hash_count_kernel(const float4* pm, int64_t n, GridArgs g, int32_t* particle_cell,
                                  uint32_t* count, uint32_t* place) {
  chain_begin();
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  // (four bodies' loads ahead of the first one's stores)
  for (int64_t w0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x - lane); w0 < n; w0 += 4 * step) {
    float4 p[4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (w0 + r * step + lane < n) p[r] = pm[w0 + r * step + lane];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int64_t i = w0 + r * step + lane;
      const bool on = i < n;
      const int32_t id = on ? cell_of(p[r], g) : 0;
      const unsigned mask = __ballot_sync(0xffffffffu, on);
      if (!mask) break;
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
}

__global__ void hash_place_kernel(const int32_t* particle_cell, const uint32_t* place,
                                  const uint32_t* start, int64_t n, uint32_t* idx) {
  chain_begin();
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i0 < n; i0 += 4 * step) {
    uint32_t at[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int64_t i = i0 + r * step;
      if (i < n) at[r] = start[particle_cell[i]] + place[i];
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (i0 + r * step < n) idx[at[r]] = (uint32_t)(i0 + r * step);
  }
}

// Bodies in cell order, two per 32-byte record (x0 x1 y0 y1 z0 z1 m0 m1), so
// that two candidates arrive as packed FP32x2 operands.  A cell starts a record:
// no candidate of a range has to be masked out, and a record's two bodies are
// targets with the same candidates.  A body with a NaN coordinate is put where its
// squared distance overflows to infinity, outside every cutoff (in the test
// d^2 < rc^2 a NaN never passes).  A slot without a body is filled the same way,
// without mass.
constexpr uint32_t kNoBody = 0xffffffffu;
constexpr float kFarAway = 3.0e38f;  // (bodies are within 1e30, where the box's bounds start)

// The bodies of each cell in ascending order, and their records: a body's place
// is the number of smaller indices in its cell.  In a cell of at most kHashCrowd
// bodies each thread compares its own.  A block meets at most two larger cells,
// its first and its last slot's; there every index of the cell is looked up among
// the block's sorted ones, so a cell of c bodies costs c * c / kHashCrowd lookups
// and not c * c compares (60 K bodies in one cell 74 us against 926).
constexpr int kHashCrowd = 256;  // threads (and slots) per block, too

__global__ void __launch_bounds__(kHashCrowd) hash_order_kernel(
    const float4* pm, int64_t n, GridArgs g, int64_t total, const uint32_t* placed,
    const uint32_t* count, const uint32_t* start, uint32_t* cells, uint32_t* idx, float* out) {
  chain_begin();
  __shared__ uint32_t s_idx[kHashCrowd], s_sorted[kHashCrowd];
  __shared__ uint32_t s_hist[2][kHashCrowd + 1];
  __shared__ uint32_t s_cell[2][2];  // first and last slot's cell: start, end
  const int tid = threadIdx.x;
  const int64_t slots = start[total];
  const int64_t p0 = blockIdx.x * (int64_t)kHashCrowd, p = p0 + tid;
  const int64_t p1 = imin64(p0 + kHashCrowd, slots);
  if (p0 >= slots) return;
  float4 b = make_float4(kFarAway, 0.f, 0.f, 0.f);
  uint32_t i = p < slots ? placed[p] : kNoBody, s = 0, e = 0, r = 0;
  if (i < n) {
    b = pm[i];
    const int32_t id = cell_of(b, g);
    if (!(b.x == b.x && b.y == b.y && b.z == b.z)) b = make_float4(kFarAway, 0.f, 0.f, b.w);
    if (!(p & 1)) cells[p >> 1] = (uint32_t)id;
    s = start[id];
    e = s + count[id];
  }
  // a cell's odd last slot holds nothing: it is not below the end of the cell
  // that the slot before it belongs to
  const uint32_t before = __shfl_up_sync(0xffffffffu, e, 1);
  if (p >= slots || ((p & 1) && p >= before)) {
    i = kNoBody;
    s = e = 0;
    b = make_float4(kFarAway, 0.f, 0.f, 0.f);
  }
  const bool crowd = e - s > (uint32_t)kHashCrowd;
  if (!crowd)
    for (uint32_t q = s; q < e; ++q) r += placed[q] < i ? 1u : 0u;
  if (__syncthreads_or(crowd)) {
    s_idx[tid] = i;
    // (the block's first slot has a body; its last two slots are of one cell)
    if (p == p0 || p == p1 - 2) {
      const int w = p == p0 ? 0 : 1;
      s_cell[w][0] = s;
      s_cell[w][1] = e;
      if (p0 == p1 - 2) s_cell[1][0] = s_cell[1][1] = 0;
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
        const uint32_t v = placed[q];
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
  if (p >= slots) return;
  const int64_t at = i != kNoBody ? (int64_t)s + r : p;
  idx[at] = i;
  float* o = out + (at >> 1) * 8 + (at & 1);
  o[0] = b.x;
  o[2] = b.y;
  o[4] = b.z;
  o[6] = b.w;
}

// The 27-cell gather.  Cells cx-1 .. cx+1 of a neighbour row are consecutive
// records, so a pair of targets walks 9 ranges, two candidates per packed step
// and without a branch on the cutoff: with 15 % of the candidates accepted almost
// every warp took both paths of a branch.  A rejected candidate's force factor is
// zero.  The squared distance uses the reference's rounding (packed operations
// round each half like the scalar ones), so neighbour counts stay bit-exact.
// A thread has the two bodies of a record as targets: with one, the candidates'
// way from L1 to the registers (32 bytes per thread and step, 67 % of that path)
// was as busy as the issue slots (4M bodies 814 us, now 678).
//
// SUB threads share a pair's records, an equal run of all nine rows' each, where
// the targets alone do not fill the GPU; their sums are added in order.  ROWS: a
// thread's run is taken row by row in a tight loop, which pays where rows are long;
// otherwise it goes on to the next row at once, without waiting for the longest
// row of the warp (of 8 cells with 24 candidates per row on average).
template <bool COUNT, int SUB, int T, bool ROWS>
__global__ void __launch_bounds__(SUB * T) hash_force_kernel(
    const float4* pairs, const uint32_t* cells, const uint32_t* idx, const uint32_t* start,
    int64_t total, GridArgs g, float cut2, float eps2, float G, float* ax, float* ay, float* az,
    int32_t* counts) {
  chain_begin();
  __shared__ uint2 s_row[9][T];  // records of each neighbour row
  const int t = threadIdx.x % T, sub = threadIdx.x / T;  // pair of the block, its thread
  const int64_t npairs = start[total] >> 1;
  const int64_t k = (int64_t)blockIdx.x * T + t;
  if ((int64_t)blockIdx.x * T >= npairs) return;
  const bool valid = k < npairs;
  const uint32_t me = (uint32_t)(valid ? k : npairs - 1);
  const float4 own0 = pairs[2 * (int64_t)me], own1 = pairs[2 * (int64_t)me + 1];
  const float px[2] = {own0.x, own0.y};
  const f2 xi[2] = {f2_make(own0.x, own0.x), f2_make(own0.y, own0.y)};
  const f2 yi[2] = {f2_make(own0.z, own0.z), f2_make(own0.w, own0.w)};
  const f2 zi[2] = {f2_make(own1.x, own1.x), f2_make(own1.y, own1.y)};
  const f2 e2 = f2_make(eps2, eps2);
  const int id = (int)cells[me];
  const int gxy = g.dims[0] * g.dims[1];
  const int cz = id / gxy;
  const int rem = id - cz * gxy;
  const int cy = rem / g.dims[0];
  const int cx = rem - cy * g.dims[0];
  const int x0 = max(cx - 1, 0), x1 = min(cx + 1, g.dims[0] - 1) + 1;
  f2 sum[2][3];
#pragma unroll
  for (int c = 0; c < 3; ++c) sum[0][c] = sum[1][c] = f2_make(0.f, 0.f);
  int cnt[2] = {0, 0};
  uint32_t len = 0;
#pragma unroll 1
  for (int r = sub; r < 9; r += SUB) {
    const int nz = cz + r / 3 - 1, ny = cy + r % 3 - 1;
    uint2 se = make_uint2(0, 0);
    if (nz >= 0 && nz < g.dims[2] && ny >= 0 && ny < g.dims[1]) {
      const int base = ny * g.dims[0] + nz * gxy;
      se = make_uint2(start[base + x0] >> 1, start[base + x1] >> 1);
    }
    s_row[r][t] = se;
    len += se.y - se.x;
  }
  auto add = [&](uint32_t j) {
    const ulonglong2* rec = reinterpret_cast<const ulonglong2*>(pairs) + 2 * (uint64_t)j;
    const ulonglong2 xy = rec[0], zm = rec[1];
    const bool other = j != me;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const f2 dx = f2_sub(f2{xy.x}, xi[q]), dy = f2_sub(f2{xy.y}, yi[q]),
               dz = f2_sub(f2{zm.x}, zi[q]);
      const f2 d2 = f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx)));
      float dl, dh;
      f2_split(d2, dl, dh);
      const bool ol = dl < cut2 && (q == 1 || other), oh = dh < cut2 && (q == 0 || other);
      const f2 s2 = f2_add(d2, e2);
      f2_split(s2, dl, dh);
      const f2 rs = f2_make(rsqrt_approx(dl), rsqrt_approx(dh));
      f2 f = f2_mul(f2_mul(f2{zm.y}, rs), f2_mul(rs, rs));
      float fl, fh;
      f2_split(f, fl, fh);
      f = f2_make(ol ? fl : 0.f, oh ? fh : 0.f);
      sum[q][0] = f2_fma(f, dx, sum[q][0]);
      sum[q][1] = f2_fma(f, dy, sum[q][1]);
      sum[q][2] = f2_fma(f, dz, sum[q][2]);
      if (COUNT) cnt[q] += (ol ? 1 : 0) + (oh ? 1 : 0);
    }
  };
  uint32_t lo = 0, hi = len;
  if constexpr (SUB > 1) {
    __syncthreads();
    len = 0;
#pragma unroll
    for (int r = 0; r < 9; ++r) len += s_row[r][t].y - s_row[r][t].x;
    // records [lo, hi) of all nine rows
    lo = (uint32_t)((uint64_t)len * sub / SUB);
    hi = (uint32_t)((uint64_t)len * (sub + 1) / SUB);
  }
  if constexpr (!ROWS) {
    // row after row without waiting for the warp's longer rows
    uint2 se = make_uint2(0, 0);
    int r = -1;
    uint32_t left = hi - lo;
    if (SUB > 1) {
      while (left > 0) {
        se = s_row[++r][t];
        if (lo < se.y - se.x) break;
        lo -= se.y - se.x;
      }
      se.x += lo;
    }
#pragma unroll 1
    for (; left > 0; --left) {
      while (se.x == se.y) se = s_row[++r][t];
      add(se.x++);
    }
  } else {
#pragma unroll 1
    for (int r = 0; r < 9 && hi > 0; ++r) {
      const uint2 se = s_row[r][t];
      const uint32_t l = se.y - se.x, a = min(lo, l), b = min(hi, l);
      for (uint32_t j = se.x + a; j < se.x + b; ++j) add(j);
      lo -= a;
      hi -= b;
    }
  }
  float v[2][3];
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float hi;
      f2_split(sum[q][c], v[q][c], hi);
      v[q][c] += hi;
    }
  if constexpr (SUB > 1) {
    __shared__ float s_sum[SUB - 1][6][T];
    __shared__ int s_cnt[COUNT ? SUB - 1 : 1][2][T];
    if (sub > 0) {
#pragma unroll
      for (int c = 0; c < 6; ++c) s_sum[sub - 1][c][t] = v[c / 3][c % 3];
      if (COUNT) {
        s_cnt[sub - 1][0][t] = cnt[0];
        s_cnt[sub - 1][1][t] = cnt[1];
      }
    }
    __syncthreads();
    if (sub > 0) return;
#pragma unroll
    for (int q = 0; q < SUB - 1; ++q) {
#pragma unroll
      for (int c = 0; c < 6; ++c) v[c / 3][c % 3] += s_sum[q][c][t];
      if (COUNT) {
        cnt[0] += s_cnt[q][0][t];
        cnt[1] += s_cnt[q][1][t];
      }
    }
  }
  if (!valid) return;
  const uint2 who = reinterpret_cast<const uint2*>(idx)[me];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const uint32_t i = q ? who.y : who.x;
    if (i == kNoBody) continue;
    const bool nan = px[q] == kFarAway;  // a NaN position has no neighbours
    ax[i] = nan ? 0.f : G * v[q][0];
    ay[i] = nan ? 0.f : G * v[q][1];
    az[i] = nan ? 0.f : G * v[q][2];
    if (COUNT) counts[i] = nan ? 0 : cnt[q];
  }
}

static unsigned grid1d(int64_t n, int threads = 256) {
  return (unsigned)std::max<int64_t>(
      1, std::min<int64_t>(ceil_div(std::max<int64_t>(n, 1), threads), (int64_t)num_sms() * 32));
}

constexpr int64_t kHashMaxCells = 100000000;  // the reference's cap

// How the gather's work is split (in us, uniform cubes):
//  threads per pair  at 8 bodies per cell 30 K: 9 take 14, 4 take 18, 1 takes 43;
//                    400 K: 90, 80, 93; 1M: 215, 186, 176;
//                    at 64 and more per cell 60 K bodies: 16 take 116, 9 take 121;
//                    500 K: 516, 460
//  rows or one run   of records per thread: 60 K at 114 per cell 121 against 128, 1M
//                    at 200 per cell 2462 against 2691; 1M at 8 per cell 291
//                    against 215.
constexpr int64_t kHashDense = 24;         // bodies per cell on average
constexpr int64_t kHashSplitMax = 131072;  // bodies
constexpr int64_t kHashWholeMin = 524288;  // bodies

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
    const float cells = std::ceil((float)q);
    g.bmin[a] = lo;
    // (checked per axis: a product of three could wrap around, as could the conversion)
    if (cells < (float)kHashMaxCells) {
      g.dims[a] = (int)cells + 1;
      total *= (int64_t)g.dims[a];
    } else {
      total = kHashMaxCells + 1;
    }
    if (total > kHashMaxCells)
      fail(NBGB_ERR_OVERFLOW, "Spatial hash grid too large: reduce cell_size or bounding box");
  }
  g.cell = cell;
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
  uint32_t* count = h.count.ensure((size_t)total + 1);
  uint32_t* start = h.start.ensure((size_t)total + 1);
  const size_t slots = (size_t)(n + std::min(n, total));  // at most
  uint32_t* placed = h.placed.ensure(slots);
  uint32_t* idx = h.idx.ensure(slots);
  uint32_t* cells = h.cells.ensure(slots / 2 + 1);
  float4* pairs = h.pairs.ensure(slots + 1);
  uint32_t* place = idx;  // free until the last kernel fills it
  uint32_t* sws = h.scan_ws.ensure(scan_workspace_elems(total + 1));
  NBGB_CUDA(cudaMemsetAsync(count, 0, ((size_t)total + 1) * sizeof(uint32_t), st));
  launch_chained(hash_count_kernel, grid1d(n), 256, 0, st, pm, n, g, pc, count, place);
  // 3. cell starts and places
  stage_mark(timer, "spatial_hash.sort");
  scan_exclusive_even_u32(count, start, total + 1, sws, st);
  launch_chained(hash_place_kernel, grid1d(n), 256, 0, st, pc, place, start, n, placed);
  // 4.-5. order within the cells, and records in that order
  stage_mark(timer, "spatial_hash.cells");
  launch_chained(hash_order_kernel, (unsigned)ceil_div((int64_t)slots, kHashCrowd), kHashCrowd, 0,
                 st, pm, n, g, total, placed, count, start, cells, idx,
                 reinterpret_cast<float*>(pairs));
  // 6. cutoff gather
  stage_mark(timer, "spatial_hash.forces");
  const float eps = c->params.softening, rc = c->params.cutoff;
  const bool counting = (c->params.flags & NBGB_FLAG_COUNT_INTERACTIONS) != 0;
  int32_t* counts = counting ? c->counts.ensure((size_t)n) : nullptr;
  const auto force = [&](auto cnt, auto sub, auto rows) {
    constexpr int S = decltype(sub)::value, T = S == 1 ? 128 : S == 4 ? 64 : 32;
    launch_chained(hash_force_kernel<decltype(cnt)::value, S, T, decltype(rows)::value>,
                   (unsigned)ceil_div((int64_t)(slots / 2), T), T * S, 0, st, pairs, cells, idx,
                   start, total, g, rc * rc, eps * eps, c->params.G, ax, ay, az, counts);
  };
  const auto pick = [&](auto cnt) {
    using std::integral_constant;
    if (n >= kHashDense * total) {
      if (n < kHashSplitMax)
        force(cnt, integral_constant<int, 16>{}, std::true_type{});
      else
        force(cnt, integral_constant<int, 9>{}, std::true_type{});
    } else if (n < kHashSplitMax) {
      force(cnt, integral_constant<int, 9>{}, std::false_type{});
    } else if (n < kHashWholeMin) {
      force(cnt, integral_constant<int, 4>{}, std::false_type{});
    } else {
      force(cnt, integral_constant<int, 1>{}, std::false_type{});
    }
  };
  if (counting)
    pick(std::true_type{});
  else
    pick(std::false_type{});
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
  std::vector<uint32_t> cnt, idx;
  try {
    cnt.resize(tot);
    idx.resize(sorted_indices ? n + std::min(n, tot) : 0);
  } catch (...) {
    return NBGB_ERR_OOM;
  }
  cudaError_t e = cudaSuccess;
  if ((cell_start || cell_end || sorted_indices) && e == cudaSuccess)
    e = cudaMemcpy(cnt.data(), h.count.ptr, tot * 4, cudaMemcpyDeviceToHost);
  if (sorted_indices && e == cudaSuccess)
    e = cudaMemcpy(idx.data(), h.idx.ptr, idx.size() * 4, cudaMemcpyDeviceToHost);
  if (particle_cells && e == cudaSuccess)
    e = cudaMemcpy(particle_cells, h.particle_cell.ptr, n * 4, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return NBGB_ERR_CUDA;
  // the slots without a body left out
  size_t at = 0, slot = 0;
  for (size_t c = 0; c < tot; ++c) {
    if (cell_start) cell_start[c] = (int32_t)at;
    if (sorted_indices)
      for (uint32_t k = 0; k < cnt[c]; ++k) sorted_indices[at + k] = (int32_t)idx[slot + k];
    at += cnt[c];
    slot += (cnt[c] + 1u) & ~1u;
    if (cell_end) cell_end[c] = (int32_t)at;
  }
  return NBGB_OK;
}

}  // extern "C"
