// bh.cu -- Barnes-Hut on the device: bounds, path keys and their order, and the
// octree from sorted keys (K2-K5), for one system or for many independent
// systems ("segments") in one pass.
//
// Replaces BarnesHutTree::build/computeForces and BarnesHutCalculator
// (src/cuda/force_barnes_hut.cu:125-583), whose octree is built on the host
// by sequential insertion and copied to the device every step.
//
// Tree.  The reference inserts bodies in Morton order into a point-region
// octree with one body per leaf, splitting leaves by float geometric
// subdivision (child centre = c +- half/2, octant bit0 = x >= c, bit1 = y,
// bit2 = z) down to depth 32, where bodies merge (:391-510).  Without the
// node-budget merge (:449-453, which only fires for N below ~64) that tree
// is canonical: a node exists for every octant-path prefix whose parent holds
// >= 2 bodies, a leaf is the shortest prefix unique to its body, and depth-32
// cells hold all their bodies.  It is built here in parallel:
//   1. per segment, the bounding box and the reference's root cube; every
//      body's path key = its 32 octants, computed with the reference's float
//      operations (levels 1..21 in a high 63-bit key, 22..32 in a low key);
//   2. order by (segment, high key, index): a sample sort (pathsort.cu), or for
//      larger sets a stable radix sort by the high key and then by segment;
//      bodies sharing segment and high key are put in (low key, Morton key,
//      index) order, i.e. the reference's insertion order inside a shared
//      depth-32 cell;
//   3. l_k = common levels of adjacent sorted keys of one segment; body k
//      starts the internal nodes of depths l_{k-1}+1 .. min(l_k, 31) and
//      (unless it shares a depth-32 cell with k-1) one leaf of depth
//      min(32, max(l_{k-1}, l_k) + 1); the first body of a segment also
//      starts the segment's root;
//   4. an exclusive scan of those counts numbers the nodes in depth-first
//      pre-order (children in octant order): every subtree, and every
//      segment's tree, is a contiguous index range, and
//      skip(P) = first node of body end(P)+1;
//   5. centres of mass bottom-up, summing children in octant order with the
//      reference's float operations (:514-538), so masses and centres of mass
//      are bit-identical (3.-5. in bh_nodes.cu).
//
// The reference walk is in bh_walk.cu, the group walk (one list per group of
// nearby bodies) in bh_group.cu; the node record, state and shared parameters
// in bh_tree.cuh.
#include <algorithm>
#include <atomic>
#include <vector>

#include "bh.cuh"
#include "bh_tree.cuh"
#include "common.cuh"
#include "geom.cuh"
#include "kernels.cuh"
#include "pathkey.cuh"
#include "pathsort.cuh"
#include "runtime.cuh"
#include "sort.cuh"

namespace nbgb {

void bh_state_delete(BHState* p) { delete p; }

// ----------------------------------------------------- segment setup --
__global__ void seg_of_kernel(const int64_t* __restrict__ base, int nseg, int64_t n,
                              int32_t* __restrict__ seg_of) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n;
       q += (int64_t)gridDim.x * blockDim.x) {
    int lo = 0, hi = nseg - 1;
    while (lo < hi) {  // last s with base[s] <= q
      const int mid = (lo + hi + 1) >> 1;
      if (base[mid] <= q)
        lo = mid;
      else
        hi = mid - 1;
    }
    seg_of[q] = lo;
  }
}

// Per-segment min/max of the bodies, and from them the reference's derived
// constants with its float operations
//   Morton scale  inv = 1.0f / (max - min + 0.001f)            (:313-320)
//   root centre   (min + max) * 0.5f                           (:418-419)
//   root half     max(ex, ey, ez) * 0.5f + 0.001f, first max   (:420-422)
// A block reduces a contiguous chunk; when the chunk lies in one segment (the
// common case) it issues one atomic per bound, otherwise each lane does; the
// last block derives the boxes.  Min/max are exact, so the result equals the
// reference's computeBoundingBoxKernel (:78-122).  mm holds [6][nseg] maxima of
// order-preserving integers (minima as the maxima of their complements) and a
// block counter, all zero before the launch and left zero for the next; the last
// block also clears the counters that the rest of the build starts from (a
// memset each would cost as much as a small kernel).
struct ZeroList {
  uint32_t* p[4];
  uint32_t words[4];
};

__device__ __forceinline__ void seg_box(const uint32_t* mm, int nseg, int s, BBox* box,
                                        uint32_t* err) {
  BBox o;
  bool ok = true;
  for (int a = 0; a < 3; ++a) {
    const float mn = float_of(~__ldcg(&mm[a * nseg + s])), mx = float_of(__ldcg(&mm[(3 + a) * nseg + s]));
    o.min[a] = mn;
    o.max[a] = mx;
    ok = ok && isfinite(mn) && isfinite(mx);
    o.inv[a] = __fdiv_rn(1.0f, __fadd_rn(__fsub_rn(mx, mn), 0.001f));
    o.center[a] = __fmul_rn(__fadd_rn(mn, mx), 0.5f);
  }
  const float ex = __fsub_rn(o.max[0], o.min[0]), ey = __fsub_rn(o.max[1], o.min[1]),
              ez = __fsub_rn(o.max[2], o.min[2]);
  float ms = ex;
  if (ms < ey) ms = ey;
  if (ms < ez) ms = ez;
  o.half = __fadd_rn(__fmul_rn(ms, 0.5f), 0.001f);
  o.valid = ok ? 1 : 0;
  if (!ok) raise_error(err, kErrBadInput);
  box[s] = o;
}

__global__ void seg_bounds_kernel(const float4* pm, SegView sv, int64_t n, int nseg,
                                  uint32_t* mm, BBox* box, ZeroList zero, uint32_t* err) {
  chain_begin();
  __shared__ float s_red[32][6];
  __shared__ int s_same;
  __shared__ bool s_last;
  const int64_t c0 = (int64_t)blockIdx.x * blockDim.x * 4;
  const int64_t c1 = imin64(c0 + (int64_t)blockDim.x * 4, n);
  if (threadIdx.x == 0) s_same = nseg == 1 || sv.seg_of[c0] == sv.seg_of[c1 - 1];
  __syncthreads();
  const bool same = s_same;
  float v[6] = {1e30f, 1e30f, 1e30f, -1e30f, -1e30f, -1e30f};
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int s0 = same && nseg > 1 ? sv.seg_of[c0] : 0;
  const int64_t d0 = sv.off[s0] - sv.base[s0];
  float4 body[4];  // (loaded ahead of the first one's atomics)
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int64_t q = c0 + (int64_t)r * blockDim.x + threadIdx.x;
    if (q < c1) body[r] = pm[same ? q + d0 : sv.arena((uint32_t)q)];
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int64_t q = c0 + (int64_t)r * blockDim.x + threadIdx.x;
    if (q < c1) {
      const float4 p = body[r];
      if (same) {
        v[0] = fminf(v[0], p.x);
        v[1] = fminf(v[1], p.y);
        v[2] = fminf(v[2], p.z);
        v[3] = fmaxf(v[3], p.x);
        v[4] = fmaxf(v[4], p.y);
        v[5] = fmaxf(v[5], p.z);
      } else {
        const int s = sv.seg_of[q];
        const float w[6] = {fminf(1e30f, p.x),  fminf(1e30f, p.y),  fminf(1e30f, p.z),
                            fmaxf(-1e30f, p.x), fmaxf(-1e30f, p.y), fmaxf(-1e30f, p.z)};
        for (int a = 0; a < 3; ++a) {
          atomicMax(&mm[a * nseg + s], ~ord_of(w[a]));
          atomicMax(&mm[(3 + a) * nseg + s], ord_of(w[3 + a]));
        }
      }
    }
  }
  if (same) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        v[a] = fminf(v[a], __shfl_down_sync(0xffffffffu, v[a], o));
        v[3 + a] = fmaxf(v[3 + a], __shfl_down_sync(0xffffffffu, v[3 + a], o));
      }
    if (lane == 0)
      for (int a = 0; a < 6; ++a) s_red[warp][a] = v[a];
    __syncthreads();
    if (threadIdx.x < 6) {
      const int a = threadIdx.x;
      float x = s_red[0][a];
      for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
        x = a < 3 ? fminf(x, s_red[w][a]) : fmaxf(x, s_red[w][a]);
      atomicMax(&mm[a * nseg + s0], a < 3 ? ~ord_of(x) : ord_of(x));
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&mm[6 * nseg], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int s = threadIdx.x; s < nseg; s += blockDim.x) seg_box(mm, nseg, s, box, err);
  __syncthreads();
  for (int i = threadIdx.x; i < 6 * nseg + 1; i += blockDim.x) mm[i] = 0;
#pragma unroll
  for (int z = 0; z < 4; ++z)
    for (uint32_t i = threadIdx.x; i < zero.words[z]; i += blockDim.x) zero.p[z][i] = 0;
}

// High path key of every body in concatenated order (values = indices).
__global__ void path_hi_index_kernel(const float4* __restrict__ pm, SegView sv, int64_t n,
                                     u64* __restrict__ hi, uint32_t* __restrict__ idx) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n;
       q += (int64_t)gridDim.x * blockDim.x) {
    u64 h, l;
    path_key(pm[sv.arena((uint32_t)q)], sv.box[sv.seg_of[q]], h, l);
    hi[q] = h;
    idx[q] = (uint32_t)q;
  }
}

__global__ void seg_key_kernel(const uint32_t* __restrict__ idx, const int32_t* __restrict__ seg_of,
                               int64_t n, uint32_t* __restrict__ sk) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x)
    sk[k] = (uint32_t)seg_of[idx[k]];
}

// Final order: segment, high path key and the body itself per position.
__global__ void path_final_kernel(const float4* __restrict__ pm, SegView sv,
                                  const uint32_t* __restrict__ body, int64_t n,
                                  int32_t* __restrict__ kseg, u64* __restrict__ hi,
                                  float4* __restrict__ spm) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t q = body[k];
    const int s = sv.seg_of[q];
    const float4 p = pm[sv.off[s] + ((int64_t)q - sv.base[s])];
    u64 h, l;
    path_key(p, sv.box[s], h, l);
    kseg[k] = s;
    hi[k] = h;
    spm[k] = p;
  }
}

__device__ __forceinline__ u64 low_key(float4 p, const BBox& b) {
  u64 h, l;
  path_key(p, b, h, l);
  return l;
}

// Order inside a run of equal (segment, high key): low key, then Morton key,
// then index.
__device__ __forceinline__ bool tie_less(u64 la, float4 pa, uint32_t a, u64 lc, float4 pc,
                                         uint32_t c, const BBox& b) {
  if (la != lc) return la < lc;
  const uint32_t ma = morton_of(pa, b), mc = morton_of(pc, b);
  if (ma != mc) return ma < mc;
  return a < c;
}

// Runs of equal (segment, high key) -- bodies sharing their first 21
// octants, tiny in practice -- are put in order, and their low keys written
// (nobody reads the low key of a body whose high key differs from its
// neighbours').  Up to kTieRun bodies: insertion-sorted by one thread.  Longer runs
// (a whole system in one such cell, beside a body 2^21 cells away): sorted by
// the block that holds their start, a bitonic network whose comparators all point one
// way, so that places past the end need no entry.  n log^2 n / 256 steps, where one
// thread took n^2 / 4: 3,000 bodies in one run 0.30 ms instead of 787, 100,000 26 ms.
constexpr int kTieThreads = 256;
constexpr int kTieRun = 32;

struct TieRun {
  int64_t first, count;
};

__device__ __noinline__ void tie_sort_run(TieRun t, const BBox& b, uint32_t* body, u64* lo, float4* spm) {
  const int tid = threadIdx.x;
  const int64_t m = t.count;
  body += t.first;
  lo += t.first;
  spm += t.first;
  for (int64_t i = tid; i < m; i += kTieThreads) lo[i] = low_key(spm[i], b);
  __syncthreads();
  auto order = [&](int64_t p, int64_t q) {  // p < q
    if (q >= m || !tie_less(lo[q], spm[q], body[q], lo[p], spm[p], body[p], b)) return;
    const uint32_t u = body[p];
    const u64 l = lo[p];
    const float4 v = spm[p];
    body[p] = body[q];
    lo[p] = lo[q];
    spm[p] = spm[q];
    body[q] = u;
    lo[q] = l;
    spm[q] = v;
  };
  for (int64_t w = 2; w < 2 * m; w <<= 1) {
    // sorted halves of w entries: the first step mirrored, then half cleaners
    for (int64_t i = tid; i < ceil_div(m, w) * (w / 2); i += kTieThreads) {
      const int64_t q = i / (w / 2) * w, o = i % (w / 2);
      order(q + o, q + w - 1 - o);
    }
    __syncthreads();
    for (int64_t h = w / 4; h > 0; h >>= 1) {
      for (int64_t i = tid; i < ceil_div(m, 2 * h) * h; i += kTieThreads) {
        const int64_t q = i / h * (2 * h) + i % h;
        order(q, q + h);
      }
      __syncthreads();
    }
  }
}

__global__ void __launch_bounds__(kTieThreads)
    tie_order_kernel(SegView sv, int64_t n, const int32_t* kseg, const u64* hi, uint32_t* body,
                     u64* lo, float4* spm) {
  chain_begin();
  __shared__ TieRun s_run[kTieThreads / kTieRun + 1];
  __shared__ int s_runs;
  auto same = [&](int64_t i, int64_t j) { return hi[i] == hi[j] && kseg[i] == kseg[j]; };
  for (int64_t k0 = blockIdx.x * (int64_t)kTieThreads; k0 + 1 < n;
       k0 += (int64_t)gridDim.x * kTieThreads) {
    const int64_t k = k0 + threadIdx.x;
    int64_t count = 0;  // of a long run that starts here
    if (k + 1 < n && same(k, k + 1) && !(k > 0 && same(k - 1, k))) {
      int64_t e = k + 1, step = 1;  // the run's last body
      for (; e + step < n && same(k, e + step); step <<= 1) e += step;
      for (; step > 0; step >>= 1)
        if (e + step < n && same(k, e + step)) e += step;
      if (e - k >= kTieRun) {
        count = e - k + 1;
      } else {
        const BBox b = sv.box[kseg[k]];
        lo[k] = low_key(spm[k], b);
        for (int64_t i = k + 1; i <= e; ++i) {
          const uint32_t cur = body[i];
          const float4 pc = spm[i];
          const u64 lc = low_key(pc, b);
          int64_t j = i - 1;
          while (j >= k && tie_less(lc, pc, cur, lo[j], spm[j], body[j], b)) {
            body[j + 1] = body[j];
            spm[j + 1] = spm[j];
            lo[j + 1] = lo[j];
            --j;
          }
          body[j + 1] = cur;
          spm[j + 1] = pc;
          lo[j + 1] = lc;
        }
      }
    }
    if (!__syncthreads_or(count > 0)) continue;
    if (threadIdx.x == 0) s_runs = 0;
    __syncthreads();
    if (count > 0) s_run[atomicAdd(&s_runs, 1)] = TieRun{k, count};
    __syncthreads();
    for (int r = 0; r < s_runs; ++r)
      tie_sort_run(s_run[r], sv.box[kseg[s_run[r].first]], body, lo, spm);
    __syncthreads();
  }
}

// Morton keys scattered back to index order (for the on-demand key sort of a
// single system).
__global__ void morton_scatter_kernel(const float4* __restrict__ spm,
                                      const uint32_t* __restrict__ body, int64_t n,
                                      const BBox* __restrict__ box, uint32_t* __restrict__ keys,
                                      uint32_t* __restrict__ idx) {
  const BBox b = *box;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t i = body[k];
    keys[i] = morton_of(spm[k], b);
    idx[i] = i;
  }
}

// --------------------------------------------- reference-identical tree --
// NBGB_FLAG_REFERENCE_TREE: the reference's host build
// (BarnesHutTree::buildTreeOnHost, force_barnes_hut.cu:391-543) replayed by
// one device thread -- insertion in Morton order, leaf splitting, the node
// budget of 2N (a leaf is no longer split once node_count + 33 >= 2N, later
// bodies merge into it, :449-453), depth-32 merges (:490-507), the
// bottom-up centre of mass in descending node order (:514-538) -- with the
// reference's float operations, then renumbered depth-first into the walk's
// node records.  The canonical device build equals this tree whenever the
// budget does not fire; for small systems (N below about 100) it can fire.
constexpr int64_t kRefTreeMaxBodies = 65536;

struct RefNode {
  float cx, cy, cz, half;
  float comx, comy, comz, mass;
  int32_t child[8];
  int32_t pidx;   // first inserted body (original index), -1 for internal nodes
  int32_t count;  // bodies
  int32_t leaf;
  int32_t size;   // nodes in the subtree (renumbering)
  int32_t minpos; // smallest sorted position of a body in the subtree
};

__device__ void ref_node_default(RefNode& r) {
  r.cx = r.cy = r.cz = r.half = 0.f;
  r.comx = r.comy = r.comz = r.mass = 0.f;
  for (int c = 0; c < 8; ++c) r.child[c] = -1;
  r.pidx = -1;
  r.count = 0;
  r.leaf = 1;
  r.size = 1;
  r.minpos = 0x7fffffff;
}

__device__ __forceinline__ int ref_octant(float x, float y, float z, const RefNode& r) {
  return (x >= r.cx ? 1 : 0) | (y >= r.cy ? 2 : 0) | (z >= r.cz ? 4 : 0);
}

// mergeParticleIntoLeaf (:355-365)
__device__ void ref_merge(RefNode& r, int32_t q, float4 p) {
  const float t = __fadd_rn(r.mass, p.w);
  r.comx = __fdiv_rn(__fadd_rn(__fmul_rn(r.comx, r.mass), __fmul_rn(p.x, p.w)), t);
  r.comy = __fdiv_rn(__fadd_rn(__fmul_rn(r.comy, r.mass), __fmul_rn(p.y, p.w)), t);
  r.comz = __fdiv_rn(__fadd_rn(__fmul_rn(r.comz, r.mass), __fmul_rn(p.z, p.w)), t);
  r.mass = t;
  r.count += 1;
  if (r.pidx < 0) r.pidx = q;
}

// allocateLeaf (:368-389); false when the node array is full
__device__ bool ref_alloc_leaf(RefNode* rn, int64_t max_nodes, int& count, int parent, int oct,
                               int32_t q, float4 p) {
  if ((int64_t)count >= max_nodes) return false;
  const int ni = count++;
  RefNode& pa = rn[parent];
  pa.child[oct] = ni;
  pa.leaf = 0;
  const float hs = __fmul_rn(pa.half, 0.5f);
  RefNode& c = rn[ni];
  ref_node_default(c);
  c.cx = __fadd_rn(pa.cx, (oct & 1) ? hs : -hs);
  c.cy = __fadd_rn(pa.cy, (oct & 2) ? hs : -hs);
  c.cz = __fadd_rn(pa.cz, (oct & 4) ? hs : -hs);
  c.half = hs;
  c.pidx = q;
  c.count = 1;
  c.mass = p.w;
  c.comx = p.x;
  c.comy = p.y;
  c.comz = p.z;
  return true;
}

struct RefTreeArgs {
  const float4* pm;       // bodies by original index (one segment at offset 0)
  const uint32_t* order;  // original indices in (Morton key, index) order
  const uint32_t* body;   // sorted position -> original index
  const BBox* box;
  int64_t n;
  int64_t cap;            // walk node records available
  RefNode* rn;            // 2n reference nodes
  int32_t* pos_of;        // original index -> sorted position
  Node* nodes;
  int32_t* parent;
  uint32_t* nstart;       // nstart[n] = node count (the walk's capacity check)
  uint32_t* scalars;      // [0] node count
  int32_t* seg_root;
  int32_t* seg_end;
  int32_t* seg_depth;
  uint32_t* err;
};

__global__ void ref_tree_kernel(RefTreeArgs a) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  const int64_t n = a.n, max_nodes = 2 * n;  // the reference's max_nodes_ (:253)
  const BBox b = *a.box;
  RefNode* rn = a.rn;
  ref_node_default(rn[0]);
  rn[0].cx = b.center[0];
  rn[0].cy = b.center[1];
  rn[0].cz = b.center[2];
  rn[0].half = b.half;
  rn[0].leaf = 0;
  rn[0].count = (int32_t)n;
  int count = 1, max_depth = 0;
  for (int64_t i = 0; i < n; ++i) {
    const int32_t q = (int32_t)a.order[i];
    const float4 p = a.pm[q];
    int cur = 0, depth = 0;
    bool merged = false;
    while (depth < kMaxDepth) {
      RefNode& nd = rn[cur];
      if (nd.leaf) {
        if ((int64_t)count + kMaxDepth + 1 >= max_nodes) {  // the node budget
          ref_merge(nd, q, p);
          merged = true;
          break;
        }
        const int32_t eq = nd.pidx;
        const float4 ep = make_float4(nd.comx, nd.comy, nd.comz, nd.mass);
        nd.leaf = 0;
        nd.pidx = -1;
        nd.count = 0;
        nd.mass = 0.f;
        nd.comx = nd.comy = nd.comz = 0.f;
        const int eo = ref_octant(ep.x, ep.y, ep.z, nd);
        if (nd.child[eo] < 0 && !ref_alloc_leaf(rn, max_nodes, count, cur, eo, eq, ep)) {
          raise_error(a.err, kErrTreeCapacity);
          return;
        }
      }
      const int oct = ref_octant(p.x, p.y, p.z, rn[cur]);
      const int ch = rn[cur].child[oct];
      if (ch < 0) {
        if (!ref_alloc_leaf(rn, max_nodes, count, cur, oct, q, p)) {
          raise_error(a.err, kErrTreeCapacity);
          return;
        }
        break;
      }
      cur = ch;
      ++depth;
    }
    if (!merged && depth >= kMaxDepth) {  // coincident bodies: merge at depth 32
      int leaf = cur;
      while (!rn[leaf].leaf)
        for (int c = 0; c < 8; ++c)
          if (rn[leaf].child[c] >= 0) {
            leaf = rn[leaf].child[c];
            break;
          }
      ref_merge(rn[leaf], q, p);
    }
    max_depth = max(max_depth, depth);
  }
  if ((int64_t)count > a.cap) {
    raise_error(a.err, kErrTreeCapacity);
    return;
  }
  for (int64_t k = 0; k < n; ++k) a.pos_of[a.body[k]] = (int32_t)k;
  // centre of mass bottom-up (children have larger indices than their
  // parent), with subtree sizes and smallest body positions
  for (int i = count - 1; i >= 0; --i) {
    RefNode& nd = rn[i];
    nd.size = 1;
    if (nd.leaf) {
      nd.minpos = a.pos_of[nd.pidx];
      continue;
    }
    float tm = 0.f, sx = 0.f, sy = 0.f, sz = 0.f;
    int32_t cnt = 0;
    nd.minpos = 0x7fffffff;
    for (int c = 0; c < 8; ++c) {
      const int ci = nd.child[c];
      if (ci < 0) continue;
      const RefNode& ch = rn[ci];
      tm = __fadd_rn(tm, ch.mass);
      sx = __fadd_rn(sx, __fmul_rn(ch.comx, ch.mass));
      sy = __fadd_rn(sy, __fmul_rn(ch.comy, ch.mass));
      sz = __fadd_rn(sz, __fmul_rn(ch.comz, ch.mass));
      cnt += ch.count;
      nd.size += ch.size;
      nd.minpos = min(nd.minpos, ch.minpos);
    }
    nd.mass = tm;
    nd.count = cnt;
    if (tm > 0.f) {
      nd.comx = __fdiv_rn(sx, tm);
      nd.comy = __fdiv_rn(sy, tm);
      nd.comz = __fdiv_rn(sz, tm);
    }
  }
  // depth-first renumbering (octant order), skip = next node after the
  // subtree, next-sibling flags for the walk records
  struct Item {
    int ref, parent, depth, next;
  };
  Item stack[8 * (kMaxDepth + 2)];
  int sp = 0, id = 0;
  stack[sp++] = Item{0, -1, 0, 0};
  while (sp > 0) {
    const Item it = stack[--sp];
    const RefNode& nd = rn[it.ref];
    const int me = id++;
    const int4 info = make_int4(me + nd.size, (it.depth << 8) | (nd.leaf ? 1 : 0),
                                nd.leaf ? a.pos_of[nd.pidx] : nd.minpos, nd.count);
    Node& o = a.nodes[me];
    o.com = make_float4(nd.comx, nd.comy, nd.comz, nd.mass);
    o.geom = make_float4(nd.cx, nd.cy, nd.cz, nd.half);
    o.info = info;
    o.walk = walk_record(info, nd.half, nd.mass, it.next != 0);
    a.parent[me] = it.parent;
    if (nd.leaf) continue;
    int last = -1;
    for (int c = 7; c >= 0; --c)
      if (nd.child[c] >= 0) {
        stack[sp++] = Item{nd.child[c], me, it.depth + 1, last >= 0 ? 1 : 0};
        last = c;
      }
  }
  a.nstart[n] = (uint32_t)count;
  a.scalars[0] = (uint32_t)count;
  a.seg_root[0] = 0;
  a.seg_end[0] = count;
  a.seg_depth[0] = max_depth;
}

static unsigned grid1d(int64_t n, int threads = 256) {
  return (unsigned)std::max<int64_t>(
      1, std::min<int64_t>(ceil_div(std::max<int64_t>(n, 1), threads), (int64_t)num_sms() * 32));
}

// ------------------------------------------------------ host driver --
size_t bh_state_bytes(const BHState* p) {
  if (!p) return 0;
  const BHState& h = *p;
  return h.tables.bytes() + h.seg_of.bytes() + h.seg_minmax.bytes() + h.box.bytes() +
         h.seg_root.bytes() + h.seg_end.bytes() + h.seg_depth.bytes() + h.mkeys.bytes() + h.mkeys_alt.bytes() + h.midx.bytes() +
         h.midx_alt.bytes() + h.klo.bytes() + h.khi.bytes() + h.khi_alt.bytes() +
         h.pidx.bytes() + h.pidx_alt.bytes() + h.sk.bytes() + h.sk_alt.bytes() + h.kseg.bytes() +
         h.psort_ws.bytes() + h.hist.bytes() + h.scan_ws.bytes() + h.lcp.bytes() + h.ncnt.bytes() + h.nstart.bytes() +
         h.scalars.bytes() + h.nodes.bytes() +
         h.node_parent.bytes() +
         h.leaf_of.bytes() + h.ref_nodes.bytes() + h.ref_pos.bytes() + h.spm.bytes() +
         h.walk_ctr.bytes() + h.groups.bytes() + h.groups2.bytes() + h.body_cost.bytes() + h.cost_acc.bytes() +
         h.group_ctr.bytes() + h.group_ovf.bytes();
}

size_t bh_bytes_estimate(int64_t n) { return (size_t)n * 480 + (64u << 10); }

BHState* bh_state_new() { return new BHState(); }

size_t bh_segment_table_bytes(const int64_t* n_per, int nseg) {
  int64_t ntask = 0;
  for (int s = 0; s < nseg; ++s)
    ntask += ceil_div(n_per[s], bh_walk_targets(bh_walk_class(n_per[s])));
  return ((size_t)nseg * 2 + 1) * sizeof(int64_t) + (size_t)ntask * sizeof(WarpTask) +
         ((size_t)nseg + 1) * sizeof(int32_t);
}

// Segment tables -- arena offsets, first concatenated index (prefix sums of
// the sizes) and warp tasks -- go up in one copy; seg_of is derived on the
// device.
void bh_set_segments(BHState& h, const int64_t* off, const int64_t* n_per, int nseg,
                     cudaStream_t st, char* staging) {
  if (nseg < 1) fail(NBGB_ERR_INVALID_ARG, "Validation Error: no Barnes-Hut segment");
  const size_t bytes = bh_segment_table_bytes(n_per, nseg);
  if (!staging) {
    NBGB_CUDA(cudaStreamSynchronize(st));  // the internal staging buffer is reused below
    staging = h.h_tables.ensure(bytes);
  }
  int64_t* hoff = reinterpret_cast<int64_t*>(staging);
  int64_t* hbase = hoff + nseg;
  WarpTask* ht = reinterpret_cast<WarpTask*>(hbase + nseg + 1);
  int64_t t = 0, n = 0;
  for (int s = 0; s < nseg; ++s) {
    if (n_per[s] < 1) fail(NBGB_ERR_INVALID_ARG, "Validation Error: empty Barnes-Hut segment");
    hoff[s] = off[s];
    hbase[s] = n;
    n += n_per[s];
  }
  // the walk's tasks by size class
  for (int cls = 0; cls < kWalkClasses; ++cls) {
    const int tw = bh_walk_targets(cls);
    for (int s = 0; s < nseg; ++s) {
      if (bh_walk_class(n_per[s]) != cls) continue;
      const int64_t end = hbase[s] + n_per[s];
      for (int64_t f = hbase[s]; f < end; f += tw) ht[t++] = WarpTask{f, end, s, 0};
    }
    if (cls < kWalkClasses - 1) h.ntasks_upto[cls] = t;
  }
  h.sort_buckets = path_sort_buckets(n_per, nseg, reinterpret_cast<int32_t*>(ht + t));
  hbase[nseg] = n;
  char* d = grow(h.tables, bytes);
  NBGB_CUDA(cudaMemcpyAsync(d, staging, bytes, cudaMemcpyHostToDevice, st));
  h.nseg = nseg;
  h.ntasks = t;
  h.n = n;
  if (n > h.reserve) h.reserve = std::max(n, h.reserve + h.reserve / 2);
  h.seg_off_p = reinterpret_cast<int64_t*>(d);
  h.seg_base_p = h.seg_off_p + nseg;
  h.tasks_p = reinterpret_cast<WarpTask*>(h.seg_base_p + nseg + 1);
  h.seg_bucket_p = reinterpret_cast<int32_t*>(h.tasks_p + t);
  int32_t* so = grow(h.seg_of, (size_t)h.reserve);
  seg_of_kernel<<<grid1d(n), 256, 0, st>>>(h.seg_base_p, nseg, n, so);
  NBGB_LAUNCH_CHECK();
}

// The bounds kernel's maxima: zero when allocated, and left zero by the kernel.
static uint32_t* seg_minmax_zeroed(BHState& h, cudaStream_t st) {
  const size_t old = h.seg_minmax.cap;
  uint32_t* mm = grow(h.seg_minmax, (size_t)h.nseg * 6 + 1);
  if (h.seg_minmax.cap != old) NBGB_CUDA(cudaMemsetAsync(mm, 0, h.seg_minmax.bytes(), st));
  return mm;
}

// Builds the trees of all segments (positions and masses read from `pm` at
// each segment's offset).
void bh_build(BHState& h, const float4* pm, cudaStream_t st, uint32_t* err, bool groups,
              int group_max, bool ref_tree, StageTimer* timer, uint32_t* total) {
  stage_mark(timer, "barnes_hut.bounds");
  h.built = false;  // until every kernel of this build is enqueued
  h.groups_ready = false;
  h.keys_valid = false;
  const int64_t n = h.n;
  const int nseg = h.nseg;
  const size_t R = (size_t)h.reserve;  // per-body buffers are sized for the reserve
  SegView sv{h.seg_off_p, h.seg_base_p, h.seg_of.ptr, grow(h.box, (size_t)nseg)};
  // 1. per-segment bounds and root cubes
  uint32_t* mm = seg_minmax_zeroed(h, st);
  const ZeroList zero{
      {reinterpret_cast<uint32_t*>(grow(h.psort_ws, path_sort_ws_bytes())),
       reinterpret_cast<uint32_t*>(grow(h.seg_depth, (size_t)nseg + 2)),
       reinterpret_cast<uint32_t*>(grow(h.group_ctr, sizeof(GroupCounters))),
       grow(h.walk_ctr, kWalkLaunches)},
      {h.sort_buckets > 0 ? (uint32_t)path_sort_zero_words() : 0u, (uint32_t)nseg + 2,
       (uint32_t)(sizeof(GroupCounters) / sizeof(uint32_t)), (uint32_t)kWalkLaunches}};
  launch_chained(seg_bounds_kernel, (unsigned)ceil_div(n, 1024), 256, 0, st, pm, sv, n, nseg, mm,
                 h.box.ptr, zero, err);
  // 2. keys and order
  uint32_t* hist = grow(h.hist, radix_hist_elems((int64_t)R));
  uint32_t* sws = grow(h.scan_ws, scan_workspace_elems((int64_t)radix_hist_elems((int64_t)R)) +
                                      scan_workspace_elems((int64_t)R + 1));
  u64* hi = grow(h.khi, R);
  u64* hi2 = grow(h.khi_alt, R);
  u64* lo = grow(h.klo, R);
  uint32_t* pb = grow(h.pidx, R);
  uint32_t* pb2 = grow(h.pidx_alt, R);
  int32_t* kseg = grow(h.kseg, R);
  float4* spm = grow(h.spm, R);
  uint32_t* cnt = grow(h.ncnt, R + 1);
  uint32_t* body = pb;
  if (h.sort_buckets > 0) {
    path_sort(pm, sv, h.seg_bucket_p, h.sort_buckets, n, nseg,
              PathSortBuffers{grow(h.psort_ws, path_sort_ws_bytes()), lo, cnt, hi2, pb2, pb, kseg,
                              hi, spm},
              timer, st);
    stage_mark(timer, "barnes_hut.order");
  } else {
    stage_mark(timer, "barnes_hut.keys");
    path_hi_index_kernel<<<grid1d(n), 256, 0, st>>>(pm, sv, n, hi, pb);
    NBGB_LAUNCH_CHECK();
    stage_mark(timer, "barnes_hut.sort");
    bool alt = false;
    radix_sort_pairs<u64>(hi, hi2, pb, pb2, n, 0, 64, hist, sws, st, &alt, err);
    body = alt ? pb2 : pb;
    uint32_t* body_other = alt ? pb : pb2;
    stage_mark(timer, "barnes_hut.order");
    if (nseg > 1) {
      // stable sort by segment: (segment, path) order
      uint32_t* sk = grow(h.sk, R);
      uint32_t* sk2 = grow(h.sk_alt, R);
      seg_key_kernel<<<grid1d(n), 256, 0, st>>>(body, h.seg_of.ptr, n, sk);
      NBGB_LAUNCH_CHECK();
      int bits = 1;
      while (bits < 31 && (1 << bits) < nseg) ++bits;
      bool alt2 = false;
      radix_sort_pairs<uint32_t>(sk, sk2, body, body_other, n, 0, ((bits + 7) / 8) * 8, hist, sws,
                                 st, &alt2, err);
      if (alt2) std::swap(body, body_other);
    }
    path_final_kernel<<<grid1d(n), 256, 0, st>>>(pm, sv, body, n, kseg, hi, spm);
    NBGB_LAUNCH_CHECK();
  }
  h.body = body;
  launch_chained(tie_order_kernel, grid1d(n), kTieThreads, 0, st, sv, n, kseg, hi, body, lo, spm);
  h.keys_valid = false;  // Morton (key, index) pairs are produced on demand
  if (ref_tree) {
    if (nseg != 1 || n > kRefTreeMaxBodies)
      fail(NBGB_ERR_INVALID_ARG,
           "Validation Error: the reference tree takes one system of at most 65536 bodies");
    // insertion order: the reference's Morton keys, stably sorted (:308-328)
    stage_mark(timer, "barnes_hut.reference_tree");
    uint32_t* mk = grow(h.mkeys, R);
    uint32_t* mi = grow(h.midx, R);
    uint32_t* mk2 = grow(h.mkeys_alt, R);
    uint32_t* mi2 = grow(h.midx_alt, R);
    morton_scatter_kernel<<<grid1d(n), 256, 0, st>>>(spm, body, n, h.box.ptr, mk, mi);
    NBGB_LAUNCH_CHECK();
    radix_sort_pairs<uint32_t>(mk, mk2, mi, mi2, n, 0, 32, hist, sws, st, &h.m_alt, err);
    h.keys_valid = true;
    const int64_t cap_min = 2 * n + 64;
    if (h.cap < cap_min) h.cap = cap_min;
    RefTreeArgs ra;
    ra.pm = pm;
    ra.order = h.m_alt ? mi2 : mi;
    ra.body = body;
    ra.box = h.box.ptr;
    ra.n = n;
    ra.cap = h.cap;
    ra.rn = reinterpret_cast<RefNode*>(grow(h.ref_nodes, (size_t)(2 * n + 1) * sizeof(RefNode)));
    ra.pos_of = grow(h.ref_pos, R);
    ra.nodes = grow(h.nodes, (size_t)h.cap);
    ra.parent = grow(h.node_parent, (size_t)h.cap);
    ra.nstart = grow(h.nstart, R + 1);
    ra.scalars = grow(h.scalars, 2);
    ra.seg_root = grow(h.seg_root, 1);
    ra.seg_end = grow(h.seg_end, 1);
    ra.seg_depth = grow(h.seg_depth, 1);
    ra.err = err;
    ref_tree_kernel<<<1, 1, 0, st>>>(ra);
    NBGB_LAUNCH_CHECK();
    h.groups_ready = false;
    h.built = true;
    return;
  }
  // 3.-5. nodes, groups, centres of mass (bh_nodes.cu)
  bh_nodes(h, groups, group_max, err, timer, total, st);
  h.built = true;
}

// Forces for every segment: acc written at each segment's arena offset.
void bh_walk(BHState& h, const BHWalkParams& p, float* ax, float* ay, float* az, int32_t* counts,
             unsigned long long* inter_total, uint32_t* err, cudaStream_t st) {
  if (p.group_walk)
    bh_group_walk(h, p, ax, ay, az, counts, inter_total, err, st);
  else
    bh_reference_walk(h, p, ax, ay, az, counts, inter_total, st);
}

// Node capacity that any realistic input fits (the canonical tree has ~1.5N
// nodes; 4N + 64 per segment leaves room for strongly clustered sets).  Used
// when there is no per-call synchronization (no read-back to regrow).
// Every buffer a canonical build (and its walk) of the current segment set
// uses, allocated ahead: bh_build then allocates nothing.  The ensemble calls
// this before it changes any state in a tick, so that running out of device
// memory aborts the tick cleanly instead of half-way through a step.
void bh_reserve_buffers(BHState& h, bool groups) {
  const int64_t n = h.n;
  const int nseg = std::max(h.nseg, 1);
  const size_t R = (size_t)h.reserve;
  const int64_t min_cap = 2 * n + 64 * (int64_t)nseg;
  if (h.cap < min_cap) h.cap = 3 * n + 64 * (int64_t)nseg;
  if (h.cap >= kMaxWalkNodes)
    fail(NBGB_ERR_OVERFLOW, "Barnes-Hut node capacity above 2^30 nodes: too many bodies in one tree build");
  grow(h.box, (size_t)nseg);
  {
    // zero for the bounds kernel, complete before any stream of the caller uses it
    const size_t old = h.seg_minmax.cap;
    grow(h.seg_minmax, (size_t)nseg * 6 + 1);
    if (h.seg_minmax.cap != old) {
      NBGB_CUDA(cudaMemset(h.seg_minmax.ptr, 0, h.seg_minmax.bytes()));
      NBGB_CUDA(cudaDeviceSynchronize());
    }
  }
  grow(h.hist, radix_hist_elems((int64_t)R));
  grow(h.scan_ws, scan_workspace_elems((int64_t)radix_hist_elems((int64_t)R)) +
                      scan_workspace_elems((int64_t)R + 1));
  grow(h.khi, R);
  grow(h.khi_alt, R);
  grow(h.klo, R);
  grow(h.pidx, R);
  grow(h.pidx_alt, R);
  grow(h.psort_ws, path_sort_ws_bytes());
  if (nseg > 1 && h.sort_buckets == 0) {
    grow(h.sk, R);
    grow(h.sk_alt, R);
  }
  grow(h.kseg, R);
  grow(h.spm, R);
  grow(h.lcp, lcp_bytes((int64_t)R));
  grow(h.ncnt, R + 1);
  grow(h.nstart, R + 1);
  grow(h.scalars, 2);
  grow(h.seg_depth, (size_t)nseg + 2);
  grow(h.nodes, (size_t)h.cap);
  grow(h.node_parent, (size_t)h.cap);
  grow(h.leaf_of, R);
  grow(h.seg_root, (size_t)nseg);
  grow(h.seg_end, (size_t)nseg);
  grow(h.walk_ctr, kWalkLaunches);
  grow(h.group_ctr, sizeof(GroupCounters));  // (cleared by the bounds kernel with either walk)
  if (groups) {
    grow(h.groups, R);
    h.groups2.ensure(h.groups.cap);
    // fresh cost estimates (zero: no order yet), complete before any stream
    // of the caller uses them
    uint32_t* bc_old = h.body_cost.ptr;
    uint32_t* bc = grow(h.body_cost, R);
    unsigned long long* acc_old = h.cost_acc.ptr;
    unsigned long long* acc = grow(h.cost_acc, 2);
    if (bc != bc_old || acc != acc_old) {
      NBGB_CUDA(cudaMemset(bc, 0, h.body_cost.cap * sizeof(uint32_t)));
      NBGB_CUDA(cudaMemset(acc, 0, 2 * sizeof(unsigned long long)));
      NBGB_CUDA(cudaDeviceSynchronize());
    }
    grow(h.group_ovf, (size_t)kOvfChunks * kOvfChunk);
  }
}

void bh_reserve_async(BHState& h) {
  const int64_t c = 4 * h.reserve + 64 * (int64_t)std::max(h.nseg, 1);
  if (h.cap < c) h.cap = std::max(c, h.cap + h.cap / 2);
}

// The calculator path: one segment at offset 0.
void bh_forces(nbgb_calculator* c, const float4* pm, int64_t n, float* ax, float* ay, float* az) {
  if (!c->bh) c->bh.reset(new BHState());
  BHState& h = *c->bh;
  cudaStream_t st = c->stream;
  uint32_t* err = c->err.ensure(1);
  if (h.nseg != 1 || h.n != n) {
    const int64_t off = 0;
    bh_set_segments(h, &off, &n, 1, st, nullptr);
  }
  const bool sync = (c->params.flags & NBGB_FLAG_SYNC) != 0;
  const bool ref_tree = (c->params.flags & NBGB_FLAG_REFERENCE_TREE) != 0;
  const bool groups = (c->params.flags & NBGB_FLAG_GROUP_WALK) != 0;
  StageTimer* timer = stage_timer(c);
  if (!sync) bh_reserve_async(h);
  const BHWalkParams wp{c->params.G, c->params.softening, c->params.theta, c->params.leaf_capacity,
                        groups ? 1 : 0};
  const bool count = (c->params.flags & NBGB_FLAG_COUNT_INTERACTIONS) != 0;
  int32_t* counts = count ? c->counts.ensure((size_t)n) : nullptr;
  auto walk = [&] {
    stage_mark(timer, "barnes_hut.walk");
    bh_walk(h, wp, ax, ay, az, counts, nullptr, err, st);
  };
  // asynchronously the reference's tree is always replayed; synchronously
  // the canonical tree is built first and replaced only where it can differ
  uint32_t* total = sync ? h.h_scalars.ensure(2) : nullptr;
  bh_build(h, pm, st, err, groups, c->params.group_size, ref_tree && !sync, timer, total);
  if (!sync) {  // capacity overflow surfaces through the device error word
    walk();
    return;
  }
  // The node count is data dependent: the build writes it to mapped host memory,
  // too, and if the capacity was too small the build's later kernels and the walk
  // have skipped their work; then once more with the capacity it takes.  The walk
  // does not wait for the host to look (14 us at 20 K bodies).
  if (!ref_tree) walk();
  NBGB_CUDA(cudaStreamSynchronize(st));
  const int64_t nodes = (int64_t)*(volatile uint32_t*)total;
  if (nodes > h.cap) {
    h.cap = nodes + nodes / 8 + 64;
    bh_build(h, pm, st, err, groups, c->params.group_size, false, timer, total);
    if (!ref_tree) walk();
  }
  // The reference stops splitting once node_count + 33 >= 2N.  Its node
  // count only grows during the insertion and ends at the canonical
  // count when the budget never fires, so a canonical count below
  // 2N - 33 proves that it never fires and the trees are the same.
  if (ref_tree) {
    if (nodes + kMaxDepth + 1 >= 2 * n)
      bh_build(h, pm, st, err, groups, c->params.group_size, true, timer, nullptr);
    walk();
  }
}

// ------------------------------------------------------------- export --
__global__ void export_nodes_kernel(const Node* __restrict__ nodes, const uint32_t* __restrict__ body,
                                    int64_t total, nbgb_octree_node* __restrict__ out) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < total;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int4 in = nodes[p].info;
    const float4 g = nodes[p].geom, cm = nodes[p].com;
    nbgb_octree_node& o = out[p];
    o.center[0] = g.x;
    o.center[1] = g.y;
    o.center[2] = g.z;
    o.half_size = g.w;
    o.center_of_mass[0] = cm.x;
    o.center_of_mass[1] = cm.y;
    o.center_of_mass[2] = cm.z;
    o.total_mass = cm.w;
    o.is_leaf = (uint8_t)(in.y & 1);
    o.pad_[0] = o.pad_[1] = o.pad_[2] = 0;
    o.particle_count = in.w;
    o.particle_index = (in.y & 1) ? (int32_t)body[in.z] : -1;
    for (int j = 0; j < 8; ++j) o.children[j] = -1;
  }
}

__global__ void export_children_kernel(const Node* __restrict__ nodes,
                                       const int32_t* __restrict__ parent,
                                       const u64* __restrict__ hi, const u64* __restrict__ lo,
                                       int64_t total, nbgb_octree_node* __restrict__ out) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < total;
       p += (int64_t)gridDim.x * blockDim.x) {
    if (parent[p] < 0) continue;  // a root
    const int4 in = nodes[p].info;
    const int d = in.y >> 8;
    const int64_t f = in.z;
    const uint32_t oct = (d <= kHiLevels) ? (uint32_t)((hi[f] >> (3 * (kHiLevels - d))) & 7u)
                                          : (uint32_t)((lo[f] >> (3 * (kMaxDepth - d))) & 7u);
    out[parent[p]].children[oct] = (int32_t)p;
  }
}

}  // namespace nbgb

using namespace nbgb;

extern "C" {

nbgb_status nbgb_bh_tree_stats(nbgb_calculator* c, int32_t* node_count, int32_t* max_depth) {
  if (!c || !c->bh || c->method != NBGB_BARNES_HUT || !c->bh->built) return NBGB_ERR_INVALID_ARG;
  BHState& h = *c->bh;
  uint32_t total = 0;
  int32_t depth = 0;
  if (cudaStreamSynchronize(c->stream) != cudaSuccess) return NBGB_ERR_CUDA;
  if (cudaMemcpy(&total, h.scalars.ptr, sizeof total, cudaMemcpyDeviceToHost) != cudaSuccess ||
      cudaMemcpy(&depth, h.seg_depth.ptr, sizeof depth, cudaMemcpyDeviceToHost) != cudaSuccess)
    return NBGB_ERR_CUDA;
  if (node_count) *node_count = (int32_t)total;
  if (max_depth) *max_depth = depth;
  return NBGB_OK;
}

nbgb_status nbgb_bh_copy_sorted_keys(nbgb_calculator* c, uint32_t* keys, int32_t* indices,
                                     size_t n) {
  if (!c || !c->bh || c->method != NBGB_BARNES_HUT || !c->bh->built) return NBGB_ERR_INVALID_ARG;
  BHState& h = *c->bh;
  if (n != (size_t)h.n || h.nseg != 1) return NBGB_ERR_INVALID_ARG;
  if (!h.keys_valid) {
    // The reference's Morton keys and their stable sort
    // (force_barnes_hut.cu:308-328), from the bodies of the last build.
    try {
      const int64_t nn = h.n;
      uint32_t* mk = h.mkeys.ensure((size_t)nn);
      uint32_t* mi = h.midx.ensure((size_t)nn);
      uint32_t* mk2 = h.mkeys_alt.ensure((size_t)nn);
      uint32_t* mi2 = h.midx_alt.ensure((size_t)nn);
      morton_scatter_kernel<<<grid1d(nn), 256, 0, c->stream>>>(h.spm.ptr, h.body, nn, h.box.ptr,
                                                              mk, mi);
      NBGB_LAUNCH_CHECK();
      radix_sort_pairs<uint32_t>(mk, mk2, mi, mi2, nn, 0, 32, h.hist.ptr, h.scan_ws.ptr,
                                 c->stream, &h.m_alt);
      h.keys_valid = true;
    } catch (const Error& e) {
      return e.status;
    }
  }
  if (cudaStreamSynchronize(c->stream) != cudaSuccess) return NBGB_ERR_CUDA;
  const uint32_t* k = h.m_alt ? h.mkeys_alt.ptr : h.mkeys.ptr;
  const uint32_t* v = h.m_alt ? h.midx_alt.ptr : h.midx.ptr;
  if (keys && cudaMemcpy(keys, k, n * 4, cudaMemcpyDeviceToHost) != cudaSuccess)
    return NBGB_ERR_CUDA;
  if (indices && cudaMemcpy(indices, v, n * 4, cudaMemcpyDeviceToHost) != cudaSuccess)
    return NBGB_ERR_CUDA;
  return NBGB_OK;
}

nbgb_status nbgb_bh_copy_nodes(nbgb_calculator* c, nbgb_octree_node* nodes, size_t capacity) {
  if (!c || !c->bh || c->method != NBGB_BARNES_HUT || !nodes || !c->bh->built)
    return NBGB_ERR_INVALID_ARG;
  BHState& h = *c->bh;
  uint32_t total32 = 0;
  if (cudaStreamSynchronize(c->stream) != cudaSuccess) return NBGB_ERR_CUDA;
  if (cudaMemcpy(&total32, h.scalars.ptr, sizeof total32, cudaMemcpyDeviceToHost) != cudaSuccess)
    return NBGB_ERR_CUDA;
  const int64_t total = total32;
  if ((size_t)total > capacity || total > h.cap) return NBGB_ERR_INVALID_ARG;
  nbgb_octree_node* d = nullptr;
  if (cudaMalloc(&d, (size_t)std::max<int64_t>(total, 1) * sizeof(nbgb_octree_node)) != cudaSuccess)
    return NBGB_ERR_OOM;
  unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(total, 256), 4096));
  export_nodes_kernel<<<blocks, 256, 0, c->stream>>>(h.nodes.ptr, h.body, total, d);
  export_children_kernel<<<blocks, 256, 0, c->stream>>>(h.nodes.ptr, h.node_parent.ptr,
                                                        h.khi.ptr, h.klo.ptr, total, d);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e == cudaSuccess)
    e = cudaMemcpy(nodes, d, (size_t)total * sizeof(nbgb_octree_node), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? NBGB_OK : NBGB_ERR_CUDA;
}

nbgb_status nbgb_copy_interaction_counts(nbgb_calculator* c, int32_t* counts, size_t n) {
  if (!c || !counts || c->method == NBGB_DIRECT_N2) return NBGB_ERR_INVALID_ARG;
  if (!(c->params.flags & NBGB_FLAG_COUNT_INTERACTIONS) || !c->counts.ptr ||
      c->counts.cap < n || (int64_t)n != c->last_n)
    return NBGB_ERR_INVALID_ARG;
  if (cudaStreamSynchronize(c->stream) != cudaSuccess) return NBGB_ERR_CUDA;
  return cudaMemcpy(counts, c->counts.ptr, n * 4, cudaMemcpyDeviceToHost) == cudaSuccess
             ? NBGB_OK
             : NBGB_ERR_CUDA;
}

int32_t nbgb_bh_group_size(uint64_t count) {
  return nbgb::bh_group_max(count > (uint64_t)INT64_MAX ? INT64_MAX : (int64_t)count);
}

}  // extern "C"
