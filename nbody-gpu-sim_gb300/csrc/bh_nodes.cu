// bh_nodes.cu -- the octree of sorted bodies: node numbering and records,
// the group walk's groups, bottom-up centres of mass (K4, K5).
//
// l_k = common levels of adjacent sorted keys of one segment (0 across a
// segment boundary); body k starts the internal nodes of depths l_{k-1}+1 ..
// min(l_k, 31) and (unless it shares a depth-32 cell with k-1) one leaf; the
// first body of a segment also starts its root.  An exclusive scan of those
// counts numbers the nodes in depth-first pre-order.  A node of depth d that
// starts at body k ends at the first body e >= k with l_e < d, and the parent
// of the first node that starts at k has depth l_{k-1} and starts after the
// last body i < k with l_i < that depth: both are found in minima of l over
// 32, 1,024, ... bodies, mostly with one 32-byte load (a search over the keys
// took a chain of 2 log2(range) loads, and linking children another chain).
#include <algorithm>

#include "bh_tree.cuh"
#include "kernels.cuh"

namespace nbgb {

// Common levels of sorted bodies i and j (low keys are written, and read, only
// where the high keys agree).
__device__ __forceinline__ int common_levels(const u64* hi, const u64* lo, int64_t i, int64_t j) {
  const u64 h0 = hi[i], h1 = hi[j];
  if (h0 != h1) return (__clzll(h0 ^ h1) - 1) / 3;  // bit 63 unused
  const u64 l0 = lo[i], l1 = lo[j];
  if (l0 != l1) return kHiLevels + (__clzll(l0 ^ l1) - 31) / 3;  // bits 63..33 unused
  return kMaxDepth;
}

// l_k and its minima over 32^1 .. 32^5 bodies, each level padded with zeros to
// whole 32-byte groups.
constexpr int kLcpLevels = 6;
struct LcpTree {
  uint8_t* at[kLcpLevels];
};

static int64_t lcp_level_bytes(int64_t n, int level) {
  for (int i = 0; i < level; ++i) n = ceil_div(n, 32);
  return ceil_div(std::max<int64_t>(n, 1), 32) * 32 + 32;
}

size_t lcp_bytes(int64_t n) {
  int64_t b = 0;
  for (int l = 0; l < kLcpLevels; ++l) b += lcp_level_bytes(n, l);
  return (size_t)b;
}

static LcpTree lcp_tree(uint8_t* base, int64_t n) {
  LcpTree t;
  for (int l = 0; l < kLcpLevels; ++l) {
    t.at[l] = base;
    base += lcp_level_bytes(n, l);
  }
  return t;
}

// Bits of the 32 bytes of group g that are below d.
__device__ __forceinline__ uint32_t below_mask(const uint8_t* level, int64_t g, int d) {
  const uint4* p = reinterpret_cast<const uint4*>(level + g * 32);
  const uint4 a = p[0], b = p[1];
  const uint32_t dd = (uint32_t)d * 0x01010101u;
  const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t lt = __vcmpltu4(w[i], dd) & 0x08040201u;  // one bit per byte, in order
    m |= ((lt | lt >> 8 | lt >> 16 | lt >> 24) & 0xFu) << (4 * i);
  }
  return m;
}

// First j >= k with l_j < d (d >= 1; the last body of a segment has l = 0).
__device__ __forceinline__ int64_t first_below(const LcpTree& t, int64_t k, int d) {
  int64_t i = k;
  int l = 0;
  uint32_t m;
  while (true) {
    m = below_mask(t.at[l], i >> 5, d) & (0xffffffffu << (i & 31));
    if (m || l == kLcpLevels - 1) break;
    i = (i >> 5) + 1;
    ++l;
  }
  while (true) {
    i = (i & ~31ll) + __ffs(m) - 1;
    if (l == 0) return i;
    --l;
    i <<= 5;
    m = below_mask(t.at[l], i >> 5, d);
  }
}

// Last i < k with l_i < d, or -1.
__device__ __forceinline__ int64_t last_below(const LcpTree& t, int64_t k, int d) {
  int64_t i = k - 1;
  int l = 0;
  uint32_t m;
  while (true) {
    if (i < 0) return -1;
    m = below_mask(t.at[l], i >> 5, d) & (0xffffffffu >> (31 - (i & 31)));
    if (m || l == kLcpLevels - 1) break;
    i = (i >> 5) - 1;
    ++l;
  }
  if (!m) return -1;
  while (true) {
    i = (i & ~31ll) + 31 - __clz(m);
    if (l == 0) return i;
    --l;
    i <<= 5;
    m = below_mask(t.at[l], i >> 5, d);
  }
}

constexpr int kNodeBlock = 256;  // bodies per block of the counting and emission kernels

struct NodeArgs {
  const int32_t* kseg;
  const u64* hi;
  const u64* lo;
  LcpTree lcp;
  uint32_t* blk;      // nodes started in each block of bodies, then their prefix
  uint32_t* done;     // blocks counted (zero before)
  uint32_t* nstart;
  uint32_t* total;    // nodes
  uint32_t* total_host;  // the same in mapped host memory (or null)
  const float4* spm;
  const BBox* box;
  const int64_t* base;  // segment s occupies sorted positions [base[s], base[s+1])
  int64_t n;
  int64_t cap;
  Node* nodes;
  int32_t* parent;
  int32_t* seg_root;
  int32_t* seg_end;
  int32_t* seg_depth;
  int32_t* leaf_of;  // per sorted body: the leaf node it starts, or -1
  uint32_t* err;
};

// What body k starts: internal nodes of depths fd .. fd + n_int - 1, a leaf, a root.
struct Starts {
  bool first, last, leaf;
  int lk, lp, fd, n_int;
  __device__ __forceinline__ uint32_t count() const {
    return (uint32_t)n_int + (leaf ? 1u : 0u) + (first ? 1u : 0u);
  }
};

__device__ __forceinline__ Starts starts_of(bool first, bool last, int lk, int lp) {
  Starts s;
  s.first = first;
  s.last = last;
  s.lk = lk;
  s.lp = lp;
  s.fd = first ? 1 : lp + 1;
  const int top = last ? 0 : min(lk, kMaxDepth - 1);
  s.n_int = max(0, top - s.fd + 1);
  s.leaf = first || lp < kMaxDepth;
  return s;
}

__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* s_w, uint32_t* sum) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_w[warp] = x;
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kNodeBlock / 32; ++w) {
    if (w < warp) before += s_w[w];
    all += s_w[w];
  }
  __syncthreads();
  *sum = all;
  return before + x - v;
}

// l_k, its minima over 32 bodies, and the nodes that each block's bodies start;
// the last block turns those into offsets and completes the minima.
__global__ void __launch_bounds__(kNodeBlock) lcp_count_kernel(NodeArgs a) {
  chain_begin();
  __shared__ uint8_t s_l[kNodeBlock + 1];  // l_{k0-1} ..
  __shared__ uint32_t s_w[kNodeBlock / 32];
  __shared__ bool s_last;
  const int tid = threadIdx.x;
  const int64_t k0 = (int64_t)blockIdx.x * kNodeBlock, k = k0 + tid;
  auto level = [&](int64_t i) {  // l_i
    if (i < 0 || i + 1 >= a.n || a.kseg[i + 1] != a.kseg[i]) return 0;
    return common_levels(a.hi, a.lo, i, i + 1);
  };
  const int lk = level(k);
  s_l[tid + 1] = (uint8_t)lk;
  if (tid == 0) s_l[0] = (uint8_t)level(k0 - 1);
  const int g = __reduce_min_sync(0xffffffffu, lk);
  if (k < (a.n + 31) / 32 * 32) a.lcp.at[0][k] = (uint8_t)lk;
  if ((tid & 31) == 0 && k < a.n) a.lcp.at[1][k >> 5] = (uint8_t)g;
  __syncthreads();
  uint32_t c = 0, sum;
  if (k < a.n) {
    const bool first = k == 0 || a.kseg[k - 1] != a.kseg[k];
    const bool last = k + 1 == a.n || a.kseg[k + 1] != a.kseg[k];
    c = starts_of(first, last, lk, first ? 0 : s_l[tid]).count();
  }
  block_scan(c, s_w, &sum);
  if (tid == 0) a.blk[blockIdx.x] = sum;
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(a.done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  uint32_t run = 0;
  for (int64_t b0 = 0; b0 < gridDim.x; b0 += kNodeBlock * 4) {
    uint32_t v[4], t = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int64_t b = b0 + tid * 4 + r;
      v[r] = b < gridDim.x ? __ldcg(&a.blk[b]) : 0u;
      t += v[r];
    }
    uint32_t at = run + block_scan(t, s_w, &sum);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int64_t b = b0 + tid * 4 + r;
      if (b < gridDim.x) a.blk[b] = at;
      at += v[r];
    }
    run += sum;
  }
  if (tid == 0) {
    a.nstart[a.n] = run;
    *a.total = run;
    if (a.total_host) *a.total_host = run;
  }
  // minima over 32^2 .. and the padding of every level
  int64_t m = (a.n + 31) / 32;  // entries of the level below
  for (int l = 2; l < kLcpLevels; ++l) {
    const uint8_t* low = a.lcp.at[l - 1];
    const int64_t pad = (m + 31) / 32 * 32 + 32, up = (m + 31) / 32;
    for (int64_t i = m + tid; i < pad; i += kNodeBlock) a.lcp.at[l - 1][i] = 0;
    __syncthreads();
    for (int64_t i = tid; i < up; i += kNodeBlock) {
      const volatile uint4* p = reinterpret_cast<const volatile uint4*>(low + i * 32);
      uint32_t x = 0xffffffffu;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        x = __vminu4(x, p[h].x);
        x = __vminu4(x, p[h].y);
        x = __vminu4(x, p[h].z);
        x = __vminu4(x, p[h].w);
      }
      x = __vminu4(x, x >> 16);
      x = __vminu4(x, x >> 8);
      a.lcp.at[l][i] = (uint8_t)x;
    }
    __syncthreads();
    m = up;
  }
  for (int64_t i = m + tid; i < (m + 31) / 32 * 32 + 32; i += kNodeBlock)
    a.lcp.at[kLcpLevels - 1][i] = 0;
  const int64_t p0 = (a.n + 31) / 32 * 32;
  if (tid < 32) a.lcp.at[0][p0 + tid] = 0;
}

// Numbers the nodes; writes the leaves and the cubes of the internal nodes that
// a body starts (on the way down to its leaf: every started depth lies above).
// parent[] of a new node holds its body (a leaf: complemented) until
// nodes_kernel has the rest.
__global__ void __launch_bounds__(kNodeBlock) emit_nodes_kernel(NodeArgs a) {
  chain_begin();
  __shared__ uint32_t s_w[kNodeBlock / 32];
  const uint32_t total = a.nstart[a.n];
  if ((int64_t)total > a.cap) {
    // (a host that reads the total builds again; the error word may hold earlier calls' bits)
    if (blockIdx.x == 0 && threadIdx.x == 0 && !a.total_host) raise_error(a.err, kErrTreeCapacity);
    return;
  }
  const int64_t k = (int64_t)blockIdx.x * kNodeBlock + threadIdx.x;
  const bool in = k < a.n;
  Starts st{};
  int32_t s = 0;
  uint32_t sum;
  if (in) {
    s = a.kseg[k];
    const bool first = k == 0 || a.kseg[k - 1] != s, last = k + 1 == a.n || a.kseg[k + 1] != s;
    st = starts_of(first, last, a.lcp.at[0][k], first ? 0 : a.lcp.at[0][k - 1]);
  }
  uint32_t idx = a.blk[blockIdx.x] + block_scan(in ? st.count() : 0u, s_w, &sum);
  if (!in) return;
  a.nstart[k] = idx;
  const float4 p = a.spm[k];
  const BBox b = a.box[s];
  if (st.first) {
    a.nodes[idx].geom = make_float4(b.center[0], b.center[1], b.center[2], b.half);
    a.parent[idx] = (int32_t)k;
    ++idx;
  }
  const uint32_t int0 = idx;
  for (int j = 0; j < st.n_int; ++j) a.parent[idx + j] = (int32_t)k;
  idx += st.n_int;
  int md = -1;
  if (!st.leaf) a.leaf_of[k] = -1;
  if (st.leaf) {
    const int ld = min(kMaxDepth, max(st.lp, st.lk) + 1), top = st.fd + st.n_int - 1;
    float cx = b.center[0], cy = b.center[1], cz = b.center[2], h = b.half;
    for (int lev = 1; lev <= ld; ++lev) {
      const uint32_t o = (p.x >= cx ? 1u : 0u) | (p.y >= cy ? 2u : 0u) | (p.z >= cz ? 4u : 0u);
      const float hs = __fmul_rn(h, 0.5f);
      cx = __fadd_rn(cx, (o & 1u) ? hs : -hs);
      cy = __fadd_rn(cy, (o & 2u) ? hs : -hs);
      cz = __fadd_rn(cz, (o & 4u) ? hs : -hs);
      h = hs;
      if (lev >= st.fd && lev <= top)
        a.nodes[int0 + (lev - st.fd)].geom = make_float4(cx, cy, cz, h);
    }
    int64_t e = k;  // bodies of one depth-32 cell
    if (st.lk >= kMaxDepth) e = first_below(a.lcp, k, kMaxDepth);
    a.nodes[idx].geom = make_float4(cx, cy, cz, h);
    a.nodes[idx].info = make_int4((int)(idx + 1), (ld << 8) | 1, (int)k, (int)(e - k + 1));
    a.parent[idx] = ~(int32_t)k;
    a.leaf_of[k] = (int32_t)idx;
    // reference max_depth_: depth of the inserting body's last loop level
    md = (ld == kMaxDepth && e > k) ? kMaxDepth : ld - 1;
  }
  // per-segment maximum: reduced over the warp where it lies in one segment,
  // one atomic and only while it can still raise the stored value
  const unsigned act = __activemask();
  const int s0 = __shfl_sync(act, s, __ffs(act) - 1);
  if (__all_sync(act, s == s0)) {
    const int m = __reduce_max_sync(act, md);
    if ((int)(threadIdx.x & 31) == __ffs(act) - 1 && m > __ldcg(&a.seg_depth[s]))
      atomicMax(&a.seg_depth[s], m);
  } else if (md > __ldcg(&a.seg_depth[s])) {
    atomicMax(&a.seg_depth[s], md);
  }
}

// One thread per node: the internal nodes' records (range end) and every
// node's parent.
__global__ void nodes_kernel(NodeArgs a) {
  chain_begin();
  const uint32_t total = a.nstart[a.n];
  if ((int64_t)total > a.cap) return;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < (int64_t)total;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int32_t v = a.parent[q];
    const int64_t k = v < 0 ? ~v : v;
    const int32_t s = a.kseg[k];
    const bool first = k == 0 || a.kseg[k - 1] != s;
    const int lp = first ? 0 : a.lcp.at[0][k - 1];
    const int r = (int)(q - (int64_t)a.nstart[k]);  // the body's r-th node
    if (v >= 0) {
      const int d = first ? r : lp + 1 + r;
      const int64_t e = d == 0 ? a.base[s + 1] - 1 : first_below(a.lcp, k, d);
      const uint32_t skip = e + 1 < a.n ? a.nstart[e + 1] : total;
      a.nodes[q].info = make_int4((int)skip, d << 8, (int)k, (int)(e - k + 1));
      if (d == 0) {
        a.seg_root[s] = (int32_t)q;
        a.seg_end[s] = (int32_t)skip;
      }
    }
    // the node above: the body's node before, or the node of depth lp around k
    int32_t up = (int32_t)q - 1;
    if (r == 0) {
      if (first) {
        up = -1;  // the root
      } else if (lp == 0) {
        up = (int32_t)a.nstart[a.base[s]];
      } else {
        const int64_t j = last_below(a.lcp, k, lp) + 1;
        const bool fj = j == 0 || a.kseg[j - 1] != s;
        up = (int32_t)(a.nstart[j] + (uint32_t)(fj ? lp : lp - 1 - a.lcp.at[0][j - 1]));
      }
    }
    a.parent[q] = up;
  }
}

// Where groups_kernel writes the group walk's groups.
struct GroupSink {
  const uint32_t* body;  // path-sorted position -> concatenated body index
  const int32_t* kseg;
  int4* groups;          // first body, count, segment: classes 0 and 1
  int4* groups2;         // classes 2 and 3
  GroupCounters* gc;
  int gmax;              // largest group (32 or 64 bodies)
  int64_t gcap;          // groups capacity
  const uint32_t* body_cost;           // last walk's cost per body
  const unsigned long long* cost_acc;  // last walk's total cost, groups
};

// The group walk's groups: roots with at most gmax bodies; below larger nodes,
// runs of consecutive children with at most gmax bodies in total (merged only
// when the parent holds at most kGroupMergeMax bodies: sibling cells of a
// large sparse node can lie far apart); depth-32 leaves larger than a group
// are split.  Every body belongs to exactly one group, and a group is one
// contiguous range of path-sorted bodies.  Groups go to four cost classes
// (GroupCounters) by the last walk's cost of their first body's group: classes
// 0 and 1 to the front and back of groups, 2 and 3 to those of groups2; the
// walk takes class 0 first, so the longest groups start early and its last
// tasks are short ones.
__global__ void groups_kernel(const Node* nodes, const uint32_t* nstart,
                              int64_t n, int64_t cap, GroupSink gs) {
  chain_begin();
  const uint32_t total = nstart[n];
  if ((int64_t)total > cap) return;
  const int gmax = gs.gmax;
  unsigned long long mean = ~0ull;  // no estimates before the first walk
  if (gs.cost_acc[1]) mean = gs.cost_acc[0] / gs.cost_acc[1];
  auto emit = [&](int f, int c) {
    const unsigned long long e = gs.body_cost[gs.body[f]];
    const int cls = mean == ~0ull ? 3 : (e > 2 * mean ? 0 : (e > mean ? 1 : (2 * e > mean ? 2 : 3)));
    const uint32_t k = atomicAdd(&gs.gc->nclass[cls], 1u);
    int4* arr = cls < 2 ? gs.groups : gs.groups2;
    const int64_t g = (cls & 1) ? gs.gcap - 1 - (int64_t)k : (int64_t)k;
    arr[g] = make_int4(f, c, gs.kseg[f], 0);
  };
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < (int64_t)total;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int4 ip = nodes[p].info;  // skip, depth << 8 | leaf, first, count
    if (ip.w <= gmax) {
      if ((ip.y >> 8) == 0) emit(ip.z, ip.w);  // a small root
      continue;
    }
    if (ip.y & 1) {
      for (int f = 0; f < ip.w; f += gmax) emit(ip.z + f, min(gmax, ip.w - f));
      continue;
    }
    const bool merge = ip.w <= kGroupMergeMax;
    int c = (int)p + 1, gf = 0, gn = 0;
    while (c < ip.x) {
      const int4 ci = nodes[c].info;
      if (ci.w > gmax) {
        if (gn) emit(gf, gn);
        gn = 0;
      } else if (gn && merge && gn + ci.w <= gmax) {
        gn += ci.w;
      } else {
        if (gn) emit(gf, gn);
        gf = ci.z;
        gn = ci.w;
      }
      c = ci.x;
    }
    if (gn) emit(gf, gn);
  }
}

// ------------------------------------------------------ centres of mass --
// Leaves: mass/com as the reference's allocateLeaf + mergeParticleIntoLeaf
// (force_barnes_hut.cu:355-389); then every node from all its children in
// octant order (:514-538).  The chain of levels is long (20 and more around a
// dense core), so what a level costs decides: an arrival counter and a walk
// along the children in global memory take about 3 us per level (65 us in all
// at 20 K bodies, 178 at 1M).  Instead
//   com_kernel      takes 512 consecutive bodies per block; the nodes they start
//                   are consecutive, and those whose subtree lies within them
//                   are summed in shared memory;
//   com_top_kernel  takes the nodes around the edges between those blocks, 32
//                   blocks per CTA; its last CTA the nodes around the edges
//                   between CTAs.  The children are listed ahead, for all nodes
//                   at once, with the centres of mass that are done, so that a level
//                   works in shared memory.
constexpr int kComBodies = 512;  // bodies per block of the centre-of-mass kernel
constexpr int kComSlots = 1280;  // nodes a block holds in shared memory (2.5 per body; about 1.5
                                 // occur)

struct ComArgs {
  Node* nodes;
  const float4* spm;
  const uint32_t* nstart;
  int64_t n;
  int64_t cap;
  const int32_t* parent;
  const int32_t* leaf_of;
  const int32_t* kseg;
  const int64_t* base;
  LcpTree lcp;
  int8_t* inner;    // per block of com_kernel: least l within it
  int group;        // blocks per CTA of com_top_kernel
  int8_t* inner2;   // per CTA of com_top_kernel: least l within its bodies
  uint32_t* done;   // its finished CTAs (zero before)
  unsigned long long* cost_acc;  // cleared: the coming walk adds up its own (or null)
};

// l_k as a node depth: -1 between segments, which share no node.
__device__ __forceinline__ int shared_depth(const ComArgs& a, int64_t k) {
  return a.kseg[k] == a.kseg[k + 1] ? (int)a.lcp.at[0][k] : -1;
}

struct ComSum {
  float m = 0.f, x = 0.f, y = 0.f, z = 0.f;
  __device__ __forceinline__ void add(float4 q) {
    m = __fadd_rn(m, q.w);
    x = __fadd_rn(x, __fmul_rn(q.x, q.w));
    y = __fadd_rn(y, __fmul_rn(q.y, q.w));
    z = __fadd_rn(z, __fmul_rn(q.z, q.w));
  }
  __device__ __forceinline__ float4 com() const {
    float4 r = make_float4(0.f, 0.f, 0.f, m);
    if (m > 0.0f) {
      r.x = __fdiv_rn(x, m);
      r.y = __fdiv_rn(y, m);
      r.z = __fdiv_rn(z, m);
    }
    return r;
  }
};

__device__ __forceinline__ float4 com_of_leaf(const float4* spm, int64_t k, int cnt) {
  const float4 b0 = spm[k];
  float m = b0.w, cx = b0.x, cy = b0.y, cz = b0.z;
  for (int j = 1; j < cnt; ++j) {
    const float4 q = spm[k + j];
    const float t = __fadd_rn(m, q.w);
    cx = __fdiv_rn(__fadd_rn(__fmul_rn(cx, m), __fmul_rn(q.x, q.w)), t);
    cy = __fdiv_rn(__fadd_rn(__fmul_rn(cy, m), __fmul_rn(q.y, q.w)), t);
    cz = __fdiv_rn(__fadd_rn(__fmul_rn(cz, m), __fmul_rn(q.z, q.w)), t);
    m = t;
  }
  return make_float4(cx, cy, cz, m);
}

struct ComShared {
  float4 com[kComSlots];
  int32_t skip[kComSlots], par[kComSlots], cnt[kComSlots], arr[kComSlots];
};

__global__ void __launch_bounds__(kComBodies) com_kernel(ComArgs a) {
  chain_begin();
  __shared__ ComShared s;
  __shared__ int s_min[kComBodies / 32];
  if (a.cost_acc && blockIdx.x == 0 && threadIdx.x < 2) a.cost_acc[threadIdx.x] = 0;
  const uint32_t total = a.nstart[a.n];
  if ((int64_t)total > a.cap) return;
  Node* nodes = a.nodes;
  const int tid = threadIdx.x;
  const int64_t k = (int64_t)blockIdx.x * kComBodies + tid;
  const int64_t k1 = imin64((int64_t)(blockIdx.x + 1) * kComBodies, a.n);
  const int s0 = (int)a.nstart[(int64_t)blockIdx.x * kComBodies];
  const int nall = (int)(k1 < a.n ? a.nstart[k1] : total) - s0, end = s0 + nall;
  const bool fits = nall <= kComSlots;
  {
    const int l = __reduce_min_sync(0xffffffffu, k + 1 < k1 ? shared_depth(a, k) : kMaxDepth);
    if ((tid & 31) == 0) s_min[tid >> 5] = l;
  }
  if (fits)
    for (int i = tid; i < nall; i += kComBodies) {
      const int4 in = nodes[s0 + i].info;
      s.skip[i] = in.x;
      s.cnt[i] = in.w;
      s.par[i] = a.parent[s0 + i];
      s.arr[i] = 0;
    }
  __syncthreads();
  if (tid == 0) {
    int l = s_min[0];
    for (int w = 1; w < kComBodies / 32; ++w) l = min(l, s_min[w]);
    a.inner[blockIdx.x] = (int8_t)l;
  }
  const int p = k < a.n ? a.leaf_of[k] : -1;
  if (!fits) {
    // more nodes than the block holds: level by level in global memory
    if (p >= 0) nodes[p].com = com_of_leaf(a.spm, k, nodes[p].info.w);
    for (int d = kMaxDepth - 1; d >= 0; --d) {
      __syncthreads();
      for (int i = tid; i < nall; i += kComBodies) {
        const int4 in = nodes[s0 + i].info;
        if ((in.y & 1) || (in.y >> 8) != d || in.x > end) continue;
        ComSum sum;
        for (int c = s0 + i + 1; c < in.x; c = nodes[c].info.x) sum.add(__ldcg(&nodes[c].com));
        __stcg(&nodes[s0 + i].com, sum.com());
      }
    }
  } else if (p >= 0) {
    const int li = p - s0;
    s.com[li] = com_of_leaf(a.spm, k, s.cnt[li]);
    int node = s.par[li], cnt = s.cnt[li];
    // up to the first node that reaches beyond the block; the child that
    // completes a node's bodies sums it
    while (node >= s0 && s.skip[node - s0] <= end) {
      const int i = node - s0;
      __threadfence_block();
      if (atomicAdd(&s.arr[i], cnt) + cnt != s.cnt[i]) break;
      __threadfence_block();
      ComSum sum;
      for (int c = i + 1; c < s.skip[i] - s0; c = s.skip[c] - s0) sum.add(s.com[c]);
      s.com[i] = sum.com();
      cnt = s.cnt[i];
      node = s.par[i];
    }
  }
  __syncthreads();
  for (int i = tid; i < nall; i += kComBodies) {
    const int q = s0 + i;
    const int4 in = nodes[q].info;
    if (in.x > end) continue;
    const float4 c = fits ? s.com[i] : __ldcg(&nodes[q].com);
    if (fits) __stcg(&nodes[q].com, c);
    nodes[q].walk = walk_record(in, nodes[q].geom.w, c.w,
                                has_next_sibling(nodes, in.x, a.parent[q]));
  }
}

constexpr int kTopThreads = 512;
constexpr int kTopGroup = 32;    // blocks of com_kernel per CTA; small systems: one CTA
constexpr int kTopSingle = 128;  // for up to this many
constexpr int kTopEdges = 1024;  // edges of one call of com_edges
constexpr int kTopNodes = 1536;  // nodes whose children are listed ahead
constexpr int kTopDone = 6144;   // their children that are summed before

struct TopShared {
  int depth[kTopEdges + 2];  // l at edge e = 1 .. E; 0 and E + 1: the outer edges
  int from[kTopEdges + 2];   // the edge's nodes have depths above this
  int first[kTopEdges + 2];  // their first place in node[], deepest first
  int tmp[kTopEdges + 2];
  int node[kTopNodes];
  int child[kTopNodes][8];   // a place in node[] (summed here), ~place in done[], or kNoChild
  float4 com[kTopNodes];
  float4 done[kTopDone];
  int ndone;
};
constexpr int kNoChild = 0x7fffffff;

// The nodes that contain at least one of E consecutive edges and neither outer
// edge.  Edge e lies before body b0 + e * step; least(u): the least l strictly between
// edges u and u + 1; left, right: l at the outer edges.  A node belongs to the
// first edge it contains: its depth is at most l there, above the least l since
// the edge before (else it would contain that one), and above the least l up to
// the right outer edge.
template <typename Least>
__device__ void com_edges(const ComArgs& a, TopShared& s, int E, int left, int right, int64_t b0,
                          int64_t step, Least least) {
  const int tid = threadIdx.x;
  auto body = [&](int e) { return b0 + e * step; };
  for (int e = tid; e <= E + 1; e += kTopThreads)
    s.depth[e] = e == 0 ? left : e == E + 1 ? right : shared_depth(a, body(e) - 1);
  __syncthreads();
  // least l from edge e to the right outer edge: suffix minima
  for (int e = tid; e <= E; e += kTopThreads) s.from[e] = min((int)least(e), s.depth[e + 1]);
  __syncthreads();
  int* x = s.from;
  int* y = s.tmp;
  for (int o = 1; o <= E; o <<= 1) {
    for (int e = tid; e <= E; e += kTopThreads) y[e] = e + o <= E ? min(x[e], x[e + o]) : x[e];
    __syncthreads();
    int* t = x;
    x = y;
    y = t;
  }
  for (int e = tid + 1; e <= E; e += kTopThreads) {
    const int lo = max(min(s.depth[e - 1], (int)least(e - 1)), x[e]);
    y[e] = lo;
    s.first[e] = max(0, s.depth[e] - lo);
  }
  __syncthreads();
  if (y != s.from)
    for (int e = tid + 1; e <= E; e += kTopThreads) s.from[e] = s.tmp[e];
  __syncthreads();
  // exclusive prefix of the counts
  x = s.first;
  y = s.tmp;
  if (tid == 0) x[0] = y[0] = 0;
  __syncthreads();
  for (int o = 1; o <= E; o <<= 1) {
    for (int e = tid + 1; e <= E; e += kTopThreads) y[e] = e - o >= 1 ? x[e] + x[e - o] : x[e];
    __syncthreads();
    int* t = x;
    x = y;
    y = t;
  }
  const int total = E > 0 ? x[E] : 0;
  for (int e = tid + 1; e <= E; e += kTopThreads) {
    const int c = max(0, s.depth[e] - s.from[e]);
    y[e] = x[e] - c;
  }
  __syncthreads();
  if (y != s.first)
    for (int e = tid + 1; e <= E; e += kTopThreads) s.first[e] = s.tmp[e];
  __syncthreads();
  // the node of depth d at edge e
  auto slot = [&](int e, int d) {
    const int64_t k = body(e) - 1;
    const int sg = a.kseg[k];
    if (d == 0) return (int)a.nstart[a.base[sg]];
    const int64_t j = last_below(a.lcp, k, d) + 1;
    const bool fj = j == 0 || a.kseg[j - 1] != sg;
    return (int)a.nstart[j] + (fj ? d : d - 1 - a.lcp.at[0][j - 1]);
  };
  auto edge_of = [&](int i) {  // last edge whose first place is not above i
    int at = 1, len = E;
    while (len > 1) {
      const int half = len >> 1;
      const bool up = s.first[at + half] <= i;
      at = up ? at + half : at;
      len = up ? len - half : half;
    }
    return at;
  };
  const bool listed = total <= kTopNodes;
  if (tid == 0) s.ndone = 0;
  __syncthreads();
  if (listed)
    for (int i = tid; i < total; i += kTopThreads) {
      const int e = edge_of(i), d = s.depth[e] - (i - s.first[e]), q = slot(e, d);
      s.node[i] = q;
      const int end = a.nodes[q].info.x;
      int c = q + 1, v[8], nd = 0;
#pragma unroll
      for (int o = 0; o < 8; ++o) {
        v[o] = kNoChild;
        if (c < end) {
          const int4 in = a.nodes[c].info;
          // a child with an edge in it is summed here: its first edge's, at depth d + 1
          const uint32_t f = (uint32_t)(in.z - b0) / (uint32_t)step,
                         l = (uint32_t)(in.z - b0 + in.w - 1) / (uint32_t)step;
          v[o] = f == l || (in.y & 1) ? ~c : s.first[f + 1] + s.depth[f + 1] - (d + 1);
          nd += v[o] < 0 ? 1 : 0;
          c = in.x;
        }
      }
      int at = nd ? atomicAdd(&s.ndone, nd) : 0;
      const bool room = at + nd <= kTopDone;
#pragma unroll
      for (int o = 0; o < 8; ++o) {
        int x = v[o];
        if (x < 0 && room) {
          s.done[at] = __ldcg(&a.nodes[~x].com);
          x = ~at++;
        }
        s.child[i][o] = x;
      }
    }
  __syncthreads();
  if (listed && s.ndone <= kTopDone && E <= kTopThreads) {
    // one thread per edge, its nodes deepest first (depth-32 cells are leaves:
    // their places are skipped)
    const int e = tid + 1;
    const bool on = e <= E;
    const int d1 = on ? s.depth[e] : -2, d0 = on ? s.from[e] : 0, i0 = on ? s.first[e] : 0;
    int i = i0 + (d1 == kMaxDepth ? 1 : 0);
    const int last = i0 + (d1 > d0 ? d1 - d0 : 0);
    for (int d = kMaxDepth - 1; d >= 0; --d) {
      if (i < last && d == d1 - (i - i0)) {
        float4 v[8];
        int c[8];
#pragma unroll
        for (int o = 0; o < 8; ++o) {
          c[o] = s.child[i][o];
          if (c[o] != kNoChild) v[o] = c[o] < 0 ? s.done[~c[o]] : s.com[c[o]];
        }
        ComSum sum;
#pragma unroll
        for (int o = 0; o < 8; ++o)
          if (c[o] != kNoChild) sum.add(v[o]);
        const float4 r = sum.com();
        s.com[i] = r;
        __stcg(&a.nodes[s.node[i]].com, r);
        ++i;
      }
      __syncthreads();
    }
  } else {
    for (int d = kMaxDepth - 1; d >= 0; --d) {
      for (int e = tid + 1; e <= E; e += kTopThreads) {
        if (d > s.depth[e] || d <= s.from[e]) continue;
        const int q = slot(e, d), end = a.nodes[q].info.x;
        ComSum sum;
        for (int c = q + 1; c < end; c = a.nodes[c].info.x) sum.add(__ldcg(&a.nodes[c].com));
        __stcg(&a.nodes[q].com, sum.com());
      }
      __syncthreads();
    }
  }
  __syncthreads();
  for (int i = tid; i < total; i += kTopThreads) {
    const int e = edge_of(i);
    const int q = listed ? s.node[i] : slot(e, s.depth[e] - (i - s.first[e]));
    const int4 in = a.nodes[q].info;
    a.nodes[q].walk = walk_record(in, a.nodes[q].geom.w, __ldcg(&a.nodes[q].com).w,
                                  has_next_sibling(a.nodes, in.x, a.parent[q]));
  }
}

__global__ void __launch_bounds__(kTopThreads) com_top_kernel(ComArgs a) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char top_smem[];
  TopShared& s = *reinterpret_cast<TopShared*>(top_smem);
  __shared__ bool s_last;
  if ((int64_t)a.nstart[a.n] > a.cap) return;
  const int64_t step = (int64_t)a.group * kComBodies;  // bodies per CTA
  const int64_t b0 = blockIdx.x * step, b1 = imin64(b0 + step, a.n);
  const int u0 = blockIdx.x * a.group;
  const int E = (int)ceil_div(b1 - b0, kComBodies) - 1;
  const int left = b0 > 0 ? shared_depth(a, b0 - 1) : -1;
  const int right = b1 < a.n ? shared_depth(a, b1 - 1) : -1;
  com_edges(a, s, E, left, right, b0, (int64_t)kComBodies, [&](int u) { return a.inner[u0 + u]; });
  if (gridDim.x == 1) return;
  // the last CTA: the edges between CTAs
  if (threadIdx.x == 0) {
    int l = kMaxDepth;
    for (int u = 0; u <= E; ++u) l = min(l, (int)a.inner[u0 + u]);
    for (int e = 1; e <= E; ++e) l = min(l, s.depth[e]);
    a.inner2[blockIdx.x] = (int8_t)l;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(a.done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  com_edges(a, s, (int)gridDim.x - 1, -1, -1, (int64_t)0, step,
            [&](int u) { return *(volatile int8_t*)&a.inner2[u]; });
}

static unsigned grid1d(int64_t n, int threads = 256) {
  return (unsigned)std::max<int64_t>(
      1, std::min<int64_t>(ceil_div(std::max<int64_t>(n, 1), threads), (int64_t)num_sms() * 32));
}

void bh_nodes(BHState& h, bool groups, int group_max, uint32_t* err, StageTimer* timer,
              uint32_t* total, cudaStream_t st) {
  stage_mark(timer, "barnes_hut.nodes");
  const int64_t n = h.n;
  const int nseg = h.nseg;
  const size_t R = (size_t)h.reserve;
  const int64_t min_cap = 2 * n + 64 * (int64_t)nseg;
  if (h.cap < min_cap) h.cap = 3 * n + 64 * (int64_t)nseg;
  if (h.cap >= kMaxWalkNodes)
    fail(NBGB_ERR_OVERFLOW, "Barnes-Hut node capacity above 2^30 nodes: too many bodies in one tree build");
  NodeArgs a;
  a.kseg = h.kseg.ptr;
  a.hi = h.khi.ptr;
  a.lo = h.klo.ptr;
  a.lcp = lcp_tree(grow(h.lcp, lcp_bytes((int64_t)R)), n);
  a.blk = h.hist.ptr;  // the sort's counters are free by now (n / 2 entries)
  int32_t* depth = grow(h.seg_depth, (size_t)nseg + 2);  // cleared by the bounds kernel
  a.seg_depth = depth;
  a.done = reinterpret_cast<uint32_t*>(depth + nseg);
  a.nstart = grow(h.nstart, R + 1);
  a.total = grow(h.scalars, 2);
  a.total_host = total;
  a.spm = h.spm.ptr;
  a.box = h.box.ptr;
  a.base = h.seg_base_p;
  a.n = n;
  a.cap = h.cap;
  a.nodes = grow(h.nodes, (size_t)h.cap);
  a.parent = grow(h.node_parent, (size_t)h.cap);
  a.seg_root = grow(h.seg_root, (size_t)nseg);
  a.seg_end = grow(h.seg_end, (size_t)nseg);
  a.leaf_of = grow(h.leaf_of, R);
  a.err = err;
  const unsigned blocks = (unsigned)ceil_div(n, kNodeBlock);
  launch_chained(lcp_count_kernel, blocks, kNodeBlock, 0, st, a);
  launch_chained(emit_nodes_kernel, blocks, kNodeBlock, 0, st, a);
  launch_chained(nodes_kernel, grid1d(h.cap), 256, 0, st, a);
  ComArgs c;
  c.cost_acc = nullptr;
  if (groups) {
    h.group_max = group_max > 0 ? group_max : bh_group_max(n);
    uint32_t* bc_old = h.body_cost.ptr;
    uint32_t* bc = grow(h.body_cost, R);
    if (bc != bc_old) NBGB_CUDA(cudaMemsetAsync(bc, 0, h.body_cost.cap * sizeof(uint32_t), st));
    unsigned long long* acc_old = h.cost_acc.ptr;
    unsigned long long* acc = grow(h.cost_acc, 2);
    if (acc != acc_old) NBGB_CUDA(cudaMemsetAsync(acc, 0, 2 * sizeof(unsigned long long), st));
    int4* gr = grow(h.groups, R);
    int4* gr2 = h.groups2.ensure(h.groups.cap);
    GroupSink gs{h.body, h.kseg.ptr, gr, gr2,
                 reinterpret_cast<GroupCounters*>(grow(h.group_ctr, sizeof(GroupCounters))),
                 h.group_max, (int64_t)h.groups.cap, bc, acc};
    launch_chained(groups_kernel, grid1d(h.cap), 256, 0, st, a.nodes, a.nstart, n, h.cap, gs);
    c.cost_acc = acc;
  }
  h.groups_ready = groups;
  stage_mark(timer, "barnes_hut.com");
  c.nodes = a.nodes;
  c.spm = a.spm;
  c.nstart = a.nstart;
  c.n = n;
  c.cap = h.cap;
  c.parent = a.parent;
  c.leaf_of = a.leaf_of;
  c.kseg = a.kseg;
  c.base = a.base;
  c.lcp = a.lcp;
  const int64_t units = ceil_div(n, kComBodies);
  c.group = units <= kTopSingle
                ? (int)units
                : (int)std::max<int64_t>(kTopGroup, ceil_div(units, kTopEdges));
  const int64_t ctas = ceil_div(units, c.group);
  c.inner = reinterpret_cast<int8_t*>(h.hist.ptr);  // the node counts are free by now
  c.inner2 = c.inner + units;
  c.done = a.done + 1;
  launch_chained(com_kernel, (unsigned)units, kComBodies, 0, st, c);
  if (units > 1) {
    NBGB_CUDA(cudaFuncSetAttribute(com_top_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(TopShared)));
    launch_chained(com_top_kernel, (unsigned)ctas, kTopThreads, sizeof(TopShared), st, c);
  }
}

}  // namespace nbgb
