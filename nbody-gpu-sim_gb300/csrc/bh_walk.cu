// bh_walk.cu -- the Barnes-Hut reference walk (K6): every target sums exactly
// the interaction set of the reference's per-target rules
// (force_barnes_hut.cu:142-249).
//
// One warp takes TW path-consecutive targets and tests 32 nodes per step, one
// per lane, against the targets' bounding box.  Most nodes are decided for all
// targets at once: with margins that cover the float rounding of the
// per-target test, a cell is accepted by every target, or opened by every
// target.  Only the nodes in between (and leaves whose cube may hold a target)
// are tested target by target, with the reference's float operations, two
// nodes per packed operation and 32 / TW fours of nodes at a time.  A stack
// item carries the mask of the targets that reach its node; an accepted cell
// or leaf goes to a list with the mask of the targets that take it: one list
// for all targets, one with masks.  Lists are summed 32 entries at a time by
// all lanes in packed FP32x2 (32 / TW lanes per target).
//
// What bounds it: instruction issue (73 % active at 24 warps per SM).  Walking
// the union of 32 targets' paths node by node, all lanes on one node, took 184
// K warp instructions per 32 targets at N = 1M; here a step of 32 nodes, 614 of
// 4,186 nodes tested target by target and two lists of 1,910 entries take half
// of that: 3.4 ms per walk (6.2 before), N = 20 K 0.20 (0.84).
#include <algorithm>
#include <atomic>

#include "bh_tree.cuh"
#include "kernels.cuh"

namespace nbgb {

struct WalkArgs {
  const Node* nodes;
  const float4* spm;
  const uint32_t* body;
  const uint32_t* nstart;
  SegView sv;
  const WarpTask* tasks;  // up to 32 consecutive targets each
  int64_t ntasks;
  const int32_t* seg_root;
  const int32_t* seg_end;
  int64_t n;
  int64_t cap;
  float theta2;
  float th_lo;  // theta2 * (1 - 2^-16)
  float th_hi;  // theta2 * (1 + 2^-16)
  float th_all_lo;  // theta2 * (1 - 2^-18): below it every target accepts
  float th_all_hi;  // theta2 * (1 + 2^-18): above it every target opens
  float eps2;
  float G;
  int leaf_cap;
  int stack_limit;  // stack items before the node-by-node fallback
  float* ax;
  float* ay;
  float* az;
  int32_t* counts;                  // per-body interaction counts (or null)
  unsigned long long* inter_total;  // sum of interactions (or null)
  uint32_t* task_ctr;               // zero before the launch (cleared by the build)
};

// The reference's opening test `size2 / dist2 < theta2` with the correctly
// rounded quotient (force_barnes_hut.cu:222-224), decided by two FP32
// products against thresholds theta2 (1 -+ 2^-16) whenever size2 is not
// within 2^-16 (relative) of theta2 * dist2 -- almost always -- and by the
// IEEE division otherwise.  With |rounding| <= 2^-24 per product, a product
// test that fires implies the exact quotient is below theta2 (1 - 2^-17),
// resp. above theta2 (1 + 2^-17), so the outcome equals the IEEE comparison.
__device__ __forceinline__ bool opening_accept(float size2, float d2, float th_lo, float th_hi,
                                               float theta2) {
  if (size2 < d2 * th_lo) return true;
  if (size2 > d2 * th_hi) return false;
  return __fdiv_rn(size2, d2) < theta2;
}

__device__ __forceinline__ void bh_add(float px, float py, float pz, float m, float xi, float yi,
                                       float zi, float eps2, float& sx, float& sy, float& sz) {
  const float dx = __fsub_rn(px, xi), dy = __fsub_rn(py, yi), dz = __fsub_rn(pz, zi);
  const float d2 = __fadd_rn(__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx))), eps2);
  const float r = rsqrt_approx(d2);
  const float f = (m * r) * (r * r);
  sx = fmaf(f, dx, sx);
  sy = fmaf(f, dy, sy);
  sz = fmaf(f, dz, sz);
}

constexpr int kWWarps = 8;     // warps per block
constexpr int kWStack = 384;   // stack items per warp
constexpr int kWRing = 64;     // entries per list
constexpr int kWMixed = 56;    // a step's mixed nodes: 32 in three groups aligned to 4, and
                               // the last group's reads past its end

struct __align__(16) WalkShared {
  unsigned long long stack[kWStack];  // node | target mask << 32
  float full[4][kWRing];              // entries of all targets: x, y, z, m
  float part[4][kWRing];              // entries of some targets
  uint32_t pmask[kWRing];
  // nodes of a step tested target by target, compacted: centre of mass, size2
  // (a leaf: mass), the cube where it may hold a target, their targets, and
  // the targets found to take the node
  float com[4][kWMixed], geom[4][kWMixed];
  uint32_t imask[kWMixed], take[kWMixed];
};

// Adds entries [base, base + cnt) (cnt a multiple of 4 REP) to the lane's
// target, replica r taking every REP-th four.  MASKED: bit tl of an entry's
// mask decides; the force factor, not the mass, is cleared (a target may sit
// on an entry it does not take).
template <bool MASKED, bool COUNT, int REP>
__device__ __forceinline__ void list_eval(const float (&e)[4][kWRing], const uint32_t* mask,
                                          int base, int cnt, int r, int tl, f2 px, f2 py, f2 pz,
                                          f2 e2, f2& ax, f2& ay, f2& az, int& count) {
  auto pair = [&](unsigned long long x, unsigned long long y, unsigned long long z,
                  unsigned long long m, uint32_t m0, uint32_t m1) {
    const f2 dx = f2_sub(f2{x}, px), dy = f2_sub(f2{y}, py), dz = f2_sub(f2{z}, pz);
    const f2 d2 = f2_fma(dx, dx, f2_fma(dy, dy, f2_fma(dz, dz, e2)));
    float l, h;
    f2_split(d2, l, h);
    const f2 rr = f2_make(rsqrt_approx(l), rsqrt_approx(h));
    f2 f = f2_mul(f2_mul(f2{m}, rr), f2_mul(rr, rr));
    if (MASKED) {
      const bool t0 = (m0 >> tl) & 1u, t1 = (m1 >> tl) & 1u;
      f2_split(f, l, h);
      f = f2_make(t0 ? l : 0.f, t1 ? h : 0.f);
      if (COUNT) count += (t0 ? 1 : 0) + (t1 ? 1 : 0);
    }
    ax = f2_fma(f, dx, ax);
    ay = f2_fma(f, dy, ay);
    az = f2_fma(f, dz, az);
  };
#pragma unroll(MASKED ? 2 : 8 / REP)
  for (int j = base + 4 * r; j < base + cnt; j += 4 * REP) {
    const ulonglong2 X = *reinterpret_cast<const ulonglong2*>(e[0] + j),
                     Y = *reinterpret_cast<const ulonglong2*>(e[1] + j),
                     Z = *reinterpret_cast<const ulonglong2*>(e[2] + j),
                     M = *reinterpret_cast<const ulonglong2*>(e[3] + j);
    uint4 mk = make_uint4(0, 0, 0, 0);
    if (MASKED) mk = *reinterpret_cast<const uint4*>(mask + j);
    pair(X.x, Y.x, Z.x, M.x, mk.x, mk.y);
    pair(X.y, Y.y, Z.y, M.y, mk.z, mk.w);
  }
}

template <bool COUNT, bool BUCKET, int TW>
__global__ void __launch_bounds__(kWWarps * 32, 3) bh_walk_kernel(WalkArgs a) {
  constexpr int REP = 32 / TW;
  constexpr uint32_t kTW = TW == 32 ? 0xffffffffu : (1u << TW) - 1u;
  extern __shared__ __align__(16) unsigned char walk_smem[];
  WalkShared& s = reinterpret_cast<WalkShared*>(walk_smem)[threadIdx.x >> 5];
  const uint32_t total = a.nstart[a.n];
  const bool tree_ok = (int64_t)total <= a.cap;
  const int lane = threadIdx.x & 31, tl = lane & (TW - 1), rr = lane / TW;
  const unsigned all = 0xffffffffu, lt = (1u << lane) - 1u;
  // persistent warps take the next task from a counter
  while (true) {
    uint32_t t32 = 0;
    if (lane == 0) t32 = atomicAdd(a.task_ctr, 1u);
    t32 = __shfl_sync(all, t32, 0);
    if ((int64_t)t32 >= a.ntasks) break;
    const WarpTask task = a.tasks[t32];
    const int64_t first = task.first;
    const int nt = (int)imin64(TW, task.end - first);
    const uint32_t fm = nt == 32 ? 0xffffffffu : (1u << nt) - 1u;  // all targets
    const bool valid = tl < nt;
    const int64_t k = first + (valid ? tl : 0);
    const float4 pi = a.spm[k];
    const f2 px = f2_make(pi.x, pi.x), py = f2_make(pi.y, pi.y), pz = f2_make(pi.z, pi.z);
    const f2 e2 = f2_make(a.eps2, a.eps2);
    // the targets' box: centre and half sizes, the halves widened past rounding
    float bx, by, bz, hx, hy, hz;
    {
      const float lx = float_of(__reduce_min_sync(all, ord_of(pi.x)));
      const float ly = float_of(__reduce_min_sync(all, ord_of(pi.y)));
      const float lz = float_of(__reduce_min_sync(all, ord_of(pi.z)));
      const float ux = float_of(__reduce_max_sync(all, ord_of(pi.x)));
      const float uy = float_of(__reduce_max_sync(all, ord_of(pi.y)));
      const float uz = float_of(__reduce_max_sync(all, ord_of(pi.z)));
      bx = __fmul_rn(__fadd_rn(lx, ux), 0.5f);
      by = __fmul_rn(__fadd_rn(ly, uy), 0.5f);
      bz = __fmul_rn(__fadd_rn(lz, uz), 0.5f);
      hx = __fmul_rn(fmaxf(__fsub_rn(ux, bx), __fsub_rn(bx, lx)), kBoxWiden);
      hy = __fmul_rn(fmaxf(__fsub_rn(uy, by), __fsub_rn(by, ly)), kBoxWiden);
      hz = __fmul_rn(fmaxf(__fsub_rn(uz, bz), __fsub_rn(bz, lz)), kBoxWiden);
      // a NaN position, which the minima and maxima need not show: target by target
      if (__any_sync(all, isnan(pi.x + pi.y + pi.z))) {
        bx = by = bz = 0.f;
        hx = hy = hz = INFINITY;
      }
    }
    f2 ax = f2_make(0.f, 0.f), ay = ax, az = ax;
    float sx = 0.f, sy = 0.f, sz = 0.f;  // single additions
    uint32_t wf = 0, rf = 0, wp = 0, rp = 0;  // list entries written / summed
    int cnt = 0;
    auto sum_full = [&](int c) {
      list_eval<false, false, REP>(s.full, nullptr, (int)(rf & (kWRing - 1)), c, rr, tl, px, py,
                                   pz, e2, ax, ay, az, cnt);
    };
    auto sum_part = [&](int c) {
      list_eval<true, COUNT, REP>(s.part, s.pmask, (int)(rp & (kWRing - 1)), c, rr, tl, px, py,
                                  pz, e2, ax, ay, az, cnt);
    };
    // appends one entry per lane that has one (mask 0: none) and sums full chunks
    auto append = [&](uint32_t mask, float x, float y, float z, float m) {
      const bool f = mask == fm, p = mask != 0 && !f;
      const unsigned bf = __ballot_sync(all, f), bp = __ballot_sync(all, p);
      if (f) {
        const int o = (int)((wf + __popc(bf & lt)) & (kWRing - 1));
        s.full[0][o] = x;
        s.full[1][o] = y;
        s.full[2][o] = z;
        s.full[3][o] = m;
      }
      if (p) {
        const int o = (int)((wp + __popc(bp & lt)) & (kWRing - 1));
        s.part[0][o] = x;
        s.part[1][o] = y;
        s.part[2][o] = z;
        s.part[3][o] = m;
        s.pmask[o] = mask;
      }
      wf += __popc(bf);
      wp += __popc(bp);
      __syncwarp();
      if (wf - rf >= 32) {
        sum_full(32);
        rf += 32;
      }
      if (wp - rp >= 32) {
        sum_part(32);
        rp += 32;
      }
      __syncwarp();
    };
    // per-target rules on one node's record
    auto contains = [&](const float4& g) {
      return fabsf(__fsub_rn(pi.x, g.x)) <= g.w && fabsf(__fsub_rn(pi.y, g.y)) <= g.w &&
             fabsf(__fsub_rn(pi.z, g.z)) <= g.w;
    };
    auto accepts = [&](const float4& cm, float size2) {
      const float dx = __fsub_rn(cm.x, pi.x), dy = __fsub_rn(cm.y, pi.y), dz = __fsub_rn(cm.z, pi.z);
      const float d2 =
          __fadd_rn(__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx))), a.eps2);
      return opening_accept(size2, d2, a.th_lo, a.th_hi, a.theta2);
    };
    // The same rules on four nodes from shared-memory rows (i a multiple of 4),
    // the opening test two per packed operation (each half rounds like the
    // scalar operation).
    auto accepts4 = [&](const float (&c)[4][kWMixed], int i, bool (&t)[4]) {
      const ulonglong2 X = *reinterpret_cast<const ulonglong2*>(&c[0][i]),
                       Y = *reinterpret_cast<const ulonglong2*>(&c[1][i]),
                       Z = *reinterpret_cast<const ulonglong2*>(&c[2][i]);
      const float4 S = *reinterpret_cast<const float4*>(&c[3][i]);
      const f2 tlo = f2_make(a.th_lo, a.th_lo), thi = f2_make(a.th_hi, a.th_hi);
      float d[4], lo[4], hi[4];
      auto two = [&](unsigned long long x, unsigned long long y, unsigned long long z, int q) {
        const f2 dx = f2_sub(f2{x}, px), dy = f2_sub(f2{y}, py), dz = f2_sub(f2{z}, pz);
        const f2 d2 = f2_add(f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx))), e2);
        f2_split(d2, d[q], d[q + 1]);
        f2_split(f2_mul(d2, tlo), lo[q], lo[q + 1]);
        f2_split(f2_mul(d2, thi), hi[q], hi[q + 1]);
      };
      two(X.x, Y.x, Z.x, 0);
      two(X.y, Y.y, Z.y, 2);
      const float z[4] = {S.x, S.y, S.z, S.w};
      bool unsure = false;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        t[q] = z[q] < lo[q];
        unsure = unsure || (!t[q] && !(z[q] > hi[q]));
      }
      if (unsure) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          t[q] = opening_accept(z[q], d[q], a.th_lo, a.th_hi, a.theta2);
      }
    };
    auto contains4 = [&](const float (&g)[4][kWMixed], int i, bool (&in)[4]) {
      const float4 X = *reinterpret_cast<const float4*>(&g[0][i]),
                   Y = *reinterpret_cast<const float4*>(&g[1][i]),
                   Z = *reinterpret_cast<const float4*>(&g[2][i]),
                   H = *reinterpret_cast<const float4*>(&g[3][i]);
      in[0] = contains(make_float4(X.x, Y.x, Z.x, H.x));
      in[1] = contains(make_float4(X.y, Y.y, Z.y, H.y));
      in[2] = contains(make_float4(X.z, Y.z, Z.z, H.z));
      in[3] = contains(make_float4(X.w, Y.w, Z.w, H.w));
    };
    // a leaf whose cube holds the target: the leaf without the target
    // (force_barnes_hut.cu:185-203)
    auto add_rest_of_leaf = [&](const float4& cm) {
      const float me = __fsub_rn(cm.w, pi.w);
      if (me > 0.0f) {
        const float cx = __fdiv_rn(__fsub_rn(__fmul_rn(cm.x, cm.w), __fmul_rn(pi.x, pi.w)), me);
        const float cy = __fdiv_rn(__fsub_rn(__fmul_rn(cm.y, cm.w), __fmul_rn(pi.y, pi.w)), me);
        const float cz = __fdiv_rn(__fsub_rn(__fmul_rn(cm.z, cm.w), __fmul_rn(pi.z, pi.w)), me);
        bh_add(cx, cy, cz, me, pi.x, pi.y, pi.z, a.eps2, sx, sy, sz);
        if (COUNT) ++cnt;
      }
    };
    int sp = tree_ok ? 1 : 0;
    if (lane == 0) s.stack[0] = (unsigned long long)(uint32_t)a.seg_root[task.seg] |
                                ((unsigned long long)fm << 32);
    __syncwarp();
    while (sp > 0) {
      if (sp + 32 > a.stack_limit) {
        // the stack is nearly full: walk the top item's subtree node by node,
        // all targets on one node (no stack); its next sibling stays
        const unsigned long long it = s.stack[sp - 1];
        const uint32_t mask = (uint32_t)(it >> 32);
        int node = (int)(uint32_t)it;
        const int4 w0 = __ldg(&a.nodes[node].walk);
        const int end = w0.x & (int)(kWalkZero - 1u);
        __syncwarp();
        if ((uint32_t)w0.w & kWalkNext) {
          if (lane == 0)
            s.stack[sp - 1] = (unsigned long long)(uint32_t)end | ((unsigned long long)mask << 32);
        } else {
          --sp;
        }
        __syncwarp();
        int resume = (rr == 0 && ((mask >> tl) & 1u)) ? 0 : 0x7fffffff;
        while (node < end) {
          const float4 cm = __ldg(&a.nodes[node].com), g = __ldg(&a.nodes[node].geom);
          const int4 w = __ldg(&a.nodes[node].walk);
          const int skip = w.x & (int)(kWalkZero - 1u);
          const bool act = node >= resume;
          bool open = false;
          if (!((uint32_t)w.x & kWalkZero)) {
            if ((uint32_t)w.x & kWalkLeaf) {
              if (act) {
                if (contains(g)) {
                  add_rest_of_leaf(cm);
                } else {
                  bh_add(cm.x, cm.y, cm.z, cm.w, pi.x, pi.y, pi.z, a.eps2, sx, sy, sz);
                  if (COUNT) ++cnt;
                }
              }
            } else {
              const bool acc = !contains(g) && accepts(cm, __int_as_float(w.y));
              if (act && acc) {
                bh_add(cm.x, cm.y, cm.z, cm.w, pi.x, pi.y, pi.z, a.eps2, sx, sy, sz);
                if (COUNT) ++cnt;
                resume = skip;
              }
              open = act && !acc;
              const int nb = (int)((uint32_t)w.w & ~kWalkNext);
              if (BUCKET && nb <= a.leaf_cap) {
                if (open)
                  for (int j = 0; j < nb; ++j)
                    if (w.z + j != k) {
                      const float4 q = a.spm[w.z + j];
                      bh_add(q.x, q.y, q.z, q.w, pi.x, pi.y, pi.z, a.eps2, sx, sy, sz);
                      if (COUNT) ++cnt;
                    }
                open = false;
              }
            }
          }
          node = __any_sync(all, open) ? node + 1 : skip;
        }
        continue;
      }
      const int m = min(sp, 32);
      sp -= m;
      const bool have = lane < m;
      const unsigned long long it = have ? s.stack[sp + lane] : 0ull;
      const int node = (int)(uint32_t)it;
      const uint32_t mask = (uint32_t)(it >> 32);
      __syncwarp();
      f2 cm_xy = f2_make(0.f, 0.f), cm_zw = cm_xy, g_xy = cm_xy, g_zw = cm_xy;
      int4 w = make_int4((int)kWalkZero, 0, 0, 0);
      if (have) {
        ld_node2(&a.nodes[node], cm_xy, cm_zw, g_xy, g_zw);
        w = __ldg(&a.nodes[node].walk);
      }
      float4 cm, ge;
      f2_split(cm_xy, cm.x, cm.y);
      f2_split(cm_zw, cm.z, cm.w);
      f2_split(g_xy, ge.x, ge.y);
      f2_split(g_zw, ge.z, ge.w);
      const uint32_t wx = (uint32_t)w.x;
      const bool leaf = (wx & kWalkLeaf) != 0;
      const float size2 = __int_as_float(w.y);
      uint32_t em = 0, om = 0;  // targets that take the node / open it
      bool mixed = false, apart = false;
      if (!(wx & kWalkZero)) {
        // Separated along an axis with a relative margin of 2^-20: no target
        // passes the containment test, whatever its rounding.
        constexpr float kSep = 1.0f + 0x1p-20f;
        apart =
            fabsf(__fsub_rn(ge.x, bx)) > __fmul_rn(__fadd_rn(ge.w, hx), kSep) ||
            fabsf(__fsub_rn(ge.y, by)) > __fmul_rn(__fadd_rn(ge.w, hy), kSep) ||
            fabsf(__fsub_rn(ge.z, bz)) > __fmul_rn(__fadd_rn(ge.w, hz), kSep);
        if (leaf) {
          if (apart)
            em = mask;
          else
            mixed = true;
        } else {
          // least and largest distance of the centre of mass from the box,
          // rounded outwards by 2^-22; the 2^-18 margins of th_all_* cover the
          // remaining rounding (some 2^-24 each) of these sums, of the
          // per-target d2 and of the quotient; extreme magnitudes are left to
          // the per-target test
          constexpr float kIn = 1.0f - 0x1p-22f, kOut = 1.0f + 0x1p-22f;
          const float cx = fabsf(__fsub_rn(cm.x, bx)), cy = fabsf(__fsub_rn(cm.y, by)),
                      cz = fabsf(__fsub_rn(cm.z, bz));
          const float nx = fmaxf(__fsub_rn(__fmul_rn(cx, kIn), hx), 0.f),
                      ny = fmaxf(__fsub_rn(__fmul_rn(cy, kIn), hy), 0.f),
                      nz = fmaxf(__fsub_rn(__fmul_rn(cz, kIn), hz), 0.f);
          const float ux = __fmaf_rn(cx, kOut, hx), uy = __fmaf_rn(cy, kOut, hy),
                      uz = __fmaf_rn(cz, kOut, hz);
          const float dmin = __fmaf_rn(nz, nz, __fmaf_rn(ny, ny, __fmaf_rn(nx, nx, a.eps2)));
          const float dmax = __fmaf_rn(uz, uz, __fmaf_rn(uy, uy, __fmaf_rn(ux, ux, a.eps2)));
          // (a NaN centre of mass shows in dmax, not in dmin, and is decided there too)
          const bool every = apart && dmin > 1e-30f && dmax < 1e37f && size2 > 1e-30f &&
                             size2 < __fmul_rn(dmin, a.th_all_lo);
          const bool none = size2 > 1e-30f && dmax < 1e37f && dmax > 1e-30f &&
                            size2 > __fmul_rn(dmax, a.th_all_hi);
          if (every)
            em = mask;
          else if (none)
            om = mask;
          else
            mixed = true;
        }
      }
      // target by target: first the nodes apart from the box (the opening test
      // alone), then those whose cube may hold a target, then such leaves
      const unsigned ba = __ballot_sync(all, mixed && apart);
      const unsigned bc = __ballot_sync(all, mixed && !apart && !leaf);
      const unsigned bl = __ballot_sync(all, mixed && leaf);
      if (ba | bc | bl) {
        const int na = __popc(ba), c0 = (na + 3) & ~3, nc = c0 + __popc(bc), l0 = (nc + 3) & ~3,
                  nl = l0 + __popc(bl);
        int at = 0;
        if (mixed) {
          at = leaf ? l0 + __popc(bl & lt) : apart ? __popc(ba & lt) : c0 + __popc(bc & lt);
          s.com[0][at] = cm.x;
          s.com[1][at] = cm.y;
          s.com[2][at] = cm.z;
          s.com[3][at] = leaf ? cm.w : size2;
          s.imask[at] = mask;
          if (!apart) {
            s.geom[0][at] = ge.x;
            s.geom[1][at] = ge.y;
            s.geom[2][at] = ge.z;
            s.geom[3][at] = ge.w;
          }
        }
        __syncwarp();
        // four nodes per replica at a time; lane l < 4 REP writes node i0 + l
        auto result = [&](int i0, int n, const bool (&t)[4]) {
          unsigned b[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) b[q] = __ballot_sync(all, t[q]);
          const unsigned w = (lane & 2) ? ((lane & 1) ? b[3] : b[2]) : ((lane & 1) ? b[1] : b[0]);
          if (lane < 4 * REP && i0 + lane < n)
            s.take[i0 + lane] = (w >> ((lane >> 2) * TW)) & kTW & s.imask[i0 + lane];
        };
        for (int i0 = 0; i0 < na; i0 += 4 * REP) {
          const int i = i0 + 4 * rr;
          bool t[4];
          accepts4(s.com, i, t);
          result(i0, na, t);
        }
        for (int i0 = c0; i0 < nc; i0 += 4 * REP) {
          const int i = i0 + 4 * rr;
          bool t[4], in[4];
          accepts4(s.com, i, t);
          contains4(s.geom, i, in);
#pragma unroll
          for (int q = 0; q < 4; ++q) t[q] = t[q] && !in[q];
          result(i0, nc, t);
        }
        for (int i0 = l0; i0 < nl; i0 += 4 * REP) {
          const int i = i0 + 4 * rr;
          bool t[4], in[4];
          contains4(s.geom, i, in);
#pragma unroll
          for (int q = 0; q < 4; ++q) t[q] = !in[q];
          result(i0, nl, t);
          if (in[0] || in[1] || in[2] || in[3])
            for (int q = 0; q < 4; ++q)
              if (in[q] && i + q < nl && ((s.imask[i + q] >> tl) & 1u))
                add_rest_of_leaf(make_float4(s.com[0][i + q], s.com[1][i + q], s.com[2][i + q],
                                             s.com[3][i + q]));
        }
        __syncwarp();
        if (mixed) {
          em = s.take[at];
          om = leaf ? 0u : mask & ~em;
        }
      }
      // an opened bucket lists its bodies
      int run = 0;
      const uint32_t run_mask = om;
      if (BUCKET && om && (int)((uint32_t)w.w & ~kWalkNext) <= a.leaf_cap) {
        run = (int)((uint32_t)w.w & ~kWalkNext);
        om = 0;
      }
      // next siblings below first children, so the walk goes depth first
      const bool next = have && ((uint32_t)w.w & kWalkNext);
      const unsigned bs = __ballot_sync(all, next), bo = __ballot_sync(all, om != 0);
      if (next)
        s.stack[sp + __popc(bs & lt)] = (unsigned long long)(wx & (kWalkZero - 1u)) |
                                        ((unsigned long long)mask << 32);
      if (om)
        s.stack[sp + __popc(bs) + __popc(bo & lt)] =
            (unsigned long long)(uint32_t)(node + 1) | ((unsigned long long)om << 32);
      sp += __popc(bs) + __popc(bo);
      if (__any_sync(all, em != 0)) append(em, cm.x, cm.y, cm.z, cm.w);
      if (BUCKET) {
        for (int j = 0; __any_sync(all, j < run); ++j) {
          uint32_t mk = 0;
          float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
          if (j < run) {
            mk = run_mask;
            const int64_t rel = (int64_t)w.z + j - first;  // the target's own body
            if (rel >= 0 && rel < nt) mk &= ~(1u << rel);
            q = a.spm[w.z + j];
          }
          append(mk, q.x, q.y, q.z, q.w);
        }
      }
      __syncwarp();
    }
    // the rest of both lists, padded with massless entries
    {
      const int lf = (int)(wf - rf), pf = (lf + 4 * REP - 1) & ~(4 * REP - 1);
      const int lp = (int)(wp - rp), pp = (lp + 4 * REP - 1) & ~(4 * REP - 1);
      if (lane >= lf && lane < pf) {
        const int o = (int)((rf + lane) & (kWRing - 1));
        s.full[0][o] = 3.0e18f;
        s.full[1][o] = s.full[2][o] = s.full[3][o] = 0.f;
      }
      if (lane >= lp && lane < pp) {
        const int o = (int)((rp + lane) & (kWRing - 1));
        s.part[0][o] = 3.0e18f;
        s.part[1][o] = s.part[2][o] = s.part[3][o] = 0.f;
        s.pmask[o] = 0;
      }
      __syncwarp();
      if (pf) sum_full(pf);
      if (pp) sum_part(pp);
      __syncwarp();
    }
    float lo, hi;
    f2_split(ax, lo, hi);
    sx += lo + hi;
    f2_split(ay, lo, hi);
    sy += lo + hi;
    f2_split(az, lo, hi);
    sz += lo + hi;
#pragma unroll
    for (int o = TW; o < 32; o <<= 1) {
      sx += __shfl_xor_sync(all, sx, o);
      sy += __shfl_xor_sync(all, sy, o);
      sz += __shfl_xor_sync(all, sz, o);
      if (COUNT) cnt += __shfl_xor_sync(all, cnt, o);
    }
    if (COUNT) cnt += (int)wf;
    const bool owner = valid && rr == 0;
    if (owner) {
      const int64_t i = a.sv.arena(a.body[k]);
      a.ax[i] = a.G * sx;
      a.ay[i] = a.G * sy;
      a.az[i] = a.G * sz;
      if (COUNT && a.counts) a.counts[i] = cnt;
    }
    if (COUNT && a.inter_total) {
      unsigned long long c = owner ? (unsigned long long)cnt : 0ull;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(all, c, o);
      if (lane == 0) atomicAdd(a.inter_total, c);
    }
  }
}

// Short walks of large systems (launch_walk has the line): the union of 32 targets'
// paths node by node, all lanes on one node, each with its own target.  No stack,
// no lists and no shared memory, so 48 to 64 warps per SM cover each other's loads;
// a visited node costs 40 instructions whatever the targets decide, which is why long
// walks take half as many the other way.  A short one is bound by the chain of that
// way's steps (first child and next sibling, seven levels of up to eight): 1M bodies in
// a cube at theta 1.5 257 us here, 563 there; at theta 0.5 2,922 and 1,958.
template <bool COUNT, bool BUCKET>
__global__ void __launch_bounds__(256, BUCKET ? 6 : (COUNT ? 7 : 8))
    bh_union_walk_kernel(WalkArgs a) {
  const uint32_t total = a.nstart[a.n];
  const bool tree_ok = (int64_t)total <= a.cap;
  const int lane = threadIdx.x & 31;
  while (true) {
    uint32_t t32 = 0;
    if (lane == 0) t32 = atomicAdd(a.task_ctr, 1u);
    t32 = __shfl_sync(0xffffffffu, t32, 0);
    if ((int64_t)t32 >= a.ntasks) break;
    const WarpTask task = a.tasks[t32];
    const int64_t k = task.first + lane;
    const bool valid = k < task.end;
    const float4 pi = valid ? a.spm[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    const f2 pi_xy = f2_make(pi.x, pi.y);
    float sx = 0.f, sy = 0.f, sz = 0.f;
    int cnt = 0;
    int resume = valid ? 0 : 0x7fffffff;
    int node = tree_ok ? a.seg_root[task.seg] : 0;
    const int node_end = tree_ok ? a.seg_end[task.seg] : 0;
    while (node < node_end) {
      f2 cm_xy, cm_zw, g_xy, g_zw;
      ld_node2(&a.nodes[node], cm_xy, cm_zw, g_xy, g_zw);
      float4 cm, g;
      f2_split(cm_xy, cm.x, cm.y);
      f2_split(cm_zw, cm.z, cm.w);
      f2_split(g_xy, g.x, g.y);
      f2_split(g_zw, g.z, g.w);
      float tx, ty;  // target minus cube centre
      f2_split(f2_sub(pi_xy, g_xy), tx, ty);
      int4 w;  // the body range is for buckets alone
      if (BUCKET) {
        w = __ldg(&a.nodes[node].walk);
      } else {
        const int2 w2 = __ldg(reinterpret_cast<const int2*>(&a.nodes[node].walk));
        w = make_int4(w2.x, w2.y, 0, 0);
      }
      const int skip = w.x & (int)(kWalkZero - 1u);
      if ((uint32_t)w.x >= kWalkZero) {  // a leaf, or without mass
        if ((uint32_t)w.x & kWalkZero) {  // force_barnes_hut.cu:172-173
          node = skip;
          continue;
        }
        if (node >= resume) {  // force_barnes_hut.cu:185-203
          float me = cm.w, cx = cm.x, cy = cm.y, cz = cm.z;
          bool use = true;
          if (fabsf(tx) <= g.w && fabsf(ty) <= g.w && fabsf(__fsub_rn(pi.z, g.z)) <= g.w) {
            me = __fsub_rn(cm.w, pi.w);  // the leaf without the target
            use = me > 0.0f;
            if (use) {
              cx = __fdiv_rn(__fsub_rn(__fmul_rn(cm.x, cm.w), __fmul_rn(pi.x, pi.w)), me);
              cy = __fdiv_rn(__fsub_rn(__fmul_rn(cm.y, cm.w), __fmul_rn(pi.y, pi.w)), me);
              cz = __fdiv_rn(__fsub_rn(__fmul_rn(cm.z, cm.w), __fmul_rn(pi.z, pi.w)), me);
            }
          }
          if (use) {
            bh_add(cx, cy, cz, me, pi.x, pi.y, pi.z, a.eps2, sx, sy, sz);
            if (COUNT) ++cnt;
          }
        }
        node = skip;
        continue;
      }
      // internal node (force_barnes_hut.cu:205-243)
      const bool active = node >= resume;
      const bool contains =
          fabsf(tx) <= g.w && fabsf(ty) <= g.w && fabsf(__fsub_rn(pi.z, g.z)) <= g.w;
      float dx, dy;
      f2_split(f2_sub(cm_xy, pi_xy), dx, dy);
      const float dz = __fsub_rn(cm.z, pi.z);
      const float d2 = __fadd_rn(__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx))), a.eps2);
      const bool accept =
          !contains && opening_accept(__int_as_float(w.y), d2, a.th_lo, a.th_hi, a.theta2);
      const bool open = active && !accept;
      if (active && accept) {
        const float r = rsqrt_approx(d2);
        const float f = (cm.w * r) * (r * r);
        sx = fmaf(f, dx, sx);
        sy = fmaf(f, dy, sy);
        sz = fmaf(f, dz, sz);
        if (COUNT) ++cnt;
        resume = skip;
      }
      if (BUCKET && (int)((uint32_t)w.w & ~kWalkNext) <= a.leaf_cap) {
        // the targets that open a bucket sum its bodies (one broadcast load each)
        if (open) {
          const int64_t self = k - w.z;
          const int nb = (int)((uint32_t)w.w & ~kWalkNext);
          for (int j = 0; j < nb; ++j) {
            const float4 q = __ldg(&a.spm[w.z + j]);
            if (j != self) {
              bh_add(q.x, q.y, q.z, q.w, pi.x, pi.y, pi.z, a.eps2, sx, sy, sz);
              if (COUNT) ++cnt;
            }
          }
        }
        node = skip;
        continue;
      }
      node = __any_sync(0xffffffffu, open) ? node + 1 : skip;
    }
    if (valid) {
      const int64_t i = a.sv.arena(a.body[k]);
      a.ax[i] = a.G * sx;
      a.ay[i] = a.G * sy;
      a.az[i] = a.G * sz;
      if (COUNT && a.counts) a.counts[i] = cnt;
    }
    if (COUNT && a.inter_total) {
      unsigned long long c = valid ? (unsigned long long)cnt : 0ull;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
      if (lane == 0) atomicAdd(a.inter_total, c);
    }
  }
}

// One resident wave of persistent warps on some of the tasks.
// (Not chained: blocks placed beside the build's last ones share SMs while others
// stay empty, forces at 20 K bodies 355 us instead of 293.)
template <typename K>
static void launch_tasks(K kern, int occ, size_t smem, WalkArgs w, const BHState& h, int64_t first,
                         int64_t last, int launch, cudaStream_t st) {
  w.tasks = h.tasks_p + first;
  w.ntasks = last - first;
  w.task_ctr = h.walk_ctr.ptr + launch;
  if (w.ntasks <= 0) return;
  const int64_t blocks = std::max<int64_t>(
      1, std::min<int64_t>(ceil_div(w.ntasks, kWWarps), (int64_t)num_sms() * occ));
  kern<<<(unsigned)blocks, kWWarps * 32, smem, st>>>(w);
  NBGB_LAUNCH_CHECK();
}

template <typename K>
static int walk_occupancy(K kern, size_t smem) {
  int b = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern, kWWarps * 32, smem);
  return std::max(b, 1);
}

template <bool COUNT, bool BUCKET, int TW>
static void launch_walk_t(const WalkArgs& w, const BHState& h, int64_t first, int64_t last,
                          int launch, cudaStream_t st) {
  constexpr size_t smem = sizeof(WalkShared) * kWWarps;
  auto kern = bh_walk_kernel<COUNT, BUCKET, TW>;
  NBGB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  static const int occ = walk_occupancy(kern, smem);
  launch_tasks(kern, occ, smem, w, h, first, last, launch, st);
}

// Sizes from which a short walk goes node by node, and from which it does so at a
// smaller theta.
constexpr int64_t kWalkUnionMin = 196608;
constexpr int64_t kWalkUnionLarge = 1310720;
constexpr int64_t kWalk32MinBodies = 32768;

// Targets per warp for a system of n bodies: 16 give twice as many, shorter
// warps with smaller boxes, which pays while one system alone leaves SMs idle;
// 32 share the traversal.  By the system's own size, so that its sums do not
// depend on what else is walked with it; the line lies below the crossing of a
// system alone (about 60,000 bodies) because many systems walked together fill
// the GPU.  Walk of one system, us (16 / 32 targets): N = 20 K 202 / 261, 50 K
// 299 / 350, 100 K 485 / 441, 1M 4,555 / 3,472.
int bh_walk_class(int64_t n) {
  return n > kWalkUnionLarge ? 0 : n >= kWalkUnionMin ? 1 : n >= kWalk32MinBodies ? 2 : 3;
}

// The walk's time, us, 32 nodes per step / node by node (Plummer sphere; cube):
//   200 K  theta 1.0   290 / 382;   194 / 206    leaf 16  391 / 380;   222 / 190
//          theta 1.25  242 / 250;   163 / 128    leaf 16  303 / 261;   178 / 120
//   1M     theta 1.0  1274 / 1481;  744 / 615    leaf 16 1648 / 1555;  789 / 647
//          theta 1.25 1070 / 955;   629 / 372
//   2M     theta 0.75 3273 / 5036; 1935 / 2081;  theta 1.0 2389 / 2913; 1407 / 1099
//   100 K  theta 1.25  143 / 202;   102 / 115
// Which way is shorter depends on the bodies, too (in a cube the lists are shorter than in
// a sphere): the lines keep the loss against the shorter way below a quarter on both
// sides.  A system's own size and the parameters decide, as above.
template <bool COUNT, bool BUCKET>
static void launch_walk(const BHState& h, const WalkArgs& w, float theta, cudaStream_t st) {
  const int64_t t32 = h.ntasks_upto[2];
  int64_t t = 0;
  if (theta > 0.875f) t = theta > 1.125f || w.leaf_cap > 8 ? h.ntasks_upto[1] : h.ntasks_upto[0];
  if (t > 0) {
    auto kern = bh_union_walk_kernel<COUNT, BUCKET>;
    static const int occ = walk_occupancy(kern, 0);
    launch_tasks(kern, occ, 0, w, h, 0, t, 0, st);
  }
  launch_walk_t<COUNT, BUCKET, 32>(w, h, t, t32, 1, st);
  launch_walk_t<COUNT, BUCKET, 16>(w, h, t32, h.ntasks, 2, st);
}

void bh_reference_walk(BHState& h, const BHWalkParams& p, float* ax, float* ay, float* az,
                       int32_t* counts, unsigned long long* inter_total, cudaStream_t st) {
  WalkArgs w;
  w.nodes = h.nodes.ptr;
  w.spm = h.spm.ptr;
  w.body = h.body;
  w.nstart = h.nstart.ptr;
  w.sv = SegView{h.seg_off_p, h.seg_base_p, h.seg_of.ptr, h.box.ptr};
  w.seg_root = h.seg_root.ptr;
  w.seg_end = h.seg_end.ptr;
  w.n = h.n;
  w.cap = h.cap;
  w.theta2 = p.theta * p.theta;
  w.th_lo = w.theta2 * (1.0f - 0x1p-16f);
  w.th_hi = w.theta2 * (1.0f + 0x1p-16f);
  w.th_all_lo = w.theta2 * (1.0f - 0x1p-18f);
  w.th_all_hi = w.theta2 * (1.0f + 0x1p-18f);
  w.eps2 = p.softening * p.softening;
  w.G = p.G;
  w.leaf_cap = p.leaf_capacity;
  w.stack_limit = std::min(bh_group_stack_limit(), kWStack);
  w.ax = ax;
  w.ay = ay;
  w.az = az;
  w.counts = counts;
  w.inter_total = inter_total;
  const bool count = counts != nullptr || inter_total != nullptr;
  const bool bucket = p.leaf_capacity > 1;
  if (count) {
    if (bucket)
      launch_walk<true, true>(h, w, p.theta, st);
    else
      launch_walk<true, false>(h, w, p.theta, st);
  } else {
    if (bucket)
      launch_walk<false, true>(h, w, p.theta, st);
    else
      launch_walk<false, false>(h, w, p.theta, st);
  }
}

}  // namespace nbgb
