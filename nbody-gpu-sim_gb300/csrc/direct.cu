// direct.cu -- tiled direct-N^2 gravity (K1), packing, energies.
//
// Replaces computeForcesDirectKernel / launchDirectForceKernel
// (src/cuda/force_direct.cu:10-98).  Law: a_i = G * sum_{j != i} m_j d
// (d^2 + eps^2)^-3/2 with d = x_j - x_i.
//
// Layout: sources are read either from the caller's SoA arrays or from a
// packed float4 (x, y, z, m) array and staged in shared memory as x, y, z and
// m rows, so that two consecutive sources arrive as the two halves of a
// packed FP32x2 operand (direct_pair.cuh).  With eps > 0 the j == i term is
// exactly 0 (d = 0), so the inner loop has no self test.
//
// Accumulation: per target and j-tile slice (at most 256 sources), two plain
// FP32 partial sums (even and odd sources); their sum is folded into a
// running (sum, error) pair with an error-free two-sum.  COMP = false adds
// the slices' sums in plain FP32.
#include "common.cuh"
#include "kernels.cuh"
#include "direct_core.cuh"
#include "direct_pair.cuh"

namespace nbgb {

// ---------------------------------------------------------------------------
// Packing: SoA (pos_x, pos_y, pos_z, mass) -> float4 (x, y, z, m), zero pad.
// ---------------------------------------------------------------------------
__global__ void pack_soa_kernel(const float* __restrict__ x, const float* __restrict__ y,
                                const float* __restrict__ z, const float* __restrict__ m,
                                int64_t n, int64_t n_pad, float4* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_pad;
       i += (int64_t)gridDim.x * blockDim.x) {
    out[i] = (i < n) ? make_float4(x[i], y[i], z[i], m[i]) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

void launch_pack_soa(const float* x, const float* y, const float* z, const float* m, int64_t n,
                     int64_t n_pad, float4* out, cudaStream_t st) {
  if (n_pad <= 0) return;
  int threads = 256;
  int64_t blocks = std::min<int64_t>(ceil_div(n_pad, threads), (int64_t)num_sms() * 8);
  pack_soa_kernel<<<(unsigned)blocks, threads, 0, st>>>(x, y, z, m, n, n_pad, out);
  NBGB_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// The direct kernel.  A CTA owns 128*I targets (blockIdx.x) and a run of
// a.jper sources (blockIdx.y); its two halves of 128 threads sum the two
// halves of every 512-source tile for the same targets and are added up in
// shared memory.  With more than one run the last CTA of a target block to
// finish adds the runs' partial sums in run order (deterministic), so no
// second launch is needed.
//
// What bounds it: the FP32 pipe (12 lane operations per interaction) once
// every SM has two CTAs, launch and memory latency below about 4,000 bodies.
// Pairing sources instead of targets leaves no operand duplication in the
// inner loop; splitting the sources over CTAs fills the GPU at every size
// (one CTA per 1,024 targets without a split before: N = 1,024 took 66 us).
// ---------------------------------------------------------------------------
template <bool SOA>
__device__ __forceinline__ float4 load_body(const DirectArgs& a, int64_t i) {
  if (SOA) return make_float4(a.sx[i], a.sy[i], a.sz[i], a.sm[i]);
  return a.src[i];
}

template <int I, bool COMP, bool ZERO_SOFT, bool SOA>
__global__ void __launch_bounds__(kDirThreads, 2) direct_kernel(DirectArgs a) {
  constexpr int T = kDirHalf * I;
  __shared__ __align__(16) float s_t[2][4][kDirTile];
  __shared__ bool s_last;
  const int tid = threadIdx.x, half = tid / kDirHalf, tl = tid % kDirHalf;
  const int64_t tgt_base = (int64_t)blockIdx.x * T;
  const int64_t j0 = (int64_t)blockIdx.y * a.jper, j1 = imin64(j0 + a.jper, a.n_src);
  const int nt = (int)ceil_div(j1 - j0, kDirTile);

  f2 xi[I], yi[I], zi[I];
  float sx[I], sy[I], sz[I], ex[I], ey[I], ez[I];
#pragma unroll
  for (int q = 0; q < I; ++q) {
    const int64_t i = tgt_base + tl + q * kDirHalf;
    const float4 p = (i < a.n_tgt) ? load_body<SOA>(a, i) : make_float4(0.f, 0.f, 0.f, 0.f);
    xi[q] = f2_make(p.x, p.x);
    yi[q] = f2_make(p.y, p.y);
    zi[q] = f2_make(p.z, p.z);
    sx[q] = sy[q] = sz[q] = ex[q] = ey[q] = ez[q] = 0.f;
  }
  // the next tile is on its way to registers while the current one is summed
  float4 v[kDirTile / kDirThreads];
  auto fetch = [&](int t) {
#pragma unroll
    for (int r = 0; r < kDirTile / kDirThreads; ++r) {
      const int64_t j = j0 + (int64_t)t * kDirTile + r * kDirThreads + tid;
      v[r] = (j < j1) ? load_body<SOA>(a, j) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto stage = [&](int b) {
#pragma unroll
    for (int r = 0; r < kDirTile / kDirThreads; ++r) {
      s_t[b][0][r * kDirThreads + tid] = v[r].x;
      s_t[b][1][r * kDirThreads + tid] = v[r].y;
      s_t[b][2][r * kDirThreads + tid] = v[r].z;
      s_t[b][3][r * kDirThreads + tid] = v[r].w;
    }
  };
  fetch(0);
  stage(0);
  __syncthreads();
  const f2 e2 = f2_make(a.eps2, a.eps2);
  for (int t = 0; t < nt; ++t) {
    if (t + 1 < nt) fetch(t + 1);
    // this half's share of the tile, in whole steps of 8 (zero mass past the end)
    const int cnt = (int)imin64(kDirTile, j1 - j0 - (int64_t)t * kDirTile);
    const int mid = ((cnt + 1) / 2 + 7) & ~7;
    const int jb = half ? mid : 0, je = half ? ((cnt + 7) & ~7) : mid;
    f2 ax[I], ay[I], az[I];
#pragma unroll
    for (int q = 0; q < I; ++q) ax[q] = ay[q] = az[q] = f2_make(0.f, 0.f);
    pair_sum<I, ZERO_SOFT>(s_t[t & 1], jb, je, xi, yi, zi, e2, ax, ay, az);
#pragma unroll
    for (int q = 0; q < I; ++q) {
      fold<COMP>(f2_sum(ax[q]), sx[q], ex[q]);
      fold<COMP>(f2_sum(ay[q]), sy[q], ey[q]);
      fold<COMP>(f2_sum(az[q]), sz[q], ez[q]);
    }
    if (t + 1 < nt) stage((t + 1) & 1);
    __syncthreads();
  }
  // add the second half's sums to the first's
  float* s_r = &s_t[0][0][0];  // 6 rows of T floats (I = 2: 6 of the 16 KB)
  static_assert(6 * T <= 2 * 4 * kDirTile, "reduction rows fit the tile buffers");
  if (half) {
#pragma unroll
    for (int q = 0; q < I; ++q) {
      const int o = tl + q * kDirHalf;
      s_r[o] = sx[q];
      s_r[T + o] = sy[q];
      s_r[2 * T + o] = sz[q];
      s_r[3 * T + o] = ex[q];
      s_r[4 * T + o] = ey[q];
      s_r[5 * T + o] = ez[q];
    }
  }
  __syncthreads();
  if (!half) {
#pragma unroll
    for (int q = 0; q < I; ++q) {
      const int o = tl + q * kDirHalf;
      const int64_t i = tgt_base + o;
      fold<COMP>(s_r[o], sx[q], ex[q]);
      fold<COMP>(s_r[T + o], sy[q], ey[q]);
      fold<COMP>(s_r[2 * T + o], sz[q], ez[q]);
      const float rx = sx[q] + (ex[q] + s_r[3 * T + o]), ry = sy[q] + (ey[q] + s_r[4 * T + o]),
                  rz = sz[q] + (ez[q] + s_r[5 * T + o]);
      if (a.splits > 1) {
        a.partial[(int64_t)blockIdx.y * a.n_tgt_pad + i] = make_float4(rx, ry, rz, 0.f);
      } else if (i < a.n_tgt) {
        a.out_x[i] = a.G * rx;
        a.out_y[i] = a.G * ry;
        a.out_z[i] = a.G * rz;
      }
    }
  }
  if (a.splits == 1) return;
  // the last CTA of this target block adds the partial sums
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(&a.ticket[blockIdx.x], 1u) == (uint32_t)(a.splits - 1);
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (tid == 0) a.ticket[blockIdx.x] = 0;  // ready for the next launch
  for (int o = tid; o < T; o += kDirThreads) {
    const int64_t i = tgt_base + o;
    if (i >= a.n_tgt) break;
    float rx = 0.f, ry = 0.f, rz = 0.f, fx = 0.f, fy = 0.f, fz = 0.f;
#pragma unroll 4
    for (int s = 0; s < a.splits; ++s) {
      const float4 p = __ldcg(&a.partial[(int64_t)s * a.n_tgt_pad + i]);
      fold<true>(p.x, rx, fx);
      fold<true>(p.y, ry, fy);
      fold<true>(p.z, rz, fz);
    }
    a.out_x[i] = a.G * (rx + fx);
    a.out_y[i] = a.G * (ry + fy);
    a.out_z[i] = a.G * (rz + fz);
  }
}

// The largest systems: one CTA of 128 threads sums 8 targets per thread, two per
// packed operation, against 256-source tiles that the bulk-copy engine streams
// in (direct_core.cuh, the ensembles' engine; sources padded to whole tiles).  Its
// long inner loop without block barriers sustains up to 2 % more than the kernel
// above (350,000 bodies 44.0 against 44.5 ms, 1M 391.5 against 401), but its blocks of
// 1,024 targets and whole tiles split unevenly below (65,536 bodies 1.65 against
// 1.58 ms, 131,072 6.38 against 6.30; plan_direct has the line).
template <bool COMP, bool ZERO_SOFT>
__global__ void __launch_bounds__(kDirHalf) direct_ring_kernel(DirectArgs a) {
  constexpr int I = 8;
  __shared__ alignas(128) float4 s_j[kRingStages][kRingTile];
  __shared__ alignas(8) uint64_t s_bar[kRingStages];
  TileRing ring{s_j, s_bar, 0};
  ring_init(ring);
  const int tid = threadIdx.x;
  const int64_t tgt_base = (int64_t)blockIdx.x * (kDirHalf * I);
  const int64_t tile0 = (int64_t)blockIdx.y * (a.jper / kRingTile);
  const int64_t tile1 = imin64(tile0 + a.jper / kRingTile, a.n_src / kRingTile);
  const int nt = (int)imax64(tile1 - tile0, 0);
  float xi[I], yi[I], zi[I];
#pragma unroll
  for (int q = 0; q < I; ++q) {
    const int64_t i = tgt_base + tid + (int64_t)q * kDirHalf;
    const float4 p = (i < a.n_tgt) ? a.src[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    xi[q] = p.x;
    yi[q] = p.y;
    zi[q] = p.z;
  }
  float sx[I], sy[I], sz[I];
  if (!direct_tiles<kDirHalf, I, true, COMP, ZERO_SOFT>(ring, a.src + tile0 * kRingTile, nt, xi, yi,
                                                        zi, a.eps2, sx, sy, sz, a.err))
    return;
#pragma unroll
  for (int q = 0; q < I; ++q) {
    const int64_t i = tgt_base + tid + (int64_t)q * kDirHalf;
    if (i >= a.n_tgt) continue;
    if (a.splits > 1) {
      a.partial[(int64_t)blockIdx.y * a.n_tgt_pad + i] = make_float4(sx[q], sy[q], sz[q], 0.f);
    } else {
      a.out_x[i] = a.G * sx[q];
      a.out_y[i] = a.G * sy[q];
      a.out_z[i] = a.G * sz[q];
    }
  }
}

// Adds the ring kernel's runs in run order.
__global__ void direct_runs_kernel(DirectArgs a) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.n_tgt;
       i += (int64_t)gridDim.x * blockDim.x) {
    float rx = 0.f, ry = 0.f, rz = 0.f, fx = 0.f, fy = 0.f, fz = 0.f;
    for (int s = 0; s < a.splits; ++s) {
      const float4 p = a.partial[(int64_t)s * a.n_tgt_pad + i];
      fold<true>(p.x, rx, fx);
      fold<true>(p.y, ry, fy);
      fold<true>(p.z, rz, fz);
    }
    a.out_x[i] = a.G * (rx + fx);
    a.out_y[i] = a.G * (ry + fy);
    a.out_z[i] = a.G * (rz + fz);
  }
}

// Targets per thread and source runs for n bodies: the pair with the least
// estimated time, in SM clocks.  The busiest SM sums k CTAs at 8.65 (one
// target per thread) or 8.95 interactions per clock together, 7.9 when it has
// only one (81, 84 and 74 % of its 128 lanes / 12 operations); each round of resident CTAs costs kCtaClocks
// to start (targets, first tile, half sums), and each run a load per target
// at the end.  Measured, us per launch: N = 5,000 16.5 (two targets per thread,
// 15 runs; 42 with one target, unsplit), N = 16,384 107 (two, 19 runs; 130
// with one target, unsplit), N = 131,072 6,262 (two, 19 runs; 6,417 with
// one); four targets per thread were nowhere faster (6,333 at N = 131,072).
// Small systems go to steps.cu.  The ring kernel takes those from kDirRingMin bodies
// on, and from kDirRingFit on where whole waves of its CTAs keep the SMs busy for 98.5 %
// of the time: its rate per busy SM is 1.6 % higher, its waves are coarser.  us, ring
// against direct_kernel: N = 262,144 (97.8 % busy) 24,993 / 24,910, 265,000 (99.2)
// 25,294 / 25,481, 270,000 (99.0) 26,191 / 26,708, 275,000 (98.1) 27,626 / 27,392,
// 280,000 (95.8) 29,119 / 28,563, 285,000 (97.1) 29,658 / 29,429, 290,000 (99.1)
// 30,195 / 30,645, 294,911 (99.0) 31,196 / 31,812.
constexpr int64_t kDirRingFit = 262144;
constexpr int64_t kDirRingMin = 294912;
constexpr double kDirRingBusy = 0.985;

// The ring kernel's plan for n bodies: runs so that the CTAs fill whole waves.
// `busy`: the part of its waves' time that is spent on the n^2 interactions.
static DirectPlan plan_ring(int64_t n, int max_splits, double* busy) {
  static const int occ = [] {
    int b = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, direct_ring_kernel<true, false>, kDirHalf, 0);
    return std::max(b, 1);
  }();
  constexpr int64_t T = (int64_t)kDirHalf * 8;
  const int64_t slots = (int64_t)num_sms() * occ;
  DirectPlan p;
  p.ring = true;
  p.per_thread = 8;
  p.i_blocks = ceil_div(n, T);
  p.n_tgt_pad = p.i_blocks * T;
  const int64_t tiles = ceil_div(n, (int64_t)kRingTile);
  double eff = -1.0;
  for (int64_t s = 1; s <= std::min<int64_t>(max_splits, tiles / 4); ++s) {
    const double waves = (double)(p.i_blocks * s) / (double)slots;
    const double e = waves / std::ceil(waves);
    const int64_t per = ceil_div(tiles, s);
    if (s > 1 && ceil_div(tiles, per) != s) continue;
    if (s == 1 || e > eff + 0.02) {
      eff = e;
      p.splits = (int)s;
      p.jper = per * kRingTile;
    }
    if (e >= 0.97) break;
  }
  *busy = (double)n * (double)n /
          ((double)(ceil_div(p.i_blocks * p.splits, slots) * slots) * (double)(p.jper * T));
  return p;
}

DirectPlan plan_direct(int64_t n, int max_splits) {
  constexpr double kCtaClocks = 3000.0, kRunClocks = 60.0;
  n = std::max<int64_t>(n, 1);
  const int64_t sms = num_sms();
  DirectPlan best;
  if ((best.small = direct_small_fit(n))) return best;
  if (n > kDirRingFit) {
    double busy = 0.0;
    const DirectPlan ring = plan_ring(n, max_splits, &busy);
    if (n >= kDirRingMin || busy >= kDirRingBusy) return ring;
  }
  double best_t = 1e300;
  for (int I = 1; I <= 2; ++I) {
    const int64_t T = (int64_t)kDirHalf * I, blocks = ceil_div(n, T);
    const int64_t s_max = std::max<int64_t>(
        1, std::min<int64_t>({ceil_div(n, 32), (int64_t)max_splits, kDirMaxBlocks / blocks}));
    for (int64_t s = 1; s <= s_max; ++s) {
      const int64_t jper = ceil_div(ceil_div(n, s), 16) * 16;
      if (ceil_div(n, jper) != s) continue;
      const int64_t k = ceil_div(blocks * s, sms);
      const double t = kCtaClocks * (double)ceil_div(k, 3) +
                       (double)k * (double)(jper * T) / (k == 1 ? 7.9 : I == 1 ? 8.65 : 8.95) +
                       (s > 1 ? 2000.0 + kRunClocks * (double)s : 0.0);
      if (t < 0.99 * best_t) {
        best_t = t;
        best.per_thread = I;
        best.i_blocks = blocks;
        best.n_tgt_pad = blocks * T;
        best.splits = (int)s;
        best.jper = jper;
      }
    }
  }
  return best;
}

template <int I, bool SOA>
static void launch_one(const DirectArgs& a, dim3 grid, bool comp, bool zs, cudaStream_t st) {
  if (zs)
    comp ? direct_kernel<I, true, true, SOA><<<grid, kDirThreads, 0, st>>>(a)
         : direct_kernel<I, false, true, SOA><<<grid, kDirThreads, 0, st>>>(a);
  else
    comp ? direct_kernel<I, true, false, SOA><<<grid, kDirThreads, 0, st>>>(a)
         : direct_kernel<I, false, false, SOA><<<grid, kDirThreads, 0, st>>>(a);
  NBGB_LAUNCH_CHECK();
}

template <bool SOA>
static void launch_direct_any(const DirectPlan& p, DirectArgs& a, bool comp, cudaStream_t st) {
  a.n_tgt_pad = p.n_tgt_pad;
  a.jper = p.jper;
  a.splits = p.splits;
  const dim3 grid((unsigned)p.i_blocks, (unsigned)p.splits);
  const bool zs = !(a.eps2 > 0.f);
  if (p.per_thread == 1)
    launch_one<1, SOA>(a, grid, comp, zs, st);
  else
    launch_one<2, SOA>(a, grid, comp, zs, st);
}

void launch_direct(const DirectPlan& p, const DirectSource& src, int64_t n, float G, float eps2,
                   bool compensated, float4* partial, uint32_t* ticket, float* ox, float* oy,
                   float* oz, cudaStream_t st, uint32_t* err) {
  if (n <= 0) return;
  if (p.small) {
    launch_direct_small(src, n, G, eps2, compensated, ox, oy, oz, st);
    return;
  }
  DirectArgs a{};
  a.src = src.pm;
  a.sx = src.x;
  a.sy = src.y;
  a.sz = src.z;
  a.sm = src.m;
  a.n_src = n;
  a.n_tgt = n;
  a.eps2 = eps2;
  a.G = G;
  a.partial = partial;
  a.ticket = ticket;
  a.out_x = ox;
  a.out_y = oy;
  a.out_z = oz;
  if (p.ring) {
    a.err = err;
    a.n_src = ceil_div(n, (int64_t)kRingTile) * kRingTile;
    a.n_tgt_pad = p.n_tgt_pad;
    a.jper = p.jper;
    a.splits = p.splits;
    const dim3 grid((unsigned)p.i_blocks, (unsigned)p.splits);
    if (eps2 > 0.f)
      compensated ? direct_ring_kernel<true, false><<<grid, kDirHalf, 0, st>>>(a)
                  : direct_ring_kernel<false, false><<<grid, kDirHalf, 0, st>>>(a);
    else
      compensated ? direct_ring_kernel<true, true><<<grid, kDirHalf, 0, st>>>(a)
                  : direct_ring_kernel<false, true><<<grid, kDirHalf, 0, st>>>(a);
    NBGB_LAUNCH_CHECK();
    if (p.splits > 1) {
      direct_runs_kernel<<<(unsigned)num_sms() * 8, 256, 0, st>>>(a);
      NBGB_LAUNCH_CHECK();
    }
  } else if (src.pm)
    launch_direct_any<false>(p, a, compensated, st);
  else
    launch_direct_any<true>(p, a, compensated, st);
}

// ---------------------------------------------------------------------------
// Energies (FP64 reductions).
// ---------------------------------------------------------------------------

// Deterministic two-level reduction of per-thread doubles: block sums go to
// `partials`, a single block then adds them in a fixed order.
template <int NV>
__device__ __forceinline__ void block_reduce_store(double (&v)[NV], double* partials) {
  __shared__ double s_red[32][NV];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k)
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) s_red[warp][k] = v[k];
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double t = (lane < nw) ? s_red[lane][k] : 0.0;
      for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
      if (lane == 0) partials[(int64_t)blockIdx.x * NV + k] = t;
    }
  }
}

template <int NV>
__global__ void finish_reduce_kernel(const double* __restrict__ partials, int nblocks,
                                     double* __restrict__ out) {
  double v[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = 0.0;
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x)
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] += partials[(int64_t)b * NV + k];
  // a tree over the 256 threads (one thread adding 256 values took 9 us each)
  block_reduce_store<NV>(v, out);
}

// KE (and optionally momentum) from FP32 SoA velocities.
__global__ void ke_f32_kernel(const float* __restrict__ vx, const float* __restrict__ vy,
                              const float* __restrict__ vz, const float* __restrict__ m,
                              int64_t n, double* partials) {
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    double a = vx[i], b = vy[i], c = vz[i], mm = m[i];
    v[0] += 0.5 * mm * (a * a + b * b + c * c);
    v[1] += mm * a;
    v[2] += mm * b;
    v[3] += mm * c;
  }
  block_reduce_store<4>(v, partials);
}

// KE and momentum from FP64 velocities.
__global__ void ke_f64_kernel(const double* __restrict__ vx, const double* __restrict__ vy,
                              const double* __restrict__ vz, const float4* __restrict__ pm,
                              int64_t n, double* partials) {
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    double a = vx[i], b = vy[i], c = vz[i], mm = pm[i].w;
    v[0] += 0.5 * mm * (a * a + b * b + c * c);
    v[1] += mm * a;
    v[2] += mm * b;
    v[3] += mm * c;
  }
  block_reduce_store<4>(v, partials);
}

// Potential: phi_i = -sum_{j != i} m_j / sqrt(d^2 + eps^2), FP32 pairs with
// one Newton step on the MUFU rsqrt (near-correctly-rounded), compensated
// per 256-body chunk; PE = G/2 sum_i m_i phi_i accumulated in FP64.
__global__ void pe_kernel(const float4* __restrict__ src, int64_t n, float eps2,
                          double* partials) {
  __shared__ float4 s_j[256];
  double acc[1] = {0.0};
  const int64_t n_chunks = ceil_div(n, 256);
  for (int64_t ib = blockIdx.x; ib * 256 < n; ib += gridDim.x) {
    int64_t i = ib * 256 + threadIdx.x;
    float4 pi = (i < n) ? src[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    float s = 0.f, e = 0.f;
    for (int64_t c = 0; c < n_chunks; ++c) {
      __syncthreads();
      int64_t j = c * 256 + threadIdx.x;
      s_j[threadIdx.x] = (j < n) ? src[j] : make_float4(0.f, 0.f, 0.f, 0.f);
      __syncthreads();
      float t = 0.f;
      const int lim = (int)imin64(256, n - c * 256);
      for (int k = 0; k < lim; ++k) {
        float4 pj = s_j[k];
        float dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
        float d2 = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, eps2)));
        float r = rsqrt_approx(d2);
        r = r * fmaf(-0.5f * d2, r * r, 1.5f);
        bool self = (c * 256 + k) == i;
        t = self ? t : fmaf(-pj.w, r, t);
      }
      float err;
      s = two_sum(s, t, err);
      e += err;
    }
    if (i < n) acc[0] += 0.5 * (double)pi.w * ((double)s + (double)e);
  }
  block_reduce_store<1>(acc, partials);
}

void launch_kinetic_f32(const float* vx, const float* vy, const float* vz, const float* m,
                        int64_t n, double* partials, int nblocks, double* out, cudaStream_t st) {
  ke_f32_kernel<<<nblocks, 256, 0, st>>>(vx, vy, vz, m, n, partials);
  NBGB_LAUNCH_CHECK();
  finish_reduce_kernel<4><<<1, 256, 0, st>>>(partials, nblocks, out);
  NBGB_LAUNCH_CHECK();
}

void launch_kinetic_f64(const double* vx, const double* vy, const double* vz, const float4* pm,
                        int64_t n, double* partials, int nblocks, double* out, cudaStream_t st) {
  ke_f64_kernel<<<nblocks, 256, 0, st>>>(vx, vy, vz, pm, n, partials);
  NBGB_LAUNCH_CHECK();
  finish_reduce_kernel<4><<<1, 256, 0, st>>>(partials, nblocks, out);
  NBGB_LAUNCH_CHECK();
}

void launch_potential(const float4* src, int64_t n, float eps2, double* partials, int nblocks,
                      double* out, cudaStream_t st) {
  pe_kernel<<<nblocks, 256, 0, st>>>(src, n, eps2, partials);
  NBGB_LAUNCH_CHECK();
  finish_reduce_kernel<1><<<1, 256, 0, st>>>(partials, nblocks, out);
  NBGB_LAUNCH_CHECK();
}

// ----------------------------------------------- FP64-state kernels --
// Forces and energies from FP64 positions in FP64 arithmetic: the full-FP64
// system variant and the energy of every FP64-state system.  Forces: 256-body
// tiles of (x, y, z, m) in shared memory, one target per thread,
// self excluded by index, rsqrt from the CUDA math library.
__global__ void __launch_bounds__(256) direct_f64_state_kernel(
    const double* __restrict__ x, const double* __restrict__ y, const double* __restrict__ z,
    const float4* __restrict__ pm, int64_t n, double G, double eps2, double* __restrict__ ax,
    double* __restrict__ ay, double* __restrict__ az) {
  __shared__ double4 s_j[256];
  for (int64_t base = (int64_t)blockIdx.x * 256; base < n; base += (int64_t)gridDim.x * 256) {
    const int64_t i = base + threadIdx.x;
    const bool valid = i < n;
    const double xi = valid ? x[i] : 0.0, yi = valid ? y[i] : 0.0, zi = valid ? z[i] : 0.0;
    double sx = 0.0, sy = 0.0, sz = 0.0;
    for (int64_t c = 0; c < n; c += 256) {
      __syncthreads();
      const int64_t j = c + threadIdx.x;
      s_j[threadIdx.x] = (j < n) ? make_double4(x[j], y[j], z[j], (double)pm[j].w)
                                 : make_double4(0.0, 0.0, 0.0, 0.0);
      __syncthreads();
      const int lim = (int)imin64(256, n - c);
      for (int k = 0; k < lim; ++k) {
        if (c + k == i) continue;
        const double4 q = s_j[k];
        const double dx = q.x - xi, dy = q.y - yi, dz = q.z - zi;
        const double d2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)));
        const double r = rsqrt(d2);
        const double f = q.w * r * r * r;
        sx = fma(f, dx, sx);
        sy = fma(f, dy, sy);
        sz = fma(f, dz, sz);
      }
    }
    if (valid) {
      ax[i] = G * sx;
      ay[i] = G * sy;
      az[i] = G * sz;
    }
  }
}

// Reciprocal square root in FP64: an FP32 seed y (relative error below 2^-22)
// and one third-order step, y + y e (1/2 + 3/8 e) with e = 1 - d y^2 (the
// binomial series of (1 - e)^(-1/2), remainder 5/16 e^3 < 2^-63, so that the last
// operation's rounding is what remains); y^2 is exact in FP64.  5 FP64 operations and
// two conversions.  Outside the seed's safe range (and for zero, infinity and NaN) the
// math library's rsqrt.
__device__ __forceinline__ double rsqrt_f64(double d) {
  const uint32_t hi = (uint32_t)__double2hiint(d);
  if (hi - 0x38f00000u > 0x0e000000u) return rsqrt(d);  // outside 2^-112 .. 2^112
  const double y = (double)rsqrt_approx((float)d);
  const double e = fma(-d, y * y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// Kinetic energy, momentum and potential energy of an FP64-state system in
// one launch.  PE: every unordered pair once, as 64 x 64 tiles of the upper
// triangle dealt out to the CTAs (a thread keeps one target of the tile, the
// sources are read from shared memory).  Bound by the FP64 pipe (2 lanes per
// clock and SM; 12 operations per pair, and the two conversions run there as well):
// small tiles, so that few bodies still reach every SM.  N = 8,191: 6.9 ms as one
// 256-target CTA per row of ordered pairs (32 CTAs), 0.93 ms now with the pipe 87 %
// busy (0.75 at its full rate).
constexpr int kPeTile = 64;

__global__ void __launch_bounds__(kPeTile) energy_f64_kernel(EnergyArgs a) {
  __shared__ double4_16a s_j[kPeTile];
  __shared__ bool s_last;
  const int tid = threadIdx.x;
  double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // KE, momentum, PE
  for (int64_t i = blockIdx.x * (int64_t)kPeTile + tid; i < a.n; i += (int64_t)gridDim.x * kPeTile) {
    const double p = a.vx[i], q = a.vy[i], r = a.vz[i], m = a.pm[i].w;
    v[0] += 0.5 * m * (p * p + q * q + r * r);
    v[1] += m * p;
    v[2] += m * q;
    v[3] += m * r;
  }
  const int64_t tiles = ceil_div(a.n, kPeTile), pairs = tiles * (tiles + 1) / 2;
  for (int64_t t = blockIdx.x; t < pairs; t += gridDim.x) {
    // row r of the triangle holds the tiles (r, r) .. (r, tiles - 1) and starts
    // at r tiles - r (r - 1) / 2; the root estimate is corrected exactly
    const double b = (double)tiles + 0.5;
    int64_t r = (int64_t)(b - sqrt(fmax(b * b - 2.0 * (double)t, 0.0)));
    r = imax64(0, imin64(r, tiles - 1));
    while (r > 0 && r * tiles - r * (r - 1) / 2 > t) --r;
    while ((r + 1) * tiles - (r + 1) * r / 2 <= t) ++r;
    const int64_t c = r + (t - (r * tiles - r * (r - 1) / 2));
    const int64_t i = r * kPeTile + tid, j = c * kPeTile + tid;
    __syncthreads();
    if (j < a.n) {
      s_j[tid].x = a.x[j];
      s_j[tid].y = a.y[j];
      s_j[tid].z = a.z[j];
      s_j[tid].w = (double)a.pm[j].w;
    }
    __syncthreads();
    if (i < a.n) {
      const double xi = a.x[i], yi = a.y[i], zi = a.z[i];
      const int lim = (int)imin64(kPeTile, a.n - c * kPeTile);
      double s = 0.0;
      // in a diagonal tile only the sources after the target
#pragma unroll 4
      for (int k = (r == c) ? tid + 1 : 0; k < lim; ++k) {
        const double dx = s_j[k].x - xi, dy = s_j[k].y - yi, dz = s_j[k].z - zi;
        s = fma(s_j[k].w, rsqrt_f64(fma(dx, dx, fma(dy, dy, fma(dz, dz, a.eps2)))), s);
      }
      v[4] -= (double)a.pm[i].w * s;
    }
  }
  block_reduce_store<5>(v, a.partials);
  if (tid == 0) {
    __threadfence();
    s_last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (tid == 0) *a.ticket = 0;  // ready for the next launch
#pragma unroll
  for (int k = 0; k < 5; ++k) v[k] = 0.0;
  for (int b = tid; b < (int)gridDim.x; b += kPeTile)
#pragma unroll
    for (int k = 0; k < 5; ++k) v[k] += __ldcg(&a.partials[(int64_t)b * 5 + k]);
  __syncthreads();
  block_reduce_store<5>(v, a.out - (int64_t)blockIdx.x * 5);
}

int energy_f64_blocks(int64_t n) {
  const int64_t tiles = ceil_div(std::max<int64_t>(n, 1), kPeTile);
  return (int)std::min<int64_t>(tiles * (tiles + 1) / 2, (int64_t)num_sms() * 8);
}

void launch_energy_f64(const EnergyArgs& a, cudaStream_t st) {
  energy_f64_kernel<<<(unsigned)energy_f64_blocks(a.n), kPeTile, 0, st>>>(a);
  NBGB_LAUNCH_CHECK();
}

void launch_direct_f64_state(const double* x, const double* y, const double* z, const float4* pm,
                             int64_t n, double G, double eps2, double* ax, double* ay, double* az,
                             cudaStream_t st) {
  if (n <= 0) return;
  const unsigned blocks =
      (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, 256), (int64_t)num_sms() * 8));
  direct_f64_state_kernel<<<blocks, 256, 0, st>>>(x, y, z, pm, n, G, eps2, ax, ay, az);
  NBGB_LAUNCH_CHECK();
}

}  // namespace nbgb

// ---------------------------------------------------------------------------
// FP64 direct sum (the full-FP64 variant; accuracy reference on the GPU).
// ---------------------------------------------------------------------------
namespace nbgb {

__global__ void direct_f64_kernel(const float4* __restrict__ src, int64_t n_src,
                                  const int64_t* __restrict__ targets, int64_t n_tgt, double G,
                                  double eps2, double* __restrict__ ax, double* __restrict__ ay,
                                  double* __restrict__ az) {
  __shared__ float4 s_j[256];
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < n_tgt;
       base += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = base + threadIdx.x;
    const bool valid = t < n_tgt;
    const int64_t i = valid ? (targets ? targets[t] : t) : 0;
    const float4 pi = src[i];
    double sx = 0.0, sy = 0.0, sz = 0.0;
    for (int64_t c = 0; c < n_src; c += 256) {
      __syncthreads();
      const int64_t j = c + threadIdx.x;
      s_j[threadIdx.x] = (j < n_src) ? src[j] : make_float4(0.f, 0.f, 0.f, 0.f);
      __syncthreads();
      const int lim = (int)imin64(256, n_src - c);
      for (int k = 0; k < lim; ++k) {
        if (c + k == i) continue;
        const float4 pj = s_j[k];
        const double dx = (double)pj.x - (double)pi.x, dy = (double)pj.y - (double)pi.y,
                     dz = (double)pj.z - (double)pi.z;
        const double d2 = dx * dx + dy * dy + dz * dz + eps2;
        const double inv = 1.0 / sqrt(d2);
        const double f = (double)pj.w * inv * inv * inv;
        sx += f * dx;
        sy += f * dy;
        sz += f * dz;
      }
    }
    if (valid) {
      ax[t] = G * sx;
      ay[t] = G * sy;
      az[t] = G * sz;
    }
  }
}

}  // namespace nbgb

extern "C" nbgb_status nbgb_direct_f64(const float* d_src_xyzm, int64_t n_src,
                                       const int64_t* d_targets, int64_t n_targets, double G,
                                       double eps, double* d_ax, double* d_ay, double* d_az,
                                       void* stream) {
  using namespace nbgb;
  try {
    if (!d_src_xyzm || !d_ax || !d_ay || !d_az || n_src < 0 || n_targets < 0)
      return NBGB_ERR_INVALID_ARG;
    if (n_targets == 0) return NBGB_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int64_t blocks = std::min<int64_t>(ceil_div(n_targets, 256), (int64_t)num_sms() * 8);
    direct_f64_kernel<<<(unsigned)blocks, 256, 0, st>>>(
        reinterpret_cast<const float4*>(d_src_xyzm), n_src, d_targets, n_targets, G, eps * eps,
        d_ax, d_ay, d_az);
    NBGB_LAUNCH_CHECK();
    return NBGB_OK;
  } catch (const Error& e) {
    return e.status;
  }
}
