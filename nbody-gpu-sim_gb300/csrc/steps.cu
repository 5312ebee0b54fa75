// steps.cu -- direct sum of a small system, and several of its Velocity-Verlet
// steps in one cooperative launch.
//
// Same update as kick_drift_kernel followed by the direct sum (integrate.cu,
// direct.cu; the reference's ParticleSystem::update, particle_system.cpp:
// 122-136): x, v in FP64, forces in FP32 from the rounded positions.
//
// What bounds it: latency.  A step of 1,024 bodies is 0.3 us of arithmetic,
// but two dependent launches took 11 us (66 + 4 us with one CTA per 1,024
// targets).  Here every CTA keeps the FP64 state of its T targets in
// registers for all steps; per step it publishes their positions, passes one
// grid barrier, copies all bodies to shared memory and sums them, so a step
// costs one barrier and one read of 16 N bytes.  T = 8, 16 or 32 targets per
// CTA, the smallest that needs no more CTAs than SMs: fewer targets per
// CTA share the sum over more threads (64 slices of the sources at T = 8).
// Measured per step in calls of 100 steps: N = 256 2.3 us, 1,024 3.1 (80
// before the sources were split, 11 as two launches), 4,864 12.
// Force calculators and a system's a(0) run the same kernel (steps = 0, an
// ordinary launch), so a trajectory does not depend on how its steps are
// grouped into calls, and the forces of a system are a calculator's, bitwise.
#include <atomic>

#include "common.cuh"
#include "direct_pair.cuh"
#include "kernels.cuh"

namespace nbgb {

constexpr int kStepThreads = 512;
constexpr int kStepWarps = kStepThreads / 32;

struct StepArgs {
  double *x, *y, *z, *vx, *vy, *vz;
  float *ax, *ay, *az;
  float4* pm;      // packed bodies, or (forces only) null: the SoA arrays
  const float *px, *py, *pz, *pw;
  float4* exch;    // [2][n] positions of the current step (ping-pong)
  uint32_t* ctr;   // arrivals at the grid barrier, CTAs done: zero before and after
  uint32_t* err;
  int n;
  int steps;       // 0: only the forces of the bodies
  double kick0, kick, dt;  // first kick, later kicks
  float eps2, G;
};

// All CTAs have arrived `round` times: false if the bounded wait ran out.
__device__ __forceinline__ bool grid_barrier(uint32_t* ctr, uint32_t target, uint32_t* err,
                                             bool* s_ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
    bool ok = false;
    for (uint32_t it = 0; it < (1u << 22); ++it) {
      uint32_t v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
      if (v >= target) {
        ok = true;
        break;
      }
    }
    if (!ok) raise_error(err, kErrWaitTimeout);
    *s_ok = ok;
  }
  __syncthreads();
  return *s_ok;
}

// TL targets per CTA; 512 / TL slices of the sources, of at most 304 sources in
// two plain FP32 sums (even and odd ones).
template <int TL, bool COMP, bool ZERO_SOFT>
__global__ void __launch_bounds__(kStepThreads, 1) direct_steps_kernel(StepArgs a) {
  constexpr int T = TL, kSlices = kStepThreads / TL;
  extern __shared__ __align__(16) float s_body[];  // rows x, y, z, m of n4 floats
  __shared__ float s_red[kStepWarps][3][T];
  __shared__ bool s_ok;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tl = tid % TL, slice = tid / TL;
  const int n4 = (a.n + 3) & ~3, base = blockIdx.x * T;
  float *sx = s_body, *sy = sx + n4, *sz = sy + n4, *sm = sz + n4;
  // owners: thread t < T keeps target base + t
  const int own = base + tid;
  const bool owner = tid < T && own < a.n;
  double px = 0, py = 0, pz = 0, u = 0, v = 0, w = 0;
  float fx = 0, fy = 0, fz = 0, mass = 0;
  if (owner && a.steps) {
    px = a.x[own];
    py = a.y[own];
    pz = a.z[own];
    u = a.vx[own];
    v = a.vy[own];
    w = a.vz[own];
    fx = a.ax[own];
    fy = a.ay[own];
    fz = a.az[own];
    mass = a.pm[own].w;
  }
  const int rounds = max(a.steps, 1);
  bool ok = true;
  for (int k = 0; k < rounds; ++k) {
    const float4* src = a.pm;
    if (a.steps) src = a.exch + (int64_t)(k & 1) * a.n;
    if (owner && a.steps) {
      const double kick = k == 0 ? a.kick0 : a.kick;
      u = fma((double)fx, kick, u);
      v = fma((double)fy, kick, v);
      w = fma((double)fz, kick, w);
      px = fma(u, a.dt, px);
      py = fma(v, a.dt, py);
      pz = fma(w, a.dt, pz);
      __stcg(&a.exch[(int64_t)(k & 1) * a.n + own], make_float4((float)px, (float)py, (float)pz, mass));
    }
    if (a.steps && !grid_barrier(a.ctr, (uint32_t)(k + 1) * gridDim.x, a.err, &s_ok)) {
      ok = false;
      break;
    }
    for (int j = tid; j < n4; j += kStepThreads) {
      float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j < a.n) q = src ? __ldcg(&src[j]) : make_float4(a.px[j], a.py[j], a.pz[j], a.pw[j]);
      sx[j] = q.x;
      sy[j] = q.y;
      sz[j] = q.z;
      sm[j] = q.w;
    }
    __syncthreads();
    const int i = min(base + tl, a.n - 1);
    const f2 xi = f2_make(sx[i], sx[i]), yi = f2_make(sy[i], sy[i]), zi = f2_make(sz[i], sz[i]);
    f2 ax = f2_make(0.f, 0.f), ay = ax, az = ax;
    const f2 e2 = f2_make(a.eps2, a.eps2);
    // the slices take quads of sources in turn: a warp's slices read
    // neighbouring 16-byte words
#pragma unroll 4
    for (int j = 4 * slice; j < n4; j += 4 * kSlices) {
      const ulonglong2 X = *reinterpret_cast<const ulonglong2*>(sx + j);
      const ulonglong2 Y = *reinterpret_cast<const ulonglong2*>(sy + j);
      const ulonglong2 Z = *reinterpret_cast<const ulonglong2*>(sz + j);
      const ulonglong2 M = *reinterpret_cast<const ulonglong2*>(sm + j);
      pair_step<ZERO_SOFT>(f2{X.x}, f2{Y.x}, f2{Z.x}, f2{M.x}, xi, yi, zi, e2, ax, ay, az);
      pair_step<ZERO_SOFT>(f2{X.y}, f2{Y.y}, f2{Z.y}, f2{M.y}, xi, yi, zi, e2, ax, ay, az);
    }
    {
      float s[3] = {f2_sum(ax), f2_sum(ay), f2_sum(az)};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int o = TL; o < 32; o <<= 1) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
        if (lane < TL) s_red[warp][c][tl] = s[c];
      }
    }
    __syncthreads();
    if (owner) {
      float s[3] = {0.f, 0.f, 0.f}, e[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int r = 0; r < kStepWarps; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) fold<COMP>(s_red[r][c][tid], s[c], e[c]);
      fx = a.G * (s[0] + e[0]);
      fy = a.G * (s[1] + e[1]);
      fz = a.G * (s[2] + e[2]);
    }
  }
  if (owner && ok && a.steps) {
    a.x[own] = px;
    a.y[own] = py;
    a.z[own] = pz;
    a.vx[own] = u;
    a.vy[own] = v;
    a.vz[own] = w;
    a.pm[own] = make_float4((float)px, (float)py, (float)pz, mass);
  }
  if (owner && ok) {
    a.ax[own] = fx;
    a.ay[own] = fy;
    a.az[own] = fz;
  }
  // the last CTA to leave (every CTA does, its waits are bounded) resets the
  // counters for the next launch
  if (a.steps && tid == 0 && atomicAdd(&a.ctr[1], 1u) == gridDim.x - 1) {
    a.ctr[0] = 0;
    a.ctr[1] = 0;
  }
}

// Cooperative launches of more CTAs than this are refused (0: none; test hook).
static std::atomic<int> g_cooperative_limit{0};
void direct_set_cooperative_limit(int ctas) { g_cooperative_limit.store(ctas); }

// False: the CTAs cannot all be resident (a share of the GPU with fewer SMs than
// the device reports), and nothing was launched.
template <int TL, bool COMP, bool ZS>
static bool launch_steps_t(StepArgs& a, cudaStream_t st) {
  const size_t smem = (size_t)((a.n + 3) & ~3) * 16;
  auto kern = direct_steps_kernel<TL, COMP, ZS>;
  // (one limit for all sizes: the attribute is the kernel's, and a smaller one set for a
  // call in another thread would refuse this one's launch)
  NBGB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(kDirectSmallMaxBodies * 16)));
  const unsigned grid = (unsigned)ceil_div(a.n, TL);
  if (a.steps) {
    void* args[] = {&a};
    const int limit = g_cooperative_limit.load(std::memory_order_relaxed);
    const cudaError_t e = limit > 0 && grid > (unsigned)limit
                              ? cudaErrorCooperativeLaunchTooLarge
                              : cudaLaunchCooperativeKernel((const void*)kern, dim3(grid),
                                                            dim3(kStepThreads), args, smem, st);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
      cudaGetLastError();
      return false;
    }
    NBGB_CUDA(e);
  } else {  // forces only: the CTAs do not wait on one another
    kern<<<grid, kStepThreads, smem, st>>>(a);
  }
  NBGB_LAUNCH_CHECK();
  return true;
}

template <int TL>
static bool launch_steps_n(StepArgs& a, bool comp, cudaStream_t st) {
  const bool zs = !(a.eps2 > 0.f);
  if (zs)
    return comp ? launch_steps_t<TL, true, true>(a, st) : launch_steps_t<TL, false, true>(a, st);
  return comp ? launch_steps_t<TL, true, false>(a, st) : launch_steps_t<TL, false, false>(a, st);
}

// Sizes for this kernel: up to 32 targets per CTA on at most one CTA per SM.
// With 64 targets per CTA it took systems of up to twice that, too: alone 4 to
// 10 % faster in calls of 20 steps (8,192 bodies 36.0 us per step against 37.5),
// but its shared memory and its one CTA per SM keep other streams' systems
// waiting (16 systems of 8,192 bodies on streams of their own 35.2 us per step,
// 25.0 with the source runs of direct_kernel), and its slices added up to 608
// sources in plain FP32.
bool direct_small_fit(int64_t n) {
  return n <= std::min<int64_t>(32 * num_sms(), kDirectSmallMaxBodies);
}

static bool launch_small(StepArgs& a, bool comp, cudaStream_t st) {
  const int64_t sms = num_sms();
  if (a.n <= 8 * sms) return launch_steps_n<8>(a, comp, st);
  if (a.n <= 16 * sms) return launch_steps_n<16>(a, comp, st);
  return launch_steps_n<32>(a, comp, st);
}

void launch_direct_small(const DirectSource& src, int64_t n, float G, float eps2, bool comp,
                         float* ox, float* oy, float* oz, cudaStream_t st) {
  StepArgs a{};
  a.pm = const_cast<float4*>(src.pm);  // only read without steps
  a.px = src.x;
  a.py = src.y;
  a.pz = src.z;
  a.pw = src.m;
  a.ax = ox;
  a.ay = oy;
  a.az = oz;
  a.n = (int)n;
  a.eps2 = eps2;
  a.G = G;
  launch_small(a, comp, st);
}

bool launch_direct_steps(const StateArrays& s, int64_t n, int32_t steps, double kick0, double kick,
                         double dt, float eps2, float G, bool comp, float4* exch, uint32_t* ctr,
                         uint32_t* err, cudaStream_t st) {
  StepArgs a{};
  a.x = s.x;
  a.y = s.y;
  a.z = s.z;
  a.vx = s.vx;
  a.vy = s.vy;
  a.vz = s.vz;
  a.ax = s.ax;
  a.ay = s.ay;
  a.az = s.az;
  a.pm = s.pm;
  a.exch = exch;
  a.ctr = ctr;
  a.err = err;
  a.n = (int)n;
  a.kick = kick;
  a.dt = dt;
  a.eps2 = eps2;
  a.G = G;
  a.steps = steps;
  a.kick0 = kick0;
  return launch_small(a, comp, st);
}

}  // namespace nbgb
