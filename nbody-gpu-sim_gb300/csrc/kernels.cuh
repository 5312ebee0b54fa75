// kernels.cuh -- launcher declarations shared by the nbgb translation units.
#pragma once

#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace nbgb {

// ----------------------------------------------------------------- direct --
constexpr int kDirThreads = 256;  // threads per CTA of the direct kernel
constexpr int kDirHalf = 128;     // threads per half: a half sums its own sources
constexpr int kDirTile = 512;     // sources per shared-memory tile (8 KB)

struct DirectArgs {
  const float4* src;                              // packed sources (x, y, z, m), or
  const float *sx, *sy, *sz, *sm;                 // the caller's SoA arrays
  int64_t n_src;
  int64_t n_tgt;                                  // the first n_tgt sources are the targets
  int64_t n_tgt_pad;
  int64_t jper;                                   // sources per run (CTA)
  int splits;                                     // runs
  float eps2;
  float G;
  float4* partial;                                // [splits][n_tgt_pad] when splits > 1
  uint32_t* ticket;                               // per target block, zero between launches
  float* out_x;
  float* out_y;
  float* out_z;
  uint32_t* err;     // device error word (ring)
};

// Bodies of a direct sum: pm (packed), or the SoA arrays when pm is null.
struct DirectSource {
  const float4* pm;
  const float *x, *y, *z, *m;
};

struct DirectPlan {
  bool small = false;     // the small-system kernel (one CTA set, no runs)
  bool ring = false;      // the tile-ring kernel of the largest systems (packed sources)
  int per_thread = 1;     // targets per thread (1 or 2; 8 with ring)
  int64_t i_blocks = 0;   // target blocks of kDirHalf * per_thread
  int64_t n_tgt_pad = 0;
  int splits = 1;         // source runs
  int64_t jper = 0;       // sources per run, a multiple of 16 (ring: of 256)
};

// Whether a direct sum may read the caller's arrays while it writes the
// accelerations (no overlap).
bool direct_from_soa(const nbgb_particle_data* d);
constexpr int kDirMaxSplits = 128;
constexpr int64_t kDirMaxBlocks = 16384;  // target blocks of a plan with several runs
DirectPlan plan_direct(int64_t n, int max_splits = kDirMaxSplits);
// Forces on all n bodies of src.  With p.splits > 1: partial holds
// splits * n_tgt_pad entries, ticket i_blocks counters that are zero before
// the launch and zero again after it.  With p.ring: no ticket, and src.pm is given,
// padded with massless bodies to a multiple of kDirRingPad.
constexpr int64_t kDirRingPad = 256;
void launch_direct(const DirectPlan& p, const DirectSource& src, int64_t n, float G, float eps2,
                   bool compensated, float4* partial, uint32_t* ticket, float* ox, float* oy,
                   float* oz, cudaStream_t st, uint32_t* err = nullptr);
void launch_pack_soa(const float* x, const float* y, const float* z, const float* m, int64_t n,
                     int64_t n_pad, float4* out, cudaStream_t st);

// Small systems (steps.cu): the forces of n bodies, or `steps` kick-drift +
// force steps in one cooperative launch (false: refused, its CTAs cannot all be
// resident; nothing has been launched).  exch: 2 n entries; ctr: two
// counters, zero before and after.
constexpr int64_t kDirectSmallMaxBodies = 4864;  // 16 bytes per body in shared memory
constexpr int32_t kDirectStepsPerLaunch = 256;   // bounds one launch's time
struct StateArrays {
  double *x, *y, *z, *vx, *vy, *vz;
  float *ax, *ay, *az;
  float4* pm;
};
bool direct_small_fit(int64_t n);
void launch_direct_small(const DirectSource& src, int64_t n, float G, float eps2, bool comp,
                         float* ox, float* oy, float* oz, cudaStream_t st);
bool launch_direct_steps(const StateArrays& s, int64_t n, int32_t steps, double kick0, double kick,
                         double dt, float eps2, float G, bool comp, float4* exch, uint32_t* ctr,
                         uint32_t* err, cudaStream_t st);
void direct_set_cooperative_limit(int ctas);  // test hook: CTAs of a launch (0: no limit)

// Energies: `partials` needs nblocks * 4 doubles; out[0..3] = KE, Px, Py, Pz
// (kinetic) or out[0] = sum_i m_i phi_i / 2 without G (potential).
void launch_kinetic_f32(const float* vx, const float* vy, const float* vz, const float* m,
                        int64_t n, double* partials, int nblocks, double* out, cudaStream_t st);
void launch_kinetic_f64(const double* vx, const double* vy, const double* vz, const float4* pm,
                        int64_t n, double* partials, int nblocks, double* out, cudaStream_t st);
void launch_potential(const float4* src, int64_t n, float eps2, double* partials, int nblocks,
                      double* out, cudaStream_t st);

// ------------------------------------------------------------- integrator --
// FP32 SoA Velocity Verlet (reference semantics).
void launch_vv_positions(const nbgb_particle_data& d, float dt, bool store_old, float4* pack,
                         int64_t n_pad, cudaStream_t st);
void launch_vv_velocities(const nbgb_particle_data& d, float dt, cudaStream_t st);
void launch_store_old(const nbgb_particle_data& d, cudaStream_t st);

// FP64-state kick-drift: v += a*kick; x += v*dt; pack (float)x into pm.xyz.
void launch_kick_drift(int64_t n, double* x, double* y, double* z, double* vx, double* vy,
                       double* vz, const float* ax, const float* ay, const float* az,
                       double kick, double dt, float4* pm, cudaStream_t st);
// FP64-state kick: v += a*kick.
void launch_kick(int64_t n, double* vx, double* vy, double* vz, const float* ax,
                 const float* ay, const float* az, double kick, cudaStream_t st);
// The same with FP64 accelerations (full-FP64 system).
void launch_kick_drift(int64_t n, double* x, double* y, double* z, double* vx, double* vy,
                       double* vz, const double* ax, const double* ay, const double* az,
                       double kick, double dt, float4* pm, cudaStream_t st);
void launch_kick(int64_t n, double* vx, double* vy, double* vz, const double* ax,
                 const double* ay, const double* az, double kick, cudaStream_t st);
// Direct forces in FP64 from FP64 positions (masses from pm.w).
void launch_direct_f64_state(const double* x, const double* y, const double* z, const float4* pm,
                             int64_t n, double G, double eps2, double* ax, double* ay, double* az,
                             cudaStream_t st);
// Energies and momentum of an FP64 state.  partials: energy_f64_blocks(n) * 5
// doubles; ticket: a counter, zero before and after; out: KE, Px, Py, Pz and
// PE without G (device or mapped host memory).
struct EnergyArgs {
  const double *x, *y, *z, *vx, *vy, *vz;
  const float4* pm;
  int64_t n;
  double eps2;
  double* partials;
  uint32_t* ticket;
  double* out;
};
int energy_f64_blocks(int64_t n);
void launch_energy_f64(const EnergyArgs& a, cudaStream_t st);

// The state of a system into mapped host memory: x, y, z, vx, vy, vz (6 n
// doubles), or rounded with the accelerations and masses (10 n floats).
struct SystemView {
  int64_t n;
  const double *x, *y, *z, *vx, *vy, *vz;
  const float *ax, *ay, *az;
  const double *ax64, *ay64, *az64;  // null unless the system is FP64 throughout
  const float4* pm;
};
void launch_export_f64(const SystemView& s, double* out, cudaStream_t st);
void launch_export_f32(const SystemView& s, float* out, cudaStream_t st);

}  // namespace nbgb
