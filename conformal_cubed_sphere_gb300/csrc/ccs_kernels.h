// ccs_kernels.h -- launch descriptors shared by the kernels and the C ABI layer.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "ccs_internal.h"
#include "ccs_softfp.cuh"

namespace ccs {

// Raises a kernel's dynamic shared-memory limit once per device: the attribute is
// held per device, so a process driving handles on several devices sets it on each
// (`done` is the kernel's own set of device bits; ordinals above 63 set it every
// launch).
inline cudaError_t smem_attr_once(const void *fn, int smem, std::atomic<uint64_t> &done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = dev >= 0 && dev < 64 ? (uint64_t)1 << dev : 0;
  if (bit && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess && bit) done.fetch_or(bit, std::memory_order_acq_rel);
  return e;
}

// Launches a stage kernel.  chained: the launch before it in the stream is the same
// step's previous stage, whose end the kernel itself waits for (stage_wait): its CTAs may
// start, and read their work items and descriptors, while that stage drains.
// Returns this launch's own status (cudaGetLastError would also report an earlier error
// that nobody has collected).
template <class... P, class... A>
cudaError_t launch_stage(void (*kernel)(P...), int grid, int block, int smem, cudaStream_t s, bool chained,
                         A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

#if defined(__CUDACC__)
// lets the next chained stage start its CTAs where they fit, called as a CTA's last tile
// nears its end (at the kernel's start it crowds the next stage's CTAs onto the SMs that
// have room: mixed C150 10.3 -> 12.0 us a stage)
__device__ __forceinline__ void stage_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// waits until the previous stage of a chained launch has ended and its writes are visible
// (returns at once in other launches).  Whatever a stage writes is read after this, and
// never as read-only data (__ldg): it changes while the kernel is already running.
__device__ __forceinline__ void stage_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
#endif

// One tile of work: instance, panel (0..5) and tile coordinates.
struct WorkItem {
  int16_t inst, panel, tx, ty;
};

// Stage kinds.  RK4 (time_scheme_mod.F90:13-44) keeps the running combination
// acc = k1 (+ 2 k2) (+ 2 k3) so that the final (acc + k4) / 6 has the reference's
// association ((k1 + 2k2) + 2k3) + k4.  RK3-TVD follows :46-67, 85-115.
enum StageKind {
  K_RK4_1 = 0,  // acc = k;          Y = Y0 + c1 k
  K_RK4_2 = 1,  // acc = acc + 2 k;  Y = Y0 + c1 k
  K_RK4_4 = 2,  // Y = Y0 + c1 ((acc + k) / 6)
  K_RK3_1 = 3,  // Y = Y0 + c1 k
  K_RK3_2 = 4,  // Y = 0.75 Y0 + 0.25 Yc + c1 k
  K_RK3_3 = 5,  // Y = Y0 / 3 + 2/3 Yc + c1 k
  K_TEND = 6    // write k only
};

// FP64 lane: everything one instance's stage launch needs.
struct F64Stage {
  Layout L;
  MeshF64 m;
  StateF64 in;   // stencil input Y_k
  StateF64 out;  // Y_{k+1} (may alias the Y0 slot: only the own cell of Y0 is read)
  const double *y0phiG, *y0u, *y0v;
  double *accphiG, *accu, *accv;
  double *zonal, *merid;  // sphere winds of Y_{k+1} when non-null
  double *tphiG, *tu, *tv;
  double dx, dy, dx60, dy60, c1;
  softfp::Divisor by_dx, by_dy, by_dx60, by_dy60;
  int kind, ediss;
  int op;  // CCS_OP_WENO, or the central-difference order 2 / 4 / 6
  double one = 1., neg0 = -0.;  // the constants of F64Ops, read at run time on purpose
};

// Mixed lane: one instance's stage launch.
struct MixedStage {
  Layout L;
  MeshMixed m;
  StateMixed in, out;
  const float *y0hp, *y0u, *y0v;
  float *lohp, *lou, *lov;  // compensation terms of the step-to-step state (interior)
  float *acchp, *accu, *accv;
  float *thp, *tu, *tv;
  float rdx, rdy, rdx60, rdy60;  // reciprocals of dx, dy, 60 dx, 60 dy
  float c1;
  float phibar;  // mean geopotential phibar (m^2 s^-2)
  float a2, inv_a2;
  float eps_E;  // WENO eps of E (m^2 s^-2 units: the reference's 1e-2)
  float eps_F;  // eps of the flux / a^2 (1e-2 / a^4)
  float eps_P;  // eps of phitG / a^2 (1e-2 / a^4)
  int kind, ediss;
  int op;             // CCS_OP_WENO, or the central-difference order 2 / 4 / 6
  float rdxc, rdyc;   // 1 / (2 dx), 1 / (12 dx) or 1 / (60 dx) for the central operator
};

// Kernel variants: the tile shape (cells per work item) of each lane's stage kernel.
// A handle runs one variant; the autotuner picks it per resolution by timing.
struct TileShape {
  int tx, ty;
};
constexpr int F64_NVAR = 3;  // 32 x 8, 16 x 16, 64 x 4 (384 threads; small launches run 8 x 8 or 16 x 8 parts)
constexpr TileShape kF64Tiles[F64_NVAR] = {{32, 8}, {16, 16}, {64, 4}};
// Mixed lane: tile shape x halo-staging schedule of phase 1.  kStageLoads: each
// thread loads its cells' raw inputs into registers and stores the derived cell
// quantities; kStageAsync: asynchronous copies (cp.async) put the raw inputs of all
// of a thread's cells into shared memory at once, then the thread derives the
// quantities in place.
constexpr int kStageLoads = 0, kStageAsync = 1;
constexpr int MX_NVAR = 4;  // 32 x 32 (256 threads), 32 x 16 (128 threads); each with both schedules
constexpr TileShape kMxTiles[MX_NVAR] = {{32, 32}, {32, 16}, {32, 32}, {32, 16}};
constexpr int kMxStaging[MX_NVAR] = {kStageLoads, kStageLoads, kStageAsync, kStageAsync};

// Whether a launch of nwork whole mixed tiles on sms SMs may be chained.  With at most two
// 32 x 32 tiles an SM, every SM has room for a third: CTAs that start early crowd onto the
// SMs that drain first, and a stage takes as long as an SM with three (us a step, four steps a
// call, chained / not: C193 66.2 / 60.0, C208 63.8 / 60.1, C224 64.2 / 60.0; with more than two
// C240 72.8 / 75.9, C256 74.1 / 76.4).  32 x 16 tiles, five an SM, are faster chained but for
// the fullest rounds (C200 56.0 / 58.0, C224 62.7 / 62.0).
constexpr bool mixed_chains(TileShape tile, int nwork, int sms) { return tile.ty != 32 || nwork > 2 * sms; }

// kernel launchers (return cudaGetLastError()); `var` indexes the tile tables
// (central: every stage in d_stages uses a central-difference operator, else WENO-Z)
cudaError_t launch_f64_stage(int var, bool central, const F64Stage *d_stages, const WorkItem *d_work, int nwork,
                             int grid, cudaStream_t s, bool chained = false);
int f64_max_grid(int var, bool central, int device);
// what a CTA of such a launch works on: a work item, or the part of one that the launch's
// size selects; and how many of them an SM of the current device holds
struct StageTile {
  int tx, ty, ctas;
};
StageTile f64_stage_tile(int var, bool central, int nwork, int grid);
// the derived metric arrays of MeshF64 (sqrtGf, rsqrtG, lamx, lamy: consecutive fields at out)
cudaError_t launch_f64_mesh_products(const Layout &L, const MeshF64 &m, double *out, cudaStream_t s);

// central: every stage in d_stages uses a central-difference operator (else WENO-Z);
// ediss: every stage reconstructs the E-flux dissipation (CCS_EDISS_RECONSTRUCT)
cudaError_t launch_mixed_stage(int var, bool central, bool ediss, const MixedStage *d_stages,
                               const WorkItem *d_work, int nwork, int grid, cudaStream_t s,
                               bool chained = false);
int mixed_max_grid(int var, int device);
cudaError_t mixed_stage_tile(int var, int nwork, StageTile *tile);
cudaError_t launch_mixed_import(const Layout &L, const double *phi, const double *u, const double *v,
                                double phibar, double inv_a2, StateMixed out, float *lohp, float *lou,
                                float *lov, cudaStream_t s);
cudaError_t launch_mixed_export(const Layout &L, StateMixed st, const float *lohp, const float *lou,
                                const float *lov, const MeshF64 &m, double phibar, double a2, double *const out[8],
                                cudaStream_t s);
cudaError_t launch_mixed_tend_export(const Layout &L, const float *thp, const float *tu, const float *tv,
                                     const MeshF64 &m, double a2, double *op, double *ou, double *ov,
                                     cudaStream_t s);
cudaError_t launch_mixed_diag(const Layout &L, StateMixed st, const float *lohp, const float *lou,
                              const float *lov, const MeshF64 &m, double phibar, double a2, double *partials,
                              int nblocks, cudaStream_t s);


// test support: correctly rounded division by a constant, see ccs_fp64.cu
cudaError_t launch_div_const_check(const double *x, int64_t n, double b, double *out, cudaStream_t s);
// test support: division by a shared divisor from its reciprocal, see ccs_fp64.cu
cudaError_t launch_div_pairs_check(const double *a, const double *b, int64_t n, double *out, cudaStream_t s);
cudaError_t launch_integer_check(int what, const double *a, const double *b, int64_t n, double *out, cudaStream_t s);

// Bounds-checked build (-DCCS_BOUNDS, ccs_bounds.cuh): the first out-of-range index
// the FP64 / mixed kernels met since the last call, (site << 48) | (index & 2^48-1),
// 0 for none; the call clears it.  Always 0 in the normal build.
unsigned long long f64_bounds_take();
unsigned long long mixed_bounds_take();
// one thread checks index i against [0, n) under `site`, accessing nothing (a no-op
// in the normal build)
cudaError_t launch_bounds_selftest(long long i, long long n, int site, cudaStream_t s);

// zero rows after each face wave-speed metric block of the mixed lane (the line
// sweep fetches one face ahead and reads faces past N in partial tiles)
constexpr int kLamPadRows = 32;

// FP64 reductions (mass / energy) over the interior of an FP64 state
cudaError_t launch_f64_diag(const Layout &L, const double *phiG, const double *phi, const double *u,
                            const double *v, const double *uC, const double *vC, const double *sqrtG,
                            const double *phis, double *partials, int nblocks, cudaStream_t s);

}  // namespace ccs
