// Host-side launch interface between the engine (engine.cu) and the kernels,
// one table per storage precision (kernels_fp64.cu, kernels_fp32.cu).  Every
// entry enqueues work on `stream` and returns the launch status.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "budget.h"
#include "common.cuh"

namespace askja {

// Makes `dev` current for the duration of one API call and gives the caller
// back its own current device on return (every entry point that switches
// devices uses it, so a caller working on another GPU keeps its device).
struct DevGuard {
  int prev = -1;
  explicit DevGuard(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    if (prev != dev) cudaSetDevice(dev);
  }
  ~DevGuard() {
    int cur = -1;
    if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
  }
  DevGuard(const DevGuard&) = delete;
  DevGuard& operator=(const DevGuard&) = delete;
};

struct LineSet;  // lines.cuh

// Launches a kernel that begins with grid_wait() (common.cuh) so that its CTAs
// may be placed while the kernel before it in the stream drains (programmatic
// dependent launch): the start of one MD step hides behind the end of the one
// before.  Everything the kernel reads or writes comes after its grid_wait().
// Graph-replayed us per step: SU(3) 8^4 FP64 6.81 -> 6.56, SU(2) 10^4 FP64
// 6.76 -> 6.01, SU(8) 4^4 FP64 6.62 -> 6.29; nothing to gain on large lattices.
template <typename... P, typename... A>
cudaError_t launch_overlapped(void (*k)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream,
                              A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}

// Flags on the mode of a force launch: each CTA also writes (sum ReTr W, sum
// tr2 P) of its links -- P before the kick with SUMS_OLD, after it with SUMS_NEW
// -- to LaunchCtx::pairs, the old pairs first.  W = U S sums every plaquette
// four times, so the two ends of a trajectory give H without passes of their own
// over the fields.
constexpr int SUMS_OLD = 4, SUMS_NEW = 8;

struct LaunchCtx {
  Lat lat;
  cudaStream_t stream;
  int order;        // effective Taylor order
  int reunit;       // reunitarise after each link update
  int rows_ns;      // row and warp-MMA kernels, FP32: project by one Newton-Schulz step per update (the engine
                    // re-orthonormalises with the determinant phase every few trajectories)
  int force_rows;   // kernel mapping: 0 automatic (thread-per-link for NC <= 4, warp MMA above),
                    // 1 row-per-thread, 4 warp MMA (NC >= 5: FP64, split TF32 for FP32 storage),
                    // 2 tensor cores (FP32, NC = 16, 32 or 64, DIM >= 2), 3 site pairs in
                    // packed FP32 (NC = 3, even n[DIM-1]; the fused kick+drift then
                    // expects the site-pair layout, see pair_swap)
  int rows_groups;  // row kernels: sites per CTA (0: default 128/NC)
  int small_occ;    // thread-per-link kernels: register budget for 0 default, 1 / 2 more resident CTAs
  unsigned* ticket; // zero between reductions (misc::publish)
  double* pairs;    // energy sums of the CTAs (SUMS_OLD / SUMS_NEW)
  unsigned* status; // tensor-core path: nonzero after a bounded wait gave up
  // row-kernel reunitarisation: run only when *gate % gate_every == 0 (null: always)
  const unsigned long long* gate;
  int gate_every;
};

// Trajectories between two full reunitarisation passes (Gram-Schmidt with the
// determinant phase) over U, where the per-update projection leaves drift: the
// tensor-core path and the other FP32 kernels of NC > 4 (Newton-Schulz per update).
constexpr int FULL_REUNIT_EVERY = 10;

// whether the tensor-core mapping exists for this shape and precision
inline bool tc_supported(int N, int D, bool fp64) { return !fp64 && (N == 16 || N == 32 || N == 64) && D >= 2; }

// whether the warp-MMA mapping exists for this colour number
inline bool m64_supported(int N) { return link_major(N); }

// whether the site-pair mapping exists (n_fast: extent of the fastest direction)
inline bool pair_supported(int N, int D, bool fp64, int n_fast) {
  return !fp64 && N == 3 && D >= 2 && n_fast % 2 == 0;
}

// Scalar reductions return their values in device memory:
//   plaq     -> out[0] temporal, out[1] spatial
//   linksums -> out[0] sum tr2(Pa), out[1] sum 1/4 tr2(Pa+Pb), out[2] UViol
//   gauss    -> out[0]
struct KernelSet {
  // mode 0: Pout = Pin - ek F(U); mode 1: also Uout = exp(i ed Pout) U;
  // mode 2 (NC >= 5): Uout = exp(i ed Pin) U; warp MMA also Pout = Pin
  cudaError_t (*force)(const LaunchCtx&, int mode, const void* U, const void* Pin, void* Pout, void* Uout, double ek,
                       double ed);
  // U = exp(i eps P) U in place and Pcopy = P
  cudaError_t (*drift)(const LaunchCtx&, void* U, const void* P, void* Pcopy, double eps);
  cudaError_t (*reunit)(const LaunchCtx&, void* U);
  cudaError_t (*plaq)(const LaunchCtx&, const void* U, double* partial, double* out);
  cudaError_t (*linksums)(const LaunchCtx&, const void* Pa, const void* Pb, const void* U, double* partial,
                          double* out);
  cudaError_t (*gauss)(const LaunchCtx&, const void* U, const void* Pi, double* partial, double* out);
  // |Tr W| / NC of every line of the set
  cudaError_t (*lines)(const LaunchCtx&, const void* U, const LineSet&, double* out);
  cudaError_t (*slice_trace)(const LaunchCtx&, const void* U, double* out);
  // eigenvalues of closed line matrices: ev[q*NC + i] (complex), *fail set on no convergence
  cudaError_t (*line_eigs)(const LaunchCtx&, const void* U, const LineSet&, double2* ev, int* fail);
  cudaError_t (*refresh)(const LaunchCtx&, void* P, uint64_t seed, const unsigned long long* traj_dev,
                         unsigned long long traj_host, double scale);
  cudaError_t (*identity)(const LaunchCtx&, void* U);
  cudaError_t (*gauss_matrices)(const LaunchCtx&, void* U, uint64_t seed);
  cudaError_t (*from_conf)(const LaunchCtx&, const void* conf, void* f);
  cudaError_t (*to_conf)(const LaunchCtx&, const void* f, void* conf);
  // canonical <-> site-pair layout of a field, in place (FP32 only)
  cudaError_t (*pair_swap)(const LaunchCtx&, void* f);
  // FourierTrafo: coef[0..n-1] (partial: 2n doubles of scratch)
  cudaError_t (*fourier)(const LaunchCtx&, const void* U, int n, double* partial, double* coef);
  // Tab for nsites sites from site0 with momenta Pa + Pb: out[k*npt + m]
  cudaError_t (*tab)(const LaunchCtx&, const void* U, const void* Pa, const void* Pb, int site0, int nsites, int npt,
                     double* out);
  // tensor-core path: the give-up path of a bounded wait, on one CTA (tc::k_wait_probe)
  cudaError_t (*wait_probe)(const LaunchCtx&, long long cycles);
};

// size (in doubles) of the partial buffer the reductions need
size_t partial_doubles(const Lat& L);

// CTAs of a force launch of the kernels that take SUMS_OLD / SUMS_NEW
int sum_ctas(const Lat& L);

// sites per CTA the row-per-thread kernels actually use for a requested value
// (0: default), after the thread-count and shared-memory limits
int rows_effective_groups(int N, bool fp64, int want);

extern const KernelSet kernels_fp64;
extern const KernelSet kernels_fp32;

}  // namespace askja
