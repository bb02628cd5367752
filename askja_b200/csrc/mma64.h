// Launches of the warp-MMA kernels (mma64.cuh: FP64, and split TF32 for FP32
// storage) for 5 <= NC <= 64: one lattice by value (table null), or the CTAs of
// many lattices of one colour number through a job table and a per-CTA list of
// (job, block).
#pragma once

#include <cuda_runtime.h>

namespace askja {
namespace m64 {

struct Job;

}  // namespace m64

struct Lat;
struct LineSet;

namespace m64 {

struct Grid {
  const Job* table = nullptr;   // device
  const int2* items = nullptr;  // device
  int ctas = 0;                 // with a table: entries of items
};

// links (k_link), sites (k_plaq) and links (k_kinetic) per CTA
int links_per_cta(int N);
int sites_per_cta(int N);
int kinetic_links_per_cta(int N);
inline int ctas_for(long n, int per) { return (int)((n + per - 1) / per); }

// FP32 storage: whether the kicks and fused updates multiply in split TF32 (else
// on the FP64 MMA), and how: 0 one accumulator for both MMAs of an 8-column step,
// 1 one each, added in FP32, 2 also the mean of their truncation put back
// (prod<float>, mma64.cuh).  The rule is that a force is no further from 64 bits
// than FP32 FMAs put it, whose error grows with NC and with the number of staples:
// rms error of a force of Haar links over the force's, x 1e-7, in 2, 3 and 4
// dimensions, FP32 row kernels | split as 0 | as 1 | as 2
//   NC = 5   1.19 1.45 1.63 | 2.07 2.19 2.20 | 1.75 1.91 1.91 | 1.66 1.72 1.72
//        6   1.27 1.57 1.80 | 2.24 2.24 2.26 | 1.88 1.89 1.97 | 1.62 1.63 1.73
//        7   1.38 1.74 1.93 | 2.24 2.29 2.27 | 1.88 1.94 1.96 | 1.61 1.66 1.68
//        8   1.52 1.80 2.05 | 2.24 2.28 2.30 | 1.91 1.94 1.97 | 1.61 1.64 1.70
//       10   1.65 2.02 2.30 | 2.15 2.24 2.28 | 1.87 1.96 1.99 | 1.70 1.75 1.80
//       11   1.72 2.08 2.42 | 2.22 2.24 2.29 | 1.89 1.94 2.01 | 1.66 1.75 1.82
//       16   2.05 2.52 2.90 | 2.27 2.33 2.38 | 1.96 2.02 2.07 | 1.67 1.73 1.79
//       17   2.13 2.59 2.99 | 2.30 2.34 2.41 | 2.00 2.05 2.13
//       24   2.53 3.07 3.54 | 2.34 2.39 2.45
//       57   3.84 4.69 5.41 | 2.49 2.60 2.71
// (the FP64 MMA: 0.3).
inline bool tf32_force(int N, int D) { return N >= (D > 2 ? 7 : 11); }
constexpr int fine_force(int NT, bool full) {
  return NT == 1 || (NT == 2 && !full) ? 2 : NT == 2 || (NT == 3 && !full) ? 1 : 0;
}

// mode 0 kick, 1 kick + drift, 2 drift (mma64.cuh); fp64: storage.  With a table
// (which holds jobs of one value of tf32_force) only N and D of `one` are read.
cudaError_t link(int N, bool fp64, const Job& one, const Grid& g, int cur, double kick_scale, int mode,
                 cudaStream_t stream);
cudaError_t plaq(int N, bool fp64, const Job& one, const Grid& g, int cur, cudaStream_t stream);
// unitarity sum of U[0]
cudaError_t uviol(int N, bool fp64, const Job& one, cudaStream_t stream);
// Gauss-law matrices of `groups` groups of links of U[0] and Pin, at kin_partial
int gauss_groups(int N, long nlinks);
cudaError_t gauss(int N, bool fp64, const Job& one, cudaStream_t stream);
// |Tr| / NC of the lines (out) or their eigenvalues (ev, fail)
cudaError_t lines(bool fp64, const Lat& L, const void* U, const LineSet& ls, double* out, double2* ev, int* fail,
                  cudaStream_t stream);
// kinetic sums of Pin (and Pin2); every colour number in one launch
cudaError_t kinetic(bool fp64, const Job& one, const Grid& g, cudaStream_t stream);

}  // namespace m64
}  // namespace askja
