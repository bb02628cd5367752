// Launches of the FP64-MMA kernels (mma64.cuh) for 5 <= NC <= 64: one lattice
// by value (table null), or the CTAs of many lattices of one colour number
// through a job table and a per-CTA list of (job, block).
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

// mode 0 kick, 1 kick + drift, 2 drift (mma64.cuh); fp64: storage
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
