// Launches of the FP64-MMA kernels (mma64.cuh) for 5 <= NC <= 64: one lattice
// by value (table null), or the CTAs of many lattices of one colour number
// through a job table and a per-CTA list of (job, block).
#pragma once

#include <cuda_runtime.h>

namespace askja {
namespace m64 {

struct Job;

struct Grid {
  const Job* table = nullptr;   // device
  const int2* items = nullptr;  // device
  int ctas = 0;                 // with a table: entries of items
};

// links (k_link) or sites (k_plaq) and links (k_kinetic) per CTA
int links_per_cta(int N);
int kinetic_links_per_cta(int N);
inline int ctas_for(long n, int per) { return (int)((n + per - 1) / per); }

// mode 0 kick, 1 kick + drift, 2 drift (mma64.cuh); fp64: storage
cudaError_t link(int N, bool fp64, const Job& one, const Grid& g, int cur, double kick_scale, int mode,
                 cudaStream_t stream);
cudaError_t plaq(int N, bool fp64, const Job& one, const Grid& g, int cur, cudaStream_t stream);
// kinetic sums of Pin at kin_partial[stride * block]; every colour number in one launch
cudaError_t kinetic(bool fp64, const Job& one, const Grid& g, int stride, cudaStream_t stream);

}  // namespace m64
}  // namespace askja
