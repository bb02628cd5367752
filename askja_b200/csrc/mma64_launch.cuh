// Instantiations of the FP64-MMA kernels for one storage type; included by the
// translation units mma64_*.cu, each of which defines a pair of entry points
// for NC a multiple of 8 (FULL) or not.
#pragma once

#include "mma64.cuh"
#include "mma64.h"

namespace askja {
namespace m64 {

template <int NT, bool FULL, typename S2>
cudaError_t launch_link(const Job& one, const Grid& g, int cur, double ks, int mode, cudaStream_t st) {
  auto k = k_link<NT, FULL, S2>;
  const size_t smem = Cta<NT>::SMEM;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const int ctas = g.table ? g.ctas : ctas_for((long)one.V * one.D, Cta<NT>::LINKS);
  k<<<ctas, Cta<NT>::THREADS, smem, st>>>(one, g.table, g.items, cur, ks, mode);
  return cudaGetLastError();
}

template <int NT, bool FULL, typename S2>
cudaError_t launch_plaq(const Job& one, const Grid& g, int cur, cudaStream_t st) {
  const int ctas = g.table ? g.ctas : ctas_for(one.V, Cta<NT>::LINKS);
  k_plaq<NT, FULL, S2><<<ctas, Cta<NT>::THREADS, 0, st>>>(one, g.table, g.items, cur);
  return cudaGetLastError();
}

#define ASKJA_M64_ENTRIES(SUFFIX, FULL, S2)                                                                      \
  cudaError_t link_##SUFFIX(int NT, const Job& one, const Grid& g, int cur, double ks, int mode, cudaStream_t st) { \
    switch (NT) {                                                                                                \
      case 1: return launch_link<1, FULL, S2>(one, g, cur, ks, mode, st);                                        \
      case 2: return launch_link<2, FULL, S2>(one, g, cur, ks, mode, st);                                        \
      case 3: return launch_link<3, FULL, S2>(one, g, cur, ks, mode, st);                                        \
      case 4: return launch_link<4, FULL, S2>(one, g, cur, ks, mode, st);                                        \
      case 5: return launch_link<5, FULL, S2>(one, g, cur, ks, mode, st);                                        \
      case 6: return launch_link<6, FULL, S2>(one, g, cur, ks, mode, st);                                        \
      case 7: return launch_link<7, FULL, S2>(one, g, cur, ks, mode, st);                                        \
      case 8: return launch_link<8, FULL, S2>(one, g, cur, ks, mode, st);                                        \
    }                                                                                                            \
    return cudaErrorInvalidValue;                                                                                \
  }                                                                                                              \
  cudaError_t plaq_##SUFFIX(int NT, const Job& one, const Grid& g, int cur, cudaStream_t st) {                   \
    switch (NT) {                                                                                                \
      case 1: return launch_plaq<1, FULL, S2>(one, g, cur, st);                                                  \
      case 2: return launch_plaq<2, FULL, S2>(one, g, cur, st);                                                  \
      case 3: return launch_plaq<3, FULL, S2>(one, g, cur, st);                                                  \
      case 4: return launch_plaq<4, FULL, S2>(one, g, cur, st);                                                  \
      case 5: return launch_plaq<5, FULL, S2>(one, g, cur, st);                                                  \
      case 6: return launch_plaq<6, FULL, S2>(one, g, cur, st);                                                  \
      case 7: return launch_plaq<7, FULL, S2>(one, g, cur, st);                                                  \
      case 8: return launch_plaq<8, FULL, S2>(one, g, cur, st);                                                  \
    }                                                                                                            \
    return cudaErrorInvalidValue;                                                                                \
  }

#define ASKJA_M64_DECLARE(SUFFIX)                                                                     \
  cudaError_t link_##SUFFIX(int NT, const Job&, const Grid&, int cur, double ks, int mode, cudaStream_t); \
  cudaError_t plaq_##SUFFIX(int NT, const Job&, const Grid&, int cur, cudaStream_t);

ASKJA_M64_DECLARE(full64)
ASKJA_M64_DECLARE(part64)
ASKJA_M64_DECLARE(full32)
ASKJA_M64_DECLARE(part32)

}  // namespace m64
}  // namespace askja
