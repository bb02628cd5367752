// Instantiations of the MMA kernels for one storage type; included by the
// translation units mma64_*.cu, each of which defines a pair of entry points
// for NC a multiple of 8 (FULL) or not.
#pragma once

#include "mma64.cuh"
#include "mma64.h"

#include <type_traits>

namespace askja {
namespace m64 {

template <int NT, bool FULL, typename S2, bool TIGHT>
cudaError_t launch_link(const Job& one, const Grid& g, int ctas, int cur, double ks, int mode, cudaStream_t st) {
  // FP32 storage: the kicks and fused updates in split TF32 where that is as exact
  // (tf32_force), unless the launch also sums the energies (two a trajectory: the
  // sums take FP64 products of the stored links) or only drifts (once a trajectory).
  // Figures beside prod.
  const bool sums = mode & (SUMS_OLD | SUMS_NEW);
  mode &= 3;
  auto k = sums ? k_link<NT, FULL, S2, true, double, TIGHT> : k_link<NT, FULL, S2, false, double, TIGHT>;
  size_t smem = Cta<NT>::SMEM;
  if constexpr (sizeof(S2) == 8) {
    if (!sums && mode != 2 && tf32_force(one.N, one.D)) {
      k = k_link<NT, FULL, S2, false, float, TIGHT>;
      smem = Cta<NT, float>::SMEM;
    }
  }
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  if (g.table) {  // a batch's launches depend on other streams' work: ordinary order
    k<<<ctas, Cta<NT>::THREADS, smem, st>>>(one, g.table, g.items, cur, ks, mode);
    return cudaGetLastError();
  }
  return launch_overlapped(k, ctas, Cta<NT>::THREADS, smem, st, one, g.table, g.items, cur, ks, mode);
}

// a CTA per SM at most: the loose register budget (beside Cta::MIN_CTAS)
template <int NT, bool FULL, typename S2>
cudaError_t launch_link(const Job& one, const Grid& g, int cur, double ks, int mode, cudaStream_t st) {
  const int ctas = g.table ? g.ctas : ctas_for((long)one.V * one.D, Cta<NT>::LINKS);
  if constexpr (NT == 5 || NT == 6)
    if (ctas <= 148) return launch_link<NT, FULL, S2, false>(one, g, ctas, cur, ks, mode, st);
  return launch_link<NT, FULL, S2, true>(one, g, ctas, cur, ks, mode, st);
}

template <int NT, bool FULL, typename S2>
cudaError_t launch_plaq(const Job& one, const Grid& g, int cur, cudaStream_t st) {
  const int ctas = g.table ? g.ctas : ctas_for(one.V, Cta<NT>::SITES);
  k_plaq<NT, FULL, S2><<<ctas, Cta<NT>::PLAQ_THREADS, 0, st>>>(one, g.table, g.items, cur);
  return cudaGetLastError();
}

// the reductions and measurements, by tile count at run time
template <bool FULL, typename S2, typename F>
cudaError_t by_tiles(int NT, F&& f) {
  switch (NT) {
    case 1: return f(std::integral_constant<int, 1>{});
    case 2: return f(std::integral_constant<int, 2>{});
    case 3: return f(std::integral_constant<int, 3>{});
    case 4: return f(std::integral_constant<int, 4>{});
    case 5: return f(std::integral_constant<int, 5>{});
    case 6: return f(std::integral_constant<int, 6>{});
    case 7: return f(std::integral_constant<int, 7>{});
    case 8: return f(std::integral_constant<int, 8>{});
  }
  return cudaErrorInvalidValue;
}

template <bool FULL, typename S2>
cudaError_t launch_uviol(int NT, const Job& one, cudaStream_t st) {
  return by_tiles<FULL, S2>(NT, [&](auto n) {
    constexpr int T = decltype(n)::value;
    k_uviol<T, FULL, S2><<<ctas_for((long)one.V * one.D, Cta<T>::SITES), Cta<T>::PLAQ_THREADS, 0, st>>>(one);
    return cudaGetLastError();
  });
}

template <bool FULL, typename S2>
cudaError_t launch_gauss(int NT, const Job& one, int groups, cudaStream_t st) {
  return by_tiles<FULL, S2>(NT, [&](auto n) {
    constexpr int T = decltype(n)::value;
    k_gauss<T, FULL, S2><<<ctas_for(groups, Cta<T>::SITES), Cta<T>::PLAQ_THREADS, 0, st>>>(one, groups);
    return cudaGetLastError();
  });
}

template <bool FULL, typename S2>
cudaError_t launch_lines(int NT, const Lat& L, const void* U, const LineSet& ls, double* out, double2* ev, int* fail,
                         cudaStream_t st) {
  return by_tiles<FULL, S2>(NT, [&](auto n) {
    constexpr int T = decltype(n)::value;
    auto k = k_lines<T, FULL, S2>;
    const size_t smem = ev ? (size_t)(L.N * L.N + 2 * L.N) * sizeof(cpx<double>) : 0;
    if (smem > 48 * 1024) {
      const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
    }
    k<<<ls.lines(), 32 * T, smem, st>>>(L, static_cast<const S2*>(U), ls, out, ev, fail);
    return cudaGetLastError();
  });
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
  }                                                                                                              \
  cudaError_t uviol_##SUFFIX(int NT, const Job& one, cudaStream_t st) {                                          \
    return launch_uviol<FULL, S2>(NT, one, st);                                                                  \
  }                                                                                                              \
  cudaError_t gauss_##SUFFIX(int NT, const Job& one, int groups, cudaStream_t st) {                              \
    return launch_gauss<FULL, S2>(NT, one, groups, st);                                                          \
  }                                                                                                              \
  cudaError_t lines_##SUFFIX(int NT, const Lat& L, const void* U, const LineSet& ls, double* out, double2* ev,   \
                             int* fail, cudaStream_t st) {                                                       \
    return launch_lines<FULL, S2>(NT, L, U, ls, out, ev, fail, st);                                              \
  }

#define ASKJA_M64_DECLARE(SUFFIX)                                                                     \
  cudaError_t link_##SUFFIX(int NT, const Job&, const Grid&, int cur, double ks, int mode, cudaStream_t); \
  cudaError_t plaq_##SUFFIX(int NT, const Job&, const Grid&, int cur, cudaStream_t);                  \
  cudaError_t uviol_##SUFFIX(int NT, const Job&, cudaStream_t);                                       \
  cudaError_t gauss_##SUFFIX(int NT, const Job&, int groups, cudaStream_t);                           \
  cudaError_t lines_##SUFFIX(int NT, const Lat&, const void* U, const LineSet&, double* out, double2* ev, int* fail, \
                             cudaStream_t);

ASKJA_M64_DECLARE(full64)
ASKJA_M64_DECLARE(part64)
ASKJA_M64_DECLARE(full32)
ASKJA_M64_DECLARE(part32)

}  // namespace m64
}  // namespace askja
