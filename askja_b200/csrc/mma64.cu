// Dispatch of the FP64-MMA kernels over storage type and tile count.
#include "mma64_launch.cuh"

namespace askja {
namespace m64 {

int links_per_cta(int N) {
  switch ((N + 7) / 8) {
    case 1: return Cta<1>::LINKS;
    case 2: return Cta<2>::LINKS;
    case 3: return Cta<3>::LINKS;
    case 4: return Cta<4>::LINKS;
    default: return 1;
  }
}

int kinetic_links_per_cta(int N) { return kin_links(N); }

cudaError_t link(int N, bool fp64, const Job& one, const Grid& g, int cur, double ks, int mode, cudaStream_t st) {
  const int NT = (N + 7) / 8;
  if (N % 8 == 0) return (fp64 ? link_full64 : link_full32)(NT, one, g, cur, ks, mode, st);
  return (fp64 ? link_part64 : link_part32)(NT, one, g, cur, ks, mode, st);
}

cudaError_t plaq(int N, bool fp64, const Job& one, const Grid& g, int cur, cudaStream_t st) {
  const int NT = (N + 7) / 8;
  if (N % 8 == 0) return (fp64 ? plaq_full64 : plaq_full32)(NT, one, g, cur, st);
  return (fp64 ? plaq_part64 : plaq_part32)(NT, one, g, cur, st);
}

cudaError_t kinetic(bool fp64, const Job& one, const Grid& g, int stride, cudaStream_t st) {
  const int ctas = g.table ? g.ctas : ctas_for((long)one.V * one.D, kin_links(one.N));
  if (fp64)
    k_kinetic<double2><<<ctas, misc::RED_THREADS, 0, st>>>(one, g.table, g.items, stride);
  else
    k_kinetic<float2><<<ctas, misc::RED_THREADS, 0, st>>>(one, g.table, g.items, stride);
  return cudaGetLastError();
}

}  // namespace m64
}  // namespace askja
