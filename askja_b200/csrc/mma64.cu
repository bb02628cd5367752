// Dispatch of the warp-MMA kernels over storage type and tile count.
#include "mma64_launch.cuh"

namespace askja {
namespace m64 {

int links_per_cta(int N) {
  const int NT = (N + 7) / 8;
  return NT == 1 ? Cta<1>::LINKS : NT == 2 ? Cta<2>::LINKS : 1;
}

int sites_per_cta(int N) {
  switch ((N + 7) / 8) {
    case 1: return Cta<1>::SITES;
    case 2: return Cta<2>::SITES;
    case 3: return Cta<3>::SITES;
    case 4: return Cta<4>::SITES;
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

cudaError_t uviol(int N, bool fp64, const Job& one, cudaStream_t st) {
  const int NT = (N + 7) / 8;
  if (N % 8 == 0) return (fp64 ? uviol_full64 : uviol_full32)(NT, one, st);
  return (fp64 ? uviol_part64 : uviol_part32)(NT, one, st);
}

// enough warps for the chip (about 24 a SM, 8 for the large matrices), one group per link at most
int gauss_groups(int N, long nlinks) {
  const int NT = (N + 7) / 8;
  const long most = 148L * (NT <= 4 ? 24 / NT : 1);
  return (int)(nlinks < most ? nlinks : most);
}

cudaError_t gauss(int N, bool fp64, const Job& one, cudaStream_t st) {
  const int NT = (N + 7) / 8, groups = gauss_groups(N, (long)one.V * one.D);
  if (N % 8 == 0) return (fp64 ? gauss_full64 : gauss_full32)(NT, one, groups, st);
  return (fp64 ? gauss_part64 : gauss_part32)(NT, one, groups, st);
}

cudaError_t lines(bool fp64, const Lat& L, const void* U, const LineSet& ls, double* out, double2* ev, int* fail,
                  cudaStream_t st) {
  const int NT = (L.N + 7) / 8;
  if (L.N % 8 == 0) return (fp64 ? lines_full64 : lines_full32)(NT, L, U, ls, out, ev, fail, st);
  return (fp64 ? lines_part64 : lines_part32)(NT, L, U, ls, out, ev, fail, st);
}

cudaError_t kinetic(bool fp64, const Job& one, const Grid& g, cudaStream_t st) {
  const int ctas = g.table ? g.ctas : ctas_for((long)one.V * one.D, kin_links(one.N));
  if (fp64)
    k_kinetic<double2><<<ctas, misc::RED_THREADS, 0, st>>>(one, g.table, g.items);
  else
    k_kinetic<float2><<<ctas, misc::RED_THREADS, 0, st>>>(one, g.table, g.items);
  return cudaGetLastError();
}

}  // namespace m64
}  // namespace askja
