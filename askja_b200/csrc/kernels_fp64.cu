// FP64 kernel table: the plain double-precision path (the reference's own
// arithmetic, used for parity against the oracle).
#include "kernels.cuh"

namespace askja {

const KernelSet kernels_fp64 = detail::make_set<double>();

size_t partial_doubles(const Lat& L) {
  const long nl = (long)L.V * L.D;
  const size_t plaq = 2 * ((L.V + misc::RED_THREADS - 1) / misc::RED_THREADS);
  const size_t links = 3 * ((nl + misc::RED_THREADS - 1) / misc::RED_THREADS);
  // partial matrices of the Gauss law and their sum
  const size_t gauss = 2 * (size_t)L.N * L.N * (detail::gauss_partials(L) + 1);
  // the warp-MMA reductions: blocks of sites and of links
  const size_t big = !m64_supported(L.N) ? 0
                                         : std::max(2 * (size_t)m64::ctas_for(L.V, m64::sites_per_cta(L.N)),
                                                    3 * (size_t)m64::ctas_for(nl, m64::sites_per_cta(L.N)));
  const size_t fourier = 2 * (size_t)L.n[0];  // FourierTrafo: one plaquette partial per site 0..N0-1
  const size_t pairs = 4 * (size_t)sum_ctas(L);  // energy sums at the two ends of a trajectory
  return std::max({plaq, big, links, gauss, fourier, pairs}) + 64;
}

int sum_ctas(const Lat& L) {
  return m64_supported(L.N) ? m64::ctas_for((long)L.V * L.D, m64::links_per_cta(L.N)) : L.B;
}

int rows_effective_groups(int N, bool fp64, int want) {
  int G;
  size_t smem;
  if (fp64)
    detail::Rows<double>::shape(N, &G, &smem, want);
  else
    detail::Rows<float>::shape(N, &G, &smem, want);
  return G;
}

}  // namespace askja
