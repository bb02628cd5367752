// Register budgets of the thread-per-link kernels (NC <= 4) by the size of the
// lattice.  Host rules only, no device code.
#pragma once

namespace askja {

inline long site_tiles(long V) { return (V + 31) / 32; }

// FP64, budget 0: whether the kernel runs that has the links of the next staple
// in flight (small::k_force_ahead, two CTAs per SM).  Where the lattice has no
// more CTAs than that it wins, above the plain kernel's resident CTAs hide the
// loads.  us per graph-replayed step, ahead / plain: SU(3) 8^4 5.6 / 6.3, 16^3
// 4.3 / 5.2, 10^4 12.2 / 11.0, 32^4 954 / 909; SU(2) 24^2 3.8 / 4.5, 8^4 5.1 / 6.3,
// 12^4 10.3 / 9.6, 16^4 22.1 / 20.9, 24^4 122 / 105, 32^4 375 / 329.
inline bool force_ahead(int N, long V) { return N <= 3 && site_tiles(V) <= 2 * 148; }

// Untuned register budget (LaunchCtx::small_occ).  Measured us per step at budget 0 and 2:
//  FP32 (residual planes), NC = 2, 3: with more tiles than four CTAs per SM
//   hold, the tight budget's resident warps hide more latency (SU(3) 32^4 469 /
//   443, SU(2) 16^4 15.5 / 12.9); below, the loose one's extra loads in flight win
//   (SU(3) 12^4 11.3 / 11.1, 10^4 7.4 / 8.4, 8^4 4.5 / 6.5).  NC = 4 spills at 2.
//  FP64, NC = 2: the budgets are the other way round (80 and 126 registers).  Up
//   to two CTAs per SM force_ahead (budget 0) wins, 24^2 3.8 / 4.0, 8^4 5.1 / 5.3;
//   then as the last wave falls, 32^3 9.1 / 9.1, 16^4 20.9 / 20.3; from 2048 tiles
//   on the plain kernel, 48^3 21.2 / 22.0, 20^4 56.7 / 57.5, 64^3 52.4 / 57.3, 32^4
//   329 / 352.  NC = 3: no difference.
inline int default_occupancy(int N, bool fp64, bool residual, long V) {
  const long tiles = site_tiles(V);
  if (fp64) return N == 2 && !force_ahead(N, V) && tiles <= 2048 ? 2 : 0;
  return residual && N <= 3 && tiles > 4 * 148 ? 2 : 0;
}

// A mapping tuned on one lattice serves later ones of the same (NC, DIM,
// precision); the thread-per-link budget (path 0) is carried only to lattices on
// the same side of the rules above, others take their own untuned one.
// Otherwise tuning FP32 SU(3) 8^4 (budget 0) cost every later 32^4 6 %, the reverse
// every later 8^4 44 %.
inline int carried_occupancy(int tuned, int path, int N, bool fp64, bool residual, long V_tuned, long V) {
  if (path != 0) return tuned;
  const int here = default_occupancy(N, fp64, residual, V);
  const bool same = here == default_occupancy(N, fp64, residual, V_tuned) &&
                    (!fp64 || force_ahead(N, V) == force_ahead(N, V_tuned));
  return same ? tuned : here;
}

}  // namespace askja
