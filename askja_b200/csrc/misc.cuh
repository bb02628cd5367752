// Reductions, measurements, momentum refresh, hot start and the Metropolis
// step.  Every reduction accumulates in FP64 whatever the storage precision
// of the links (FP32 links are promoted on load) and writes one partial per
// block; the last block to do so sums them in block order (publish; a pass of
// one block, k_finish, in static_plaq.cu), so results are deterministic run to
// run.
//
// The reductions take the colour number, 2 to 4, as a template parameter NT and
// are fully unrolled; those of NC >= 5 are in mma64.cuh.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"

namespace askja {
namespace misc {

constexpr int RED_THREADS = 256;

// Block-wide sum of K doubles; thread 0 gets the result.
template <int K>
__device__ __forceinline__ void block_sum(double (&v)[K]) {
  __shared__ double sh[K][RED_THREADS / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; k++) {
    double x = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) sh[k][wid] = x;
  }
  __syncthreads();
  if (wid == 0) {
#pragma unroll
    for (int k = 0; k < K; k++) {
      double x = lane < (int)(blockDim.x >> 5) ? sh[k][lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      v[k] = x;
    }
  }
  __syncthreads();
}

// Sum nblocks partials of width K (layout partial[b*K + k]) into out[k].
template <int K>
__global__ void k_finish(const double* __restrict__ partial, int nblocks, double* __restrict__ out) {
  double v[K];
#pragma unroll
  for (int k = 0; k < K; k++) v[k] = 0.0;
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x)
#pragma unroll
    for (int k = 0; k < K; k++) v[k] += partial[(size_t)b * K + k];
  block_sum<K>(v);
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < K; k++) out[k] = v[k];
}

// Writes this block's K sums (in thread 0) to the partials and lets the last
// block to do so add them up, in block order whatever the finishing order, into
// out (not null): no launch of its own for the total.  *ticket counts the
// blocks, zero before and after.  Without a ticket k_finish adds the partials up,
// in the same order (one_launch).
template <int K>
__device__ __forceinline__ void publish(const double (&v)[K], double* __restrict__ partial, double* __restrict__ out,
                                        unsigned* ticket) {
  __shared__ bool last;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < K; k++) partial[(size_t)blockIdx.x * K + k] = v[k];
    if (!ticket) return;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  if (!ticket) return;
  __syncthreads();
  if (!last) return;
  __threadfence();
  double s[K];
#pragma unroll
  for (int k = 0; k < K; k++) s[k] = 0.0;
#pragma unroll 8
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
#pragma unroll
    for (int k = 0; k < K; k++) s[k] += __ldcg(partial + (size_t)b * K + k);
  block_sum<K>(s);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < K; k++) out[k] = s[k];
    *ticket = 0;
  }
}

// The ticket for a reduction of nb blocks by KERNEL, or none above so many waves of
// its resident blocks.  A block waits for its fence and its number before it leaves
// its SM, about 1.2 us of each wave, unless other blocks' loads fill that time; the
// launch of k_finish takes 1 to 3 us.
template <auto KERNEL>
unsigned* one_launch(unsigned nb, unsigned waves, unsigned* ticket) {
  static const unsigned resident = [] {
    int n = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, KERNEL, RED_THREADS, 0) == cudaSuccess ? n : 1;
  }();
  return nb <= (size_t)waves * 148 * resident ? ticket : nullptr;
}
// The waves, us a call with a ticket / without.  FP64 fields: SU(2) 32^4 kinetic
// (15 waves) 91 / 96, SU(3) 24^4 57.1 / 58.5, 32^4 plaquettes (14) 263 / 260; SU(4)
// 16^4 kinetic (3.5) 32.2 / 34.6, 24^4 (17) 90.8 / 81.1.  FP32: plaquettes SU(3) 24^4
// (4.4) 139.7 / 141.8, 32^4 (14) 373 / 364; kinetic SU(2) 24^4 (4.4) 40.4 / 42.8, 32^4
// (14) 90 / 80; SU(3) 24^4 (7) 53.0 / 46.1, 32^4 121 / 105; UViol SU(4) 16^4 (2.3) 40.4
// / 33.1.
constexpr unsigned ticket_waves(bool fp64, int N, bool links) {
  return fp64 ? (N <= 3 ? 1u << 20 : 4) : N == 2 || !links ? 5 : 2;
}
// The sums of a reduction that had no ticket.
template <int K>
cudaError_t total(unsigned nb, const double* partial, double* out, const unsigned* ticket, cudaStream_t st) {
  if (!ticket) k_finish<K><<<1, RED_THREADS, 0, st>>>(partial, (int)nb, out);
  return cudaGetLastError();
}

// Plaquette sums per site (sun.cpp:507-537 EnergyMag; measurements4d.cpp:885-927
// PlaqExp).  partial[b*2 + 0] = temporal planes (0,k), [b*2+1] = spatial (j,k), j>=1.
// ReTr(A B C^dag D^dag) is evaluated as Re sum_ij (AB)_ij conj((DC)_ij).
template <int NT, typename S2>
__device__ __forceinline__ void plaq_site(const Lat& L, const S2* __restrict__ U, int s, double (&v)[2]) {
  constexpr int N = NT;
  if (s < L.V && counted(L, s)) {
    for (int mu = 0; mu < L.D; mu++) {
      const int xpmu = nb_plus(L, mu, s);
      for (int nu = mu + 1; nu < L.D; nu++) {
        const int xpnu = nb_plus(L, nu, s);
        double tr = 0.0;
#pragma unroll
        for (int i = 0; i < N; i++)
#pragma unroll
          for (int j = 0; j < N; j++) {
            cpx<double> ab = czero<double>(), dc = czero<double>();
#pragma unroll
            for (int k = 0; k < N; k++) {
              cmac(ab, ldc<double>(U + eoffn<NT>(L, mu, i * N + k, s)), ldc<double>(U + eoffn<NT>(L, nu, k * N + j, xpmu)));
              cmac(dc, ldc<double>(U + eoffn<NT>(L, nu, i * N + k, s)), ldc<double>(U + eoffn<NT>(L, mu, k * N + j, xpnu)));
            }
            // explicit fma: the same rounding in every kernel that inlines this
            tr = fma(ab.re, dc.re, tr);
            tr = fma(ab.im, dc.im, tr);
          }
        v[mu == 0 ? 0 : 1] += 1.0 - tr / N;
      }
    }
  }
}

template <int NT, typename S2>
__global__ void __launch_bounds__(RED_THREADS) k_plaq(Lat L, const S2* __restrict__ U, double* __restrict__ partial,
                                                      double* __restrict__ out, unsigned* ticket) {
  double v[2] = {0.0, 0.0};
  plaq_site<NT, S2>(L, U, blockIdx.x * blockDim.x + threadIdx.x, v);
  block_sum<2>(v);
  publish<2>(v, partial, out, ticket);
}

// Per-link sums: [0] = sum ReTr(A A) for A = Pa (sun.cpp:540-548 simpleenergyEl),
// [1] = sum 1/4 ReTr((Pa+Pb)^2) (sun.cpp:560-567 EnergyEl, when Pb != null),
// [2] = sum ReTr((U U^dag - 1)^2) (sun.cpp:441-471 UViol, when U != null).
template <int NT, typename S2>
__device__ __forceinline__ void link_sums(const Lat& L, const S2* __restrict__ Pa, const S2* __restrict__ Pb,
                                          const S2* __restrict__ U, long t, double (&v)[3]) {
  constexpr int N = NT;
  if (t < (long)L.V * L.D && counted(L, (int)(t % L.V))) {
    const int d = (int)(t / L.V);
    const int s = (int)(t - (long)d * L.V);
    if (Pa) {
      double a = 0.0, b = 0.0;
#pragma unroll
      for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = 0; j < N; j++) {
          const cpx<double> x = ldc<double>(Pa + eoffn<NT>(L, d, i * N + j, s));
          const cpx<double> y = ldc<double>(Pa + eoffn<NT>(L, d, j * N + i, s));
          a = fma(x.re, y.re, a);
          a = fma(-x.im, y.im, a);
          if (Pb) {
            const cpx<double> x2 = ldc<double>(Pb + eoffn<NT>(L, d, i * N + j, s));
            const cpx<double> y2 = ldc<double>(Pb + eoffn<NT>(L, d, j * N + i, s));
            b = fma(x.re + x2.re, y.re + y2.re, b);
            b = fma(-(x.im + x2.im), y.im + y2.im, b);
          }
        }
      v[0] = a;
      v[1] = 0.25 * b;
    }
    if (U) {
      double c = 0.0;
      // FP64 links are held whole (24^4: SU(3) 70 -> 58 us a call, SU(4) 111 -> 86); FP32 ones, promoted, would
      // cost a resident block, and are read again from L1
      constexpr bool HOLD = sizeof(S2) == 16 && N > 2;
      cpx<double> m[HOLD ? N * N : 1];
      if constexpr (HOLD)
#pragma unroll
        for (int i = 0; i < N * N; i++) m[i] = ldc<double>(U + eoffn<NT>(L, d, i, s));
      auto u = [&](int i, int k) {
        if constexpr (HOLD)
          return m[i * N + k];
        else
          return ldc<double>(U + eoffn<NT>(L, d, i * N + k, s));
      };
#pragma unroll
      for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = 0; j < N; j++) {
          cpx<double> aij = czero<double>(), aji = czero<double>();
#pragma unroll
          for (int k = 0; k < N; k++) {
            cmac_nc(aij, u(i, k), u(j, k));
            cmac_nc(aji, u(j, k), u(i, k));
          }
          if (i == j) {
            aij.re -= 1.0;
            aji.re -= 1.0;
          }
          c = fma(aij.re, aji.re, c);
          c = fma(-aij.im, aji.im, c);
        }
      v[2] = c;
    }
  }
}

template <int NT, typename S2>
__global__ void __launch_bounds__(RED_THREADS) k_linksums(Lat L, const S2* __restrict__ Pa, const S2* __restrict__ Pb,
                                                          const S2* __restrict__ U, double* __restrict__ partial,
                                                          double* __restrict__ out, unsigned* ticket) {
  double v[3] = {0.0, 0.0, 0.0};
  link_sums<NT, S2>(L, Pa, Pb, U, (long)blockIdx.x * blockDim.x + threadIdx.x, v);
  block_sum<3>(v);
  publish<3>(v, partial, out, ticket);
}

// Slice averages for measurements4d.cpp:357-408 scalarLoopcorr:
// out[x0] = mean over the x0-slice of ReTr U_{D-1} / NC.  Blocked fields: one CTA
// per slice, of as many threads as there may be: the slices are few and their loads
// are all the kernel does (SU(3) 16^4: 22 us with 256 threads).
constexpr int SLICE_THREADS = 1024;
template <typename S2>
__global__ void __launch_bounds__(SLICE_THREADS) k_slice_trace(Lat L, const S2* __restrict__ U,
                                                               double* __restrict__ out) {
  __shared__ double sh[SLICE_THREADS / 32];
  const int N = L.N;
  const int slice = L.stride[0];
  double v = 0.0;
  for (int s = blockIdx.x * slice + threadIdx.x; s < (blockIdx.x + 1) * slice; s += SLICE_THREADS) {
    const S2* p = U + bbase(L, L.D - 1, s);
    double t = 0.0;
    for (int k = 0; k < N; k++) t += (double)p[(size_t)k * (N + 1) * 32].x;
    v += t / N;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = sh[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) out[blockIdx.x] = v / slice;
  }
}

// The same for link-major fields, where a diagonal element lies in a sector of its
// own: a cluster of CTAs per slice, since one SM fetches sectors too slowly, and a
// thread per element (us a call, with a CTA per slice and a thread per site / so:
// SU(12) 8^4 30 / 25.7, SU(32) 6^4 30 / 26, SU(64) 4^4 30 / 23).
constexpr int SLICE_CTAS = 8;
template <typename S2>
__global__ void __cluster_dims__(SLICE_CTAS, 1, 1) __launch_bounds__(RED_THREADS)
    k_slice_trace_major(Lat L, const S2* __restrict__ U, double* __restrict__ out) {
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  __shared__ double part;
  const int N = L.N, slice = L.stride[0], x0 = blockIdx.x / SLICE_CTAS;
  const S2* p = U + mbase(L, L.D - 1, x0 * slice);
  const long n = (long)slice * N;
  double v[1] = {0.0};
#pragma unroll 4
  for (long q = (long)cluster.block_rank() * RED_THREADS + threadIdx.x; q < n; q += SLICE_CTAS * RED_THREADS) {
    const long s = q / N;
    v[0] += (double)p[s * (N * N) + (q - s * N) * (N + 1)].x;
  }
  block_sum<1>(v);
  if (threadIdx.x == 0) part = v[0];
  cluster.sync();
  if (cluster.block_rank() == 0 && threadIdx.x == 0) {
    double t = 0.0;
    for (int r = 0; r < SLICE_CTAS; r++) t += *cluster.map_shared_rank(&part, r);
    out[x0] = t / ((double)N * slice);
  }
  cluster.sync();  // the others' shared memory stays until it has been read
}

// Momentum refresh (sun.cpp:209-252 initializeE with the reference's
// generator basis, sun.cpp:142-189): P = scale * sum_a xi_a T_a,
// scale = sqrt(2 NC / beta).  xi_a are Philox normals: link l = s*D + d
// (U-conf order), block j = a/4, counter (j, l_lo, l_hi, traj), key = seed.
// The explicit basis: for the p-th pair i<j (row-major), T_2p has 1/2 at
// (i,j),(j,i); T_2p+1 has -i/2 at (i,j), +i/2 at (j,i); the m-th diagonal
// generator is norm_m * diag(1,..,1 (m+1 times), -(m+1), 0, ..),
// norm_m = sqrt(1 / (2 (m+1)(m+2))).
// The entries of one link's momentum in generation order: emit(i, j, value)
// for the upper and lower entry of every off-diagonal pair, then the diagonal
// from the last row up.  Shared by the matrix refresh below and the refresh of
// the residual-plane FP32 mode (split.cuh), so both draw identical momenta.
template <typename Emit>
__device__ __forceinline__ void refresh_entries(const Lat& L, uint64_t seed, uint32_t traj, double scale, int d, int s,
                                                Emit&& emit) {
  const int N = L.N;
  const unsigned long long lk = (unsigned long long)s * L.D + d;
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  int cur_blk = -1;
  double g[4];
  auto normal = [&](int a) -> double {
    const int blk = a >> 2;
    if (blk != cur_blk) {
      u32x4 c;
      c.x = (uint32_t)blk;
      c.y = (uint32_t)lk;
      c.z = (uint32_t)(lk >> 32);
      c.w = traj;
      normals4(philox4x32_10(c, k0, k1), g);
      cur_blk = blk;
    }
    return g[a & 3];
  };
  int p = 0;
  for (int i = 0; i < N; i++)
    for (int j = i + 1; j < N; j++, p++) {
      const double xs = normal(2 * p), xa = normal(2 * p + 1);
      emit(i, j, mkc<double>(0.5 * scale * xs, -0.5 * scale * xa));
      emit(j, i, mkc<double>(0.5 * scale * xs, 0.5 * scale * xa));
    }
  // diagonal: P_dd = scale * (S_d - d * norm_{d-1} xi_{d-1}),  S_d = sum_{m>=d} norm_m xi_m
  const int a0 = N * (N - 1);
  double suffix = 0.0;
  for (int dd = N - 1; dd >= 0; dd--) {
    double val = suffix;
    if (dd >= 1) {
      const int m = dd - 1;
      const double nm = sqrt(0.5 / ((double)(m + 1) * (m + 2)));
      const double xm = normal(a0 + m);
      val -= dd * nm * xm;
      suffix += nm * xm;
    }
    emit(dd, dd, mkc<double>(scale * val, 0.0));
  }
}

template <typename S2>
__device__ __forceinline__ void refresh_link(const Lat& L, S2* __restrict__ P, uint64_t seed, uint32_t traj,
                                             double scale, long t) {
  if (t >= (long)L.V * L.D) return;
  const int N = L.N;
  const int d = (int)(t / L.V);
  const int s = (int)(t - (long)d * L.V);
  S2* p = P + bbase(L, d, s);
  refresh_entries(L, seed, traj, scale, d, s,
                  [&](int i, int j, const cpx<double>& v) { stc(p + (i * N + j) * 32, v); });
}

// refresh_link for link-major fields, a thread per Philox block: block b of a
// link holds the normals of the off-diagonal pairs 2b and 2b + 1, and one more
// thread per link (in warps of their own, after all pairs) draws the diagonal.
// The same draws and arithmetic per entry, so the momenta are identical.  What
// bounds it is the FP64 log / sqrt / sincospi of each block; a CTA per link left
// most threads on the empty lower triangle and all of them behind the serial
// diagonal (SU(64) 4x8x16 138 us, SU(32) 8^4 414 us).
__host__ __device__ inline int refresh_pair_blocks(int N) { return (N * (N - 1) / 2 + 1) / 2; }
inline long refresh_threads(const Lat& L) { return (long)L.V * L.D * (refresh_pair_blocks(L.N) + 1); }

template <typename S2>
__device__ __forceinline__ void refresh_block(const Lat& L, S2* __restrict__ P, uint64_t seed, uint32_t traj,
                                              double scale, long t) {
  const int N = L.N, nb = refresh_pair_blocks(N);
  const long nl = (long)L.V * L.D;
  if (t >= nl * (nb + 1)) return;
  const bool diag = t >= nl * nb;
  const long l = diag ? t - nl * nb : t / nb;
  const int d = (int)(l / L.V);
  const int s = (int)(l - (long)d * L.V);
  const unsigned long long lk = (unsigned long long)s * L.D + d;
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  S2* p = P + (size_t)l * (N * N);
  auto block = [&](int blk, double (&g)[4]) {
    u32x4 c;
    c.x = (uint32_t)blk;
    c.y = (uint32_t)lk;
    c.z = (uint32_t)(lk >> 32);
    c.w = traj;
    normals4(philox4x32_10(c, k0, k1), g);
  };
  double g[4];
  if (!diag) {
    const int b = (int)(t - l * nb);
    block(b, g);
    // row i of pair q (row-major upper triangle): the first row whose end lies beyond q
    const int q = 2 * b;
    const float m = N - 0.5f;
    int i = (int)(m - sqrtf(fmaxf(m * m - 2.0f * q, 0.0f)));
    while (i > 0 && i * (2 * N - i - 1) / 2 > q) i--;
    while ((i + 1) * (2 * N - i - 2) / 2 <= q) i++;
    int j = i + 1 + q - i * (2 * N - i - 1) / 2;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      if (i >= N - 1) break;  // an odd pair count: the block's second half is the diagonal's
      const double xs = g[2 * h], xa = g[2 * h + 1];
      stc(p + i * N + j, mkc<double>(0.5 * scale * xs, -0.5 * scale * xa));
      stc(p + j * N + i, mkc<double>(0.5 * scale * xs, 0.5 * scale * xa));
      if (++j == N) {
        i++;
        j = i + 1;
      }
    }
    return;
  }
  const int a0 = N * (N - 1);
  int cur = -1;
  double suffix = 0.0;
  for (int dd = N - 1; dd >= 0; dd--) {
    double val = suffix;
    if (dd >= 1) {
      const int m = dd - 1;
      const double nm = sqrt(0.5 / ((double)(m + 1) * (m + 2)));
      const int a = a0 + m;
      if ((a >> 2) != cur) {
        block(a >> 2, g);
        cur = a >> 2;
      }
      const int r = a & 3;
      const double xm = r == 0 ? g[0] : r == 1 ? g[1] : r == 2 ? g[2] : g[3];
      val -= dd * nm * xm;
      suffix += nm * xm;
    }
    stc(p + dd * N + dd, mkc<double>(scale * val, 0.0));
  }
}

template <typename S2>
__global__ void __launch_bounds__(128) k_refresh_blocks(Lat L, S2* __restrict__ P, uint64_t seed,
                                                        const unsigned long long* __restrict__ traj_dev,
                                                        unsigned long long traj_host, double scale) {
  const uint32_t traj = (uint32_t)(traj_dev ? *traj_dev : traj_host);
  refresh_block<S2>(L, P, seed, traj, scale, (long)blockIdx.x * blockDim.x + threadIdx.x);
}

template <typename S2>
__global__ void k_refresh(Lat L, S2* __restrict__ P, uint64_t seed, const unsigned long long* __restrict__ traj_dev,
                          unsigned long long traj_host, double scale) {
  const uint32_t traj = (uint32_t)(traj_dev ? *traj_dev : traj_host);
  refresh_link<S2>(L, P, seed, traj, scale, (long)blockIdx.x * blockDim.x + threadIdx.x);
}

// Cold start (sun.cpp:194-207): every link the identity.
// (Padding sites get the identity too.)
template <typename S2>
__global__ void k_identity(Lat L, S2* __restrict__ U) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)field_elems(L)) return;
  int d, s, e;
  field_index(L, t, &d, &s, &e);
  stc(U + t, mkc<double>(e % (L.N + 1) == 0 ? 1.0 : 0.0, 0.0));
}

// Complex Gaussian matrices (unit variance per component pair) for the Haar
// hot start; counter (0x48000000 | j, l_lo, l_hi, 0) keeps them apart from
// the momentum stream.  A reunitarisation pass (MGS rows + det phase) turns
// them into Haar-distributed SU(N) links.
template <typename S2>
__global__ void k_gauss_matrices(Lat L, S2* __restrict__ U, uint64_t seed) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)L.V * L.D) return;
  const int N = L.N;
  const int d = (int)(t / L.V);
  const int s = (int)(t - (long)d * L.V);
  const unsigned long long lk = (unsigned long long)s * L.D + d;
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  for (int e0 = 0; e0 < N * N; e0 += 2) {
    u32x4 c;
    c.x = 0x48000000u | (uint32_t)(e0 >> 1);
    c.y = (uint32_t)lk;
    c.z = (uint32_t)(lk >> 32);
    c.w = 0u;
    double g[4];
    normals4(philox4x32_10(c, k0, k1), g);
    stc(U + eoff(L, d, e0, s), mkc<double>(g[0], g[1]));
    if (e0 + 1 < N * N) stc(U + eoff(L, d, e0 + 1, s), mkc<double>(g[2], g[3]));
  }
}

// Device-side trajectory bookkeeping.  The Metropolis test of sun.cpp:1249-1318
// in FP64: H = beta * (EnergyMag + simpleenergyEl / (2 NC)); accept when
// H_new < H_old (case 1) or u < exp(H_old - H_new) (case 2), u a Philox uniform
// with counter (0xFFFFFFFF, 0, 0, traj).
struct TrajState {
  double h_old;
  double h_new;
  double dh;
  double u;
  int accepted;  // 0 reject, 1 case 1, 2 case 2
  int pad;
  unsigned long long traj;  // trajectory counter (momentum refresh / Metropolis stream)
  unsigned long long n_acc, n_acc1, n_rej, n_tot;
};

// sums: [0] = action (temporal), [1] = action (spatial), [2] = kinetic
static __global__ void k_energy(const double* __restrict__ sums, double beta, int N, double* __restrict__ h_out) {
  *h_out = beta * ((sums[0] + sums[1]) + sums[2] / (2.0 * N));
}

__device__ __forceinline__ void metropolis(TrajState* st, uint64_t seed, double* __restrict__ log_out, int log_cap) {
  const double hn = st->h_new, ho = st->h_old;
  u32x4 c;
  c.x = 0xFFFFFFFFu;
  c.y = 0u;
  c.z = 0u;
  c.w = (uint32_t)st->traj;
  const u32x4 w = philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
  const double u = u01(w.x);
  int acc = 0;
  if (hn < ho)
    acc = 1;
  else if (u < exp(-hn + ho))
    acc = 2;
  st->dh = hn - ho;
  st->u = u;
  st->accepted = acc;
  st->n_tot++;
  if (acc) st->n_acc++;
  if (acc == 1) st->n_acc1++;
  if (!acc) st->n_rej++;
  if (log_out && log_cap > 0) {
    const unsigned long long k = st->traj % (unsigned long long)log_cap;
    log_out[4 * k + 0] = ho;
    log_out[4 * k + 1] = hn;
    log_out[4 * k + 2] = hn - ho;
    log_out[4 * k + 3] = (double)acc;
  }
  st->traj++;
}

// Sums of n pairs by a CTA of ENERGY_THREADS, the same order for a chain alone
// and in a batch; four running sums a thread keep the loads of the long lists
// (a pair per CTA of the force launch) in flight.
constexpr int ENERGY_THREADS = 1024;
__device__ __forceinline__ void sum_pairs(const double2* __restrict__ p, int n, double (&v)[2]) {
  __shared__ double2 sh[ENERGY_THREADS / 32];
  double2 a[4] = {};
  int i = threadIdx.x;
  for (; i + 3 * ENERGY_THREADS < n; i += 4 * ENERGY_THREADS)
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const double2 z = p[i + u * ENERGY_THREADS];
      a[u].x += z.x;
      a[u].y += z.y;
    }
  for (; i < n; i += ENERGY_THREADS) {
    a[0].x += p[i].x;
    a[0].y += p[i].y;
  }
  double x = (a[0].x + a[1].x) + (a[2].x + a[3].x), y = (a[0].y + a[1].y) + (a[2].y + a[3].y);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    x += __shfl_down_sync(0xffffffffu, x, o);
    y += __shfl_down_sync(0xffffffffu, y, o);
  }
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = make_double2(x, y);
  __syncthreads();
  if (threadIdx.x < 32) {
    x = sh[threadIdx.x].x;
    y = sh[threadIdx.x].y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      x += __shfl_down_sync(0xffffffffu, x, o);
      y += __shfl_down_sync(0xffffffffu, y, o);
    }
  }
  v[0] = x;
  v[1] = y;
  __syncthreads();
}

// H from the pairs of a force launch: W = sum ReTr(U S) counts each of the
// D (D-1) / 2 plaquettes per site four times, K = sum tr2 P.
__device__ __forceinline__ double energy_of(const double (&v)[2], double beta, const Lat& L) {
  const double np = 0.5 * L.D * (L.D - 1) * (double)L.V;
  return beta * ((np - v[0] / (4.0 * L.N)) + v[1] / (2.0 * L.N));
}

__device__ __forceinline__ void energies_and_test(const double* __restrict__ pairs, int ctas, const Lat& L, double beta,
                                                  TrajState* st, uint64_t seed, double* __restrict__ log_out,
                                                  int log_cap) {
  double a[2], b[2];
  sum_pairs(reinterpret_cast<const double2*>(pairs), ctas, a);
  sum_pairs(reinterpret_cast<const double2*>(pairs) + ctas, ctas, b);
  if (threadIdx.x == 0) {
    st->h_old = energy_of(a, beta, L);
    st->h_new = energy_of(b, beta, L);
    metropolis(st, seed, log_out, log_cap);
  }
}

static __global__ void __launch_bounds__(ENERGY_THREADS)
    k_energies_metropolis(const double* __restrict__ pairs, int ctas, Lat L, double beta, TrajState* st, uint64_t seed,
                          double* __restrict__ log_out, int log_cap) {
  energies_and_test(pairs, ctas, L, beta, st, seed, log_out, log_cap);
}

static __global__ void k_metropolis(TrajState* st, uint64_t seed, double* __restrict__ log_out, int log_cap) {
  metropolis(st, seed, log_out, log_cap);
}

// takeconfiguration / loadconfiguration (sun.cpp:725-742) after the test:
// accepted -> Uconf = U, rejected -> U = Uconf.  Vectorised 16-byte copy.
static __global__ void k_accept_copy(const TrajState* __restrict__ st, uint4* __restrict__ U, uint4* __restrict__ Uconf,
                              long n16) {
  const bool acc = st->accepted != 0;
  uint4* dst = acc ? Uconf : U;
  const uint4* src = acc ? U : Uconf;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += (long)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

// Conversion between the host U-conf layout (FP64, [site][dir][row][col][re,im])
// and the device layout in either precision.
template <typename S2>
__global__ void k_from_conf(Lat L, const double2* __restrict__ conf, S2* __restrict__ f) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)field_elems(L)) return;
  // t indexes the device field
  int d, s, e;
  if (!field_index(L, t, &d, &s, &e)) {
    stc(f + t, mkc<double>(0.0, 0.0));
    return;
  }
  const double2 v = conf[((size_t)s * L.D + d) * (L.N * L.N) + e];
  stc(f + t, mkc<double>(v.x, v.y));
}

template <typename S2>
__global__ void k_to_conf(Lat L, const S2* __restrict__ f, double2* __restrict__ conf) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int NN = L.N * L.N;
  const long tot = (long)L.V * L.D * NN;
  if (t >= tot) return;
  // t indexes the conf output: t = (s*D + d)*NN + e
  const long lk = t / NN;
  const int e = (int)(t - lk * NN);
  const int s = (int)(lk / L.D);
  const int d = (int)(lk - (long)s * L.D);
  const cpx<double> v = ldc<double>(f + eoff(L, d, e, s));
  conf[t] = make_double2(v.re, v.im);
}

// Non-finite scan of a host-uploaded U-conf buffer: counts NaN/Inf doubles.
static __global__ void k_count_nonfinite(const double* __restrict__ x, long n, unsigned long long* __restrict__ count) {
  unsigned long long c = 0;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    if (!isfinite(x[i])) c++;
  if (c) atomicAdd(count, c);
}

// ---- the plaquettes of a site by a whole CTA, any NC (FourierTrafo: a few sites) ----
// Plaquette sums of one site (same sums as plaq_site): B = U_nu(x+mu) and
// C = U_mu(x+nu) staged in shared memory as FP64 ([N][N+1]), thread t owns row
// t / 4 and the columns j = 4q + t % 4 of AB and DC (A = U_mu(x), D = U_nu(x)
// read from global), tr = sum Re (AB)_ij conj((DC)_ij); partial[s*2 + {0,1}].
template <typename S2>
__global__ void __launch_bounds__(RED_THREADS) k_plaq_big(Lat L, const S2* __restrict__ U, double* __restrict__ partial) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = L.N, NP = N + 1;
  cpx<double>* Bs = reinterpret_cast<cpx<double>*>(smem_raw);
  cpx<double>* Cs = Bs + N * NP;
  const int s = blockIdx.x;
  const int tid = threadIdx.x;
  const int rows_per_pass = RED_THREADS / 4;
  double trt = 0.0, trs = 0.0;
  int nt = 0, ns = 0;
  for (int mu = 0; mu < L.D; mu++) {
    const int xpmu = nb_plus(L, mu, s);
    for (int nu = mu + 1; nu < L.D; nu++) {
      const int xpnu = nb_plus(L, nu, s);
      __syncthreads();
      for (int e = tid; e < N * N; e += RED_THREADS) {
        const int r = e / N, c = e - (e / N) * N;
        Bs[r * NP + c] = ldc<double>(U + eoff(L, nu, e, xpmu));
        Cs[r * NP + c] = ldc<double>(U + eoff(L, mu, e, xpnu));
      }
      __syncthreads();
      double tr = 0.0;
      for (int i0 = 0; i0 < N; i0 += rows_per_pass) {
        const int i = i0 + tid / 4;
        if (i >= N) continue;
        cpx<double> ab[16], dc[16];
#pragma unroll
        for (int q = 0; q < 16; q++) ab[q] = dc[q] = czero<double>();
        for (int k = 0; k < N; k++) {
          const cpx<double> a = ldc<double>(U + eoff(L, mu, i * N + k, s));
          const cpx<double> d = ldc<double>(U + eoff(L, nu, i * N + k, s));
#pragma unroll
          for (int q = 0; q < 16; q++) {
            const int j = 4 * q + (tid & 3);
            if (j < N) {
              cmac(ab[q], a, Bs[k * NP + j]);
              cmac(dc[q], d, Cs[k * NP + j]);
            }
          }
        }
#pragma unroll
        for (int q = 0; q < 16; q++) {
          tr = fma(ab[q].re, dc[q].re, tr);
          tr = fma(ab[q].im, dc[q].im, tr);
        }
      }
      if (mu == 0) {
        trt += tr;
        nt++;
      } else {
        trs += tr;
        ns++;
      }
    }
  }
  double v[2] = {trt, trs};
  block_sum<2>(v);
  if (tid == 0) {
    const bool in = counted(L, s);
    partial[(size_t)s * 2 + 0] = in ? nt - v[0] / N : 0.0;
    partial[(size_t)s * 2 + 1] = in ? ns - v[1] / N : 0.0;
  }
}

}  // namespace misc
}  // namespace askja
