// Closed Wilson / Polyakov lines and the Gauss law for NC <= 4 (blocked
// fields), and the finishing sums of the Gauss law for every NC.  NC >= 5:
// mma64.cuh.
#pragma once

#include "eig.cuh"
#include "misc.cuh"
#include "small.cuh"

namespace askja {

// Lines of several directions in one launch: line q with first[i] <= q <
// first[i+1] runs along dir[i] through all n[dir] links, from the site
// (q - first[i]) * start_stride[i] (whose coordinate along dir is 0).
struct LineSet {
  int sets;
  int dir[ASKJA_MAX_DIM];
  int start_stride[ASKJA_MAX_DIM];
  int first[ASKJA_MAX_DIM + 1];

  void add(int d, int lines, int stride) {
    if (sets == 0) first[0] = 0;
    dir[sets] = d;
    start_stride[sets] = stride;
    first[sets + 1] = first[sets] + lines;
    sets++;
  }
  int lines() const { return sets ? first[sets] : 0; }
};

__device__ __forceinline__ int line_of(const LineSet& ls, int q, int* start) {
  int i = 0;
  while (i + 1 < ls.sets && q >= ls.first[i + 1]) i++;
  *start = (q - ls.first[i]) * ls.start_stride[i];
  return ls.dir[i];
}

namespace lines {

// Product of the links of one line, by one warp (result in lane 0): each lane
// multiplies its share of the links in registers, then neighbouring lanes'
// products are joined pairwise.  A warp walking the line link by link, a
// row per thread, waited for a load and two barriers per link (SU(3) 16^4:
// 54 us for 16 lines of 16 links).
template <int N, typename S2>
__device__ __forceinline__ void warp_product(small::Mat<N, double>& W, const Lat& L, const S2* __restrict__ U, int dir,
                                             int start) {
  const int lane = threadIdx.x & 31, n = L.n[dir];
  const int per = (n + 31) / 32;
  const int k0 = min(n, lane * per), k1 = min(n, k0 + per);
#pragma unroll
  for (int i = 0; i < N; i++)
#pragma unroll
    for (int j = 0; j < N; j++) W.a[i][j] = mkc<double>(i == j ? 1.0 : 0.0, 0.0);
  for (int k = k0; k < k1; k++) {
    small::Mat<N, double> M, T;
    small::load(M, U, L, dir, start + k * L.stride[dir]);
    if (k == k0) {
      W = M;
    } else {
      small::mul_nn(T, W, M);
      W = T;
    }
  }
  const int used = (n + per - 1) / per;  // lanes with links
  for (int o = 1; o < used; o <<= 1) {
    small::Mat<N, double> R, T;
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
      for (int j = 0; j < N; j++) {
        R.a[i][j].re = __shfl_down_sync(0xffffffffu, W.a[i][j].re, o);
        R.a[i][j].im = __shfl_down_sync(0xffffffffu, W.a[i][j].im, o);
      }
    small::mul_nn(T, W, R);
    if ((lane & (2 * o - 1)) == 0 && lane + o < used) W = T;
  }
}

// out[q] = |Tr W_q| / NC, a warp per line
template <int N, typename S2>
__global__ void __launch_bounds__(128) k_lines(Lat L, const S2* __restrict__ U, const __grid_constant__ LineSet ls,
                                               int nlines, double* __restrict__ out) {
  const int q = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (q >= nlines) return;
  int start;
  const int dir = line_of(ls, q, &start);
  small::Mat<N, double> W;
  warp_product<N>(W, L, U, dir, start);
  if ((threadIdx.x & 31) == 0) {
    double tr = 0.0, ti = 0.0;
#pragma unroll
    for (int k = 0; k < N; k++) {
      tr += W.a[k][k].re;
      ti += W.a[k][k].im;
    }
    out[q] = hypot(tr, ti) / N;
  }
}

// eigenvalues of the line matrices: ev[q*N + i]
template <int N, typename S2>
__global__ void __launch_bounds__(32) k_line_eigs(Lat L, const S2* __restrict__ U, const __grid_constant__ LineSet ls,
                                                  double2* __restrict__ ev, int* __restrict__ fail) {
  __shared__ cpx<double> H[N * N], v[N], e[N];
  int start;
  const int dir = line_of(ls, blockIdx.x, &start);
  small::Mat<N, double> W;
  warp_product<N>(W, L, U, dir, start);
  if (threadIdx.x == 0)
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
      for (int j = 0; j < N; j++) H[i * N + j] = W.a[i][j];
  __syncwarp();
  eig::hessenberg_qr(H, N, v, e, fail);
  __syncwarp();
  if (threadIdx.x < N) ev[(size_t)blockIdx.x * N + threadIdx.x] = make_double2(e[threadIdx.x].re, e[threadIdx.x].im);
}

// Gauss law (sun.cpp:415-438): the lattice sum of Pi_j(x) - U_j^dag(x-j) Pi_j(x-j) U_j(x-j)
// over all sites and directions.  Re-indexing x -> x+j turns every term into a
// function of one link l: Pi_l - U_l^dag Pi_l U_l.  Thread per link with both
// matrices in registers and a grid stride; each CTA's summed matrix goes to
// partial[b*2*N*N + 2e + {0,1}].  (An element per thread, which formed
// Pi U anew for every element and walked its 256 links one by one, took 300 us
// on SU(3) 16^4.)
template <int N, typename S2>
__global__ void __launch_bounds__(128) k_gauss(Lat L, const S2* __restrict__ U, const S2* __restrict__ Pi,
                                               double* __restrict__ partial) {
  __shared__ double sh[4][2 * N * N];
  small::Mat<N, double> G;
  small::zero(G);
  const long nl = (long)L.V * L.D;
  for (long l = (long)blockIdx.x * blockDim.x + threadIdx.x; l < nl; l += (long)gridDim.x * blockDim.x) {
    const int d = (int)(l / L.V);
    const int s = (int)(l - (long)d * L.V);
    small::Mat<N, double> u, p;
    small::load(u, U, L, d, s);
    small::load(p, Pi, L, d, s);
#pragma unroll
    for (int j = 0; j < N; j++) {
      cpx<double> c[N];  // column j of Pi U
#pragma unroll
      for (int a = 0; a < N; a++) {
        c[a] = czero<double>();
#pragma unroll
        for (int b = 0; b < N; b++) cmac(c[a], p.a[a][b], u.a[b][j]);
      }
#pragma unroll
      for (int i = 0; i < N; i++) {
        cpx<double> t = czero<double>();
#pragma unroll
        for (int a = 0; a < N; a++) cmac_cn(t, u.a[a][i], c[a]);
        G.a[i][j].re += p.a[i][j].re - t.re;
        G.a[i][j].im += p.a[i][j].im - t.im;
      }
    }
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < N; i++)
#pragma unroll
    for (int j = 0; j < N; j++) {
      double re = G.a[i][j].re, im = G.a[i][j].im;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        re += __shfl_down_sync(0xffffffffu, re, o);
        im += __shfl_down_sync(0xffffffffu, im, o);
      }
      if (lane == 0) {
        sh[wid][2 * (i * N + j)] = re;
        sh[wid][2 * (i * N + j) + 1] = im;
      }
    }
  __syncthreads();
  for (int e = threadIdx.x; e < 2 * N * N; e += blockDim.x)
    partial[(size_t)blockIdx.x * (2 * N * N) + e] = (sh[0][e] + sh[1][e]) + (sh[2][e] + sh[3][e]);
}

// Sum of the partials of every matrix component (a warp each), over ngroups
// partial matrices of 2 NC^2 doubles.
static __global__ void __launch_bounds__(256) k_gauss_sum(const double* __restrict__ partial, int ngroups, int n2,
                                                          double* __restrict__ sum) {
  const int e = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (e >= n2) return;
  double x = 0.0;
  for (int g = lane; g < ngroups; g += 32) x += partial[(size_t)g * n2 + e];
  x = eig::warp_sum(x);
  if (lane == 0) sum[e] = x;
}

// tr2 of the summed matrix
static __global__ void __launch_bounds__(misc::RED_THREADS) k_gauss_finish(const double* __restrict__ sum, int N,
                                                                           double* __restrict__ out) {
  double v[1] = {0.0};
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
    const int i = e / N, j = e - (e / N) * N, t = j * N + i;
    v[0] += sum[2 * e] * sum[2 * t] - sum[2 * e + 1] * sum[2 * t + 1];
  }
  misc::block_sum<1>(v);
  if (threadIdx.x == 0) *out = v[0];
}

}  // namespace lines
}  // namespace askja
