// Link update, plaquette and kinetic sums for 5 <= NC <= 64 on the FP64 tensor
// instruction (mma.sync m8n8k4 f64; tcgen05 has no FP64 kind), for FP64 and
// FP32 storage; the kicks and fused updates of FP32 storage, NC >= 7 or 11, in TF32
// split in two (see prod).
//
// A matrix is cut into 8 x 8 tiles (NT = ceil(NC / 8) of them a side); one warp
// owns the eight rows 8w .. 8w+7 of every left operand and result, NT warps
// own a link.  A complex product is four real MMAs per 8 x 8 x 4 block.
//
// Register layout of a tile (the accumulator layout of the instruction): lane
// holds row lane / 4, columns 2 (lane % 4) + {0, 1}.  The sum over k may run in
// any order as long as both operands use the same one, so the k-steps take the
// columns {0, 2, 4, 6} and {1, 3, 5, 7} of a tile: an accumulator tile is then
// the left operand of the next product as it stands, with no exchange between
// lanes.  A right operand Y^dag is a row-pattern load of Y (lane: row lane / 4,
// columns 2 (lane % 4) + e), a right operand Y a column-pattern load (rows
// 2 (lane % 4) + e, column lane / 4); both read whole sectors of the row-major
// matrix of one link (link-major fields, common.cuh), straight from L1 / L2.
// The staple sum
//   S = sum_nu [U_nu(x+mu) U_mu(x+nu)^dag] U_nu(x)^dag
//             + [U_nu(x+mu-nu)^dag U_mu(x-nu)^dag] U_nu(x-nu)
// has a load or the accumulator before it as every left operand, and two of its
// six links per plane as column-pattern loads.  A column load touches four
// lines per quarter-warp, 32 L1 wavefronts a matrix against 8 for a row load:
// accumulating S^dag instead spares S its way through shared memory but makes
// four of the six links column loads (SU(8) 10^4: 573 wavefronts a link, L1
// 80 % busy, 117 us an update).  Four matrices per link cross the warps' rows,
// through one shared-memory tile of row stride 8 NT + 1 (conflict-free for rows
// and columns): S, W = U S (the kick needs its transpose), X = i eps P and X^3
// (right operands of the series).
//
// What bounds it: the FP64 pipe.  One 8 x 8 x 4 MMA takes 4 cycles of an SM
// (36.8 TFLOP/s measured with independent accumulators); a link update of
// LEVEL 8 in four dimensions is 18 products of NT^3 * 8 MMAs.  Operand loads
// are 8 shared-bandwidth cycles per 32 cycles of MMA.
#pragma once

#include "launch.h"
#include "lines.cuh"
#include "misc.cuh"
#include "mma64.h"

namespace askja {
namespace m64 {

// One lattice's fields, as the kernels read them: by value for a single chain,
// from a table (with a per-CTA list of table index and block) for a batch.
struct Job {
  const int* nbr;
  int V, D, N;
  int order;    // Taylor order of the drift
  int project;  // FP32 storage: project the links read onto U(N) to first order (see drift)
  int r0, r1;   // sites counted by the reductions (Lat)
  void* U[2];   // links in U[cur], updated links to U[cur ^ 1]
  const void* Pin;
  const void* Pin2;  // second momenta of k_kinetic, or null
  void* Pout;
  double kick;  // kick step (times the launch's kick scale)
  double dt;    // drift step
  double* pairs;  // energy sums of the CTAs (SUMS_OLD, then SUMS_NEW)
  int ctas;       // CTAs of this job's link launch
  double* plaq_partial;
  double* kin_partial;
  double* out;       // totals of a reduction launched for one lattice (misc::publish)
  unsigned* ticket;
};

// CTA shapes.  Link update: four warps a CTA (one link from NT = 3 on) at the
// tightest register budget that does not spill much.  Small CTAs fill the last
// wave better and cost nothing, the warps of different links being independent:
// us per fused step against eight-warp CTAs of 2-3 a SM, SU(8) 10^4 112 -> 105,
// SU(16) 6^4 102 -> 99, SU(24) 6^3 51 -> 43, SU(32) 6^4 751 -> 722 (94 % of the
// MMA rate).  Plaquette: about eight warps, a site each NT.
// R: the arithmetic (double: FP64 MMA; float: split TF32 MMA, see prod).
template <int NT, typename R = double>
struct Cta {
  static constexpr int LINKS = NT == 1 ? 4 : NT == 2 ? 2 : 1;
  static constexpr int SITES = NT == 1 ? 8 : NT == 2 ? 4 : NT <= 4 ? 2 : 1;
  static constexpr int THREADS = 32 * NT * LINKS;
  static constexpr int PLAQ_THREADS = 32 * NT * SITES;
  using V2 = typename Storage<R>::type;
  static constexpr int LD = 8 * NT + (sizeof(R) == 8 ? 1 : 2);  // conflict-free column reads
  static constexpr int TILE = 8 * NT * LD;  // complex numbers of one link's tile
  // small matrices keep the rows of X and X^2 in registers; larger ones read X
  // back from the momenta and keep X^2 in a second tile
  static constexpr bool KEEP = NT <= (sizeof(R) == 8 ? 2 : 4);
  static constexpr int TILES = KEEP ? 1 : 2;
  static constexpr size_t SMEM = (size_t)LINKS * TILES * TILE * sizeof(V2);
  // resident CTAs the register budget is set for, us a step beside the next choice:
  // float (with FINE 0) at 6 / 8 and 4 / 5 / 3 CTAs (NT = 1, 2) SU(8) 10^4 90 / 93, SU(16) 6^4 74 /
  // 80 / 76; 5 / 4 / 6 (NT = 3) SU(24) 6^3 29 / 36 / 31; 3 / 4 / 2 (NT = 4) SU(32) 8^4
  // 1686 / 1749 / 1880.  NT = 5, 6: one CTA of NT warps a SM (200 to 255 registers)
  // leaves it idle at every barrier; two (168, spills of 4 to 116 bytes): SU(40) 6^3
  // FP64 262 -> 207, FP32 206 -> 161, SU(48) 6^3 371 -> 298 and 292 -> 242, SU(45) 5x6x6
  // 319 -> 262 and 291 -> 221.  A third spills more (SU(40) 6^3 189, 143, but 4x4 38 ->
  // 42), as a second does at NT = 7 (SU(50) 5^3 FP64 317 -> 339); FP64 NT = 8 has no
  // shared memory for it.  A lattice of at most a link per SM keeps the whole register
  // file to one CTA (k_link with TIGHT false; SU(48) 4x4 FP32 45 / 54, 10x10 89 / 73).
  static constexpr int MIN_CTAS = NT > 4 ? (NT <= 6 ? 2 : 1)
                                  : sizeof(R) == 8 ? (NT == 1 ? 8 : NT == 2 ? 4 : NT == 3 ? 5 : 4)
                                                   : (NT == 1 ? 6 : NT == 2 ? 4 : NT == 3 ? 5 : 3);
};

template <typename R>
struct AccT {
  R re[2], im[2];  // columns 2j, 2j + 1
};
template <typename R>
struct OpT {
  R re, im;
};
using Acc = AccT<double>;
using Op = OpT<double>;

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

template <int NT, typename R>
__device__ __forceinline__ void zero(AccT<R> (&c)[NT]) {
#pragma unroll
  for (int t = 0; t < NT; t++) c[t].re[0] = c[t].re[1] = c[t].im[0] = c[t].im[1] = R(0);
}

// Loads of fields that the launch does not write, coherent and volatile: k_link
// is resident while the launch before still writes them, so they must not be
// ld.global.nc nor move above its grid_wait (common.cuh).  Left free to move with
// their operands (asm without volatile), the loads of NT = 1 spilt 208 bytes
// instead of 44 in FP64.
// Two consecutive complex numbers of a row (c even):
__device__ __forceinline__ void ld_pair(const double2* p, Op& a, Op& b) {
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a.re), "=d"(a.im), "=d"(b.re), "=d"(b.im) : "l"(p));
}
template <typename R>
__device__ __forceinline__ void ld_pair(const float2* p, OpT<R>& a, OpT<R>& b) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  a.re = v.x;
  a.im = v.y;
  b.re = v.z;
  b.im = v.w;
}
// one
__device__ __forceinline__ double2 ld_value(const double2* p) {
  double2 v;
  asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ float2 ld_value(const float2* p) {
  float2 v;
  asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
// the same from memory that this launch may write, and to memory
__device__ __forceinline__ void ld_pair_rw(const double2* p, Op& a, Op& b) {
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(a.re), "=d"(a.im), "=d"(b.re), "=d"(b.im)
               : "l"(p)
               : "memory");
}
template <typename R>
__device__ __forceinline__ void ld_pair_rw(const float2* p, OpT<R>& a, OpT<R>& b) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  a.re = v.x;
  a.im = v.y;
  b.re = v.z;
  b.im = v.w;
}
__device__ __forceinline__ void st_pair(double2* p, const Op& a, const Op& b) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a.re), "d"(a.im), "d"(b.re), "d"(b.im)
               : "memory");
}
template <typename R>
__device__ __forceinline__ void st_pair(float2* p, const OpT<R>& a, const OpT<R>& b) {
  *reinterpret_cast<float4*>(p) = make_float4((float)a.re, (float)a.im, (float)b.re, (float)b.im);
}
__device__ __forceinline__ double round_to(const double2*, double v) { return v; }
__device__ __forceinline__ double round_to(const float2*, double v) { return (double)(float)v; }
__device__ __forceinline__ float round_to(const float2*, float v) { return v; }
__device__ __forceinline__ double2 pack(const double2*, double re, double im) { return make_double2(re, im); }
__device__ __forceinline__ float2 pack(const float2*, double re, double im) {
  return make_float2((float)re, (float)im);
}
template <typename R = double, typename S2>
__device__ __forceinline__ OpT<R> ld_one(const S2* p) {
  const S2 v = ld_value(p);
  OpT<R> o;
  o.re = (R)v.x;
  o.im = (R)v.y;
  return o;
}
template <typename R = double>
__device__ __forceinline__ OpT<R> op0() {
  OpT<R> o;
  o.re = o.im = R(0);
  return o;
}

// Who this thread is within its link, and the two load patterns.  FULL: NC = 8 NT.
template <int NT, bool FULL>
struct Who {
  int w, q, j, n;  // row block, lane / 4, lane % 4, NC (when not FULL)
  __device__ __forceinline__ int N() const { return FULL ? 8 * NT : n; }
  // row 8 rb + q, columns 8 cb + 2 j + {0, 1}
  template <typename R, typename S2>
  __device__ __forceinline__ void rows(const S2* m, int rb, int cb, OpT<R> (&o)[2]) const {
    const int r = 8 * rb + q, c = 8 * cb + 2 * j;
    if constexpr (FULL) {
      ld_pair(m + r * N() + c, o[0], o[1]);
    } else {
      o[0] = r < n && c < n ? ld_one<R>(m + r * n + c) : op0<R>();
      o[1] = r < n && c + 1 < n ? ld_one<R>(m + r * n + c + 1) : op0<R>();
    }
  }
  // own rows, columns 8 t + 2 j + {0, 1}, of a matrix this launch also writes
  template <typename R, typename S2>
  __device__ __forceinline__ void own(const S2* m, int t, OpT<R> (&o)[2]) const {
    const int r = 8 * w + q, c = 8 * t + 2 * j;
    if constexpr (FULL) {
      ld_pair_rw(m + r * N() + c, o[0], o[1]);
    } else {
#pragma unroll
      for (int e = 0; e < 2; e++) {
        o[e] = op0<R>();
        if (r < n && c + e < n) {
          const S2 v = m[r * n + c + e];
          o[e].re = (R)v.x;
          o[e].im = (R)v.y;
        }
      }
    }
  }
  // the same elements to a matrix
  template <typename R, typename S2>
  __device__ __forceinline__ void put(S2* m, int t, const OpT<R> (&o)[2]) const {
    const int r = 8 * w + q, c = 8 * t + 2 * j;
    if constexpr (FULL) {
      st_pair(m + r * N() + c, o[0], o[1]);
    } else {
#pragma unroll
      for (int e = 0; e < 2; e++)
        if (r < n && c + e < n) m[r * n + c + e] = pack(m, o[e].re, o[e].im);
    }
  }
  // rows 8 rb + 2 j + {0, 1}, column 8 cb + q
  template <typename R, typename S2>
  __device__ __forceinline__ void cols(const S2* m, int rb, int cb, OpT<R> (&o)[2]) const {
    const int r = 8 * rb + 2 * j, c = 8 * cb + q;
    if constexpr (FULL) {
      o[0] = ld_one<R>(m + r * N() + c);
      o[1] = ld_one<R>(m + (r + 1) * N() + c);
    } else {
      o[0] = r < n && c < n ? ld_one<R>(m + r * n + c) : op0<R>();
      o[1] = r + 1 < n && c < n ? ld_one<R>(m + (r + 1) * n + c) : op0<R>();
    }
  }
};

// c += A B (CONJ false) or A conj(B) (CONJ true: the right operand is given as
// the elements of Y for the product with Y^dag).  fa(kb, a): the left operand's
// own-row elements of tile column kb, fb(kb, t, b): the right operand's.
//
// FP32 arithmetic (R = float): m16n8k8 TF32 MMAs on the 16 x 8 stack [Re A; Im A],
//   [Re; Im] C += [Re A; Im A] Re B + [-Im A; Re A] Im B,
// whose accumulator rows q and q + 8 are the real and imaginary parts of the
// same elements as the FP64 layout's (k slots j and j + 4 take the columns 2j and
// 2j + 1).  Every operand is split x = hi + lo, hi rounded to TF32's 11 bits; hi hi
// starts each 8-column step from a zero accumulator and is added to c in FP32
// with round to nearest (the tensor cores' own accumulation rounds toward zero:
// chained, it would scale the staple sum by 1 - 1e-6), lo hi + hi lo, 2^-11
// smaller, is chained.  Six MMAs of 2.1 SM cycles per 8 x 8 x 8 complex block
// against 32 cycles for the eight FP64 ones (measured 276 TFLOP/s TF32, 36.8
// FP64); what bounds it is the wait for operands and their splitting.
// FINE (products of the force, fine_force in mma64.h): what is left of the error
// is the truncation of hi hi.  1: the MMAs of Re B and Im B each start from zero
// and are added in FP32, one truncation less on the sum.  2: and the mean of what
// truncation takes, 2^-23 / 3 of a result (half a unit in the last place of a
// mantissa spread over its binade evenly in the logarithm), goes into the cross
// terms.  us per fused step, FP64 MMA on FP32 storage -> split TF32: SU(8) 10^4
// 106 -> 98 (FINE 0: 91), SU(12) 6^4 114 -> 92 (85), SU(16) 6^4 102 -> 78 (75),
// SU(17) 6^3 46 -> 36 (35), SU(24) 6^3 43 -> 31, SU(48) 6^3 431 -> 244; SU(5)
// 17x15x13 stays on the FP64 MMA, 28.3 against 24.9 with FINE 0 (row kernels 28.7).
// Two row blocks a warp, sharing a right operand's split, gained nothing (SU(16)
// 73, SU(32) 8^4 1782 against 1684); the next plane's links prefetched to L1
// cost 3 to 10 %.
template <int NT, bool CONJ, int KU, int FINE = 0, typename FA, typename FB>
__device__ __forceinline__ void prod(Acc (&c)[NT], FA&& fa, FB&& fb) {
#pragma unroll KU
  for (int kb = 0; kb < NT; kb++) {
    Op a[2];
    fa(kb, a);
    const double n0 = CONJ ? -a[0].re : -a[0].im, n1 = CONJ ? -a[1].re : -a[1].im;
#pragma unroll
    for (int t = 0; t < NT; t++) {
      Op b[2];
      fb(kb, t, b);
      dmma(c[t].re, a[0].re, b[0].re);
      dmma(c[t].im, CONJ ? a[0].im : a[0].re, CONJ ? b[0].re : b[0].im);
      dmma(c[t].re, CONJ ? a[0].im : n0, b[0].im);
      dmma(c[t].im, CONJ ? n0 : a[0].im, CONJ ? b[0].im : b[0].re);
      dmma(c[t].re, a[1].re, b[1].re);
      dmma(c[t].im, CONJ ? a[1].im : a[1].re, CONJ ? b[1].re : b[1].im);
      dmma(c[t].re, CONJ ? a[1].im : n1, b[1].im);
      dmma(c[t].im, CONJ ? n1 : a[1].im, CONJ ? b[1].im : b[1].re);
    }
  }
}

__device__ __forceinline__ void tmma(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// x = hi + lo, hi with TF32's mantissa (rounded to nearest in magnitude)
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
  hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  lo = __float_as_uint(x - __uint_as_float(hi));
}

template <int NT, bool CONJ, int KU, int FINE = 0, typename FA, typename FB>
__device__ __forceinline__ void prod(AccT<float> (&c)[NT], FA&& fa, FB&& fb) {
  float cor[NT][4];
#pragma unroll
  for (int t = 0; t < NT; t++) cor[t][0] = cor[t][1] = cor[t][2] = cor[t][3] = 0.f;
#pragma unroll KU
  for (int kb = 0; kb < NT; kb++) {
    OpT<float> a[2];
    fa(kb, a);
    constexpr uint32_t SIGN = 0x80000000u;
    uint32_t h1[4], l1[4], h2[4], l2[4];  // [Re; Im] and [-Im; Re] (CONJ: [Im; -Re])
#pragma unroll
    for (int e = 0; e < 2; e++) {
      split_tf32(a[e].re, h1[2 * e], l1[2 * e]);
      split_tf32(a[e].im, h1[2 * e + 1], l1[2 * e + 1]);
      h2[2 * e] = CONJ ? h1[2 * e + 1] : h1[2 * e + 1] ^ SIGN;
      l2[2 * e] = CONJ ? l1[2 * e + 1] : l1[2 * e + 1] ^ SIGN;
      h2[2 * e + 1] = CONJ ? h1[2 * e] ^ SIGN : h1[2 * e];
      l2[2 * e + 1] = CONJ ? l1[2 * e] ^ SIGN : l1[2 * e];
    }
#pragma unroll
    for (int t = 0; t < NT; t++) {
      OpT<float> b[2];
      fb(kb, t, b);
      uint32_t rh[2], rl[2], ih[2], il[2];
#pragma unroll
      for (int e = 0; e < 2; e++) {
        split_tf32(b[e].re, rh[e], rl[e]);
        split_tf32(b[e].im, ih[e], il[e]);
      }
      float m[4] = {0.f, 0.f, 0.f, 0.f};
      tmma(m, h1, rh);
      if constexpr (FINE > 0) {
        float m2[4] = {0.f, 0.f, 0.f, 0.f};
        tmma(m2, h2, ih);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          m[i] += m2[i];
          if constexpr (FINE > 1) cor[t][i] = fmaf(m[i], 0x1.555556p-25f, cor[t][i]);
        }
      } else {
        tmma(m, h2, ih);
      }
      tmma(cor[t], l1, rh);
      tmma(cor[t], l2, ih);
      tmma(cor[t], h1, rl);
      tmma(cor[t], h2, il);
      c[t].re[0] += m[0];
      c[t].re[1] += m[1];
      c[t].im[0] += m[2];
      c[t].im[1] += m[3];
    }
  }
#pragma unroll
  for (int t = 0; t < NT; t++) {
    c[t].re[0] += cor[t][0];
    c[t].re[1] += cor[t][1];
    c[t].im[0] += cor[t][2];
    c[t].im[1] += cor[t][3];
  }
}

// the rows of an accumulator as left operand
template <int NT, typename R>
__device__ __forceinline__ void from_acc(const AccT<R> (&c)[NT], int kb, OpT<R> (&a)[2]) {
  a[0].re = c[kb].re[0];
  a[0].im = c[kb].im[0];
  a[1].re = c[kb].re[1];
  a[1].im = c[kb].im[1];
}

// Barrier over the NT warps of link slot `slot` (a warp's own tile: NT = 1).
template <int NT>
__device__ __forceinline__ void link_sync(int slot) {
  if constexpr (NT == 1)
    __syncwarp();
  else
    asm volatile("bar.sync %0, %1;" ::"r"(slot + 1), "r"(32 * NT) : "memory");
}

// the same barrier, and whether any thread of the link says so
template <int NT>
__device__ __forceinline__ bool link_any(int slot, bool mine) {
  if constexpr (NT == 1) {
    return __any_sync(0xffffffffu, mine);
  } else {
    uint32_t any;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.or.pred q, %2, %3, p;\n selp.u32 %0, 1, 0, q;\n}"
        : "=r"(any)
        : "r"((uint32_t)mine), "r"(slot + 1), "r"(32 * NT)
        : "memory");
    return any != 0;
  }
}

// own rows of an accumulator to a field matrix
template <int NT, bool FULL, typename R, typename S2>
__device__ __forceinline__ void store_rows(S2* m, const Who<NT, FULL>& me, const AccT<R> (&c)[NT]) {
#pragma unroll
  for (int t = 0; t < NT; t++) {
    OpT<R> o[2];
    from_acc(c, t, o);
    me.put(m, t, o);
  }
}

// own rows of an accumulator to the link's shared tile
template <int NT, bool FULL, typename R, typename V2>
__device__ __forceinline__ void tile_rows(V2* S, const Who<NT, FULL>& me, const AccT<R> (&c)[NT]) {
  V2* p = S + (8 * me.w + me.q) * Cta<NT, R>::LD + 2 * me.j;
#pragma unroll
  for (int t = 0; t < NT; t++)
#pragma unroll
    for (int e = 0; e < 2; e++) p[8 * t + e] = pack(S, c[t].re[e], c[t].im[e]);
}

// column-pattern read of the shared tile (right operand)
template <int NT, bool FULL, typename R, typename V2>
__device__ __forceinline__ void tile_cols(const V2* S, const Who<NT, FULL>& me, int rb, int cb, OpT<R> (&o)[2]) {
  const V2* p = S + (8 * rb + 2 * me.j) * Cta<NT, R>::LD + 8 * cb + me.q;
#pragma unroll
  for (int e = 0; e < 2; e++) {
    const V2 v = p[e * Cta<NT, R>::LD];
    o[e].re = v.x;
    o[e].im = v.y;
  }
}

__device__ __forceinline__ double inv_factorial(int k, int order) {
  constexpr double f[9] = {1.0,       1.0,       1.0 / 2,   1.0 / 6,   1.0 / 24,
                           1.0 / 120, 1.0 / 720, 1.0 / 5040, 1.0 / 40320};
  double v = 0.0;
#pragma unroll
  for (int i = 0; i < 9; i++)
    if (i == k && i <= order) v = f[i];
  return v;
}

// mode 0: Pout = Pin - kick F(U);  1: the same, and Uout = exp(i dt Pout) U;
// 2: Uout = exp(i dt Pin) U and Pout = Pin.  SUMS (mode 0, 1): v += (ReTr W, ReTr P P) of own
// rows, P after a kick alone (the end of a trajectory), before a kick and drift
// (its start).
//
// The exponential is the Taylor sum by Paterson-Stockmeyer in blocks of three
// terms (X^2, X^3, then Horner in X^3: 5 products for order 8, 4 for order 6,
// U included, instead of 8 and 6 by Horner), formed without its identity term:
// U' = U + (E - 1) U.  P is not assumed Hermitian.
// FP32 storage with `project`: U' = U + (E - 1 - (U U^dag - 1) / 2) U, the
// Newton-Schulz step on the links as read; it differs from projecting U' by
// |E - 1| times the defect that the FP32 store left, which the next update
// removes in turn.  That is enough while E is unitary to rounding.  Where rows
// of U' say that it is not (low LEVEL, large steps) or that U was not (uploaded
// links), U' takes the step itself, U' - (U' U'^dag - 1) U' / 2: one vote a link,
// SU(8) 10^4 90.3 -> 91.0, SU(32) 6^4 541 -> 546 us a step; left to the next update,
// links after SU(8) steps of 0.1 at LEVEL 2 were 7e-3 off U(8) instead of 5e-5.
constexpr float ROW_TOLERANCE = 0x1p-22f;  // of a squared row length; rounding of stored entries: std 3e-8

template <int NT, bool FULL, typename S2, bool SUMS, typename R>
__device__ __forceinline__ void update_link(const Job& job, int idx, const Who<NT, FULL>& me, int slot, int cur,
                                            double kick_scale, int mode, typename Cta<NT, R>::V2* S, double (&v)[2]) {
  using CT = Cta<NT, R>;
  using V2 = typename CT::V2;
  using Acc = AccT<R>;
  using Op = OpT<R>;
  // left operands from memory: the k loop stays rolled for large NC; in TF32, whose
  // k step is three times the instructions, by two at NT = 4 (unrolled it runs out
  // of instruction cache: SU(32) 8^4 2040 us a step, by two 1684, by one 1727; SU(24)
  // 6^3 30.5 unrolled, 32.3 by one; FP64 SU(32) 6^4 720 unrolled, 749 by two)
  constexpr int KU = NT < 4 ? NT : NT > 4 ? 1 : sizeof(R) == 4 ? 2 : 4;
  constexpr int FINE = fine_force(NT, FULL);
  const int lane = threadIdx.x & 31;
  const int V = job.V, D = job.D;
  const int x = idx / D, mu = idx - x * D;
  const size_t NN = FULL ? (size_t)64 * NT * NT : (size_t)me.n * me.n;
  const S2* U = static_cast<const S2*>(job.U[cur]);
  const int* __restrict__ nbr = job.nbr;
  auto link = [&](int d, int s) { return U + ((size_t)d * V + s) * NN; };
  const size_t own = ((size_t)mu * V + x) * NN;
  const S2* Ux = U + own;
  const int r = 8 * me.w + me.q;
  Acc X[NT];  // rows of X = i dt P

  // ReTr(P P) of own rows, through the tile
  auto kinetic = [&](const S2* P) {
    Op p[2], q[2];
#pragma unroll
    for (int t = 0; t < NT; t++) {
      me.own(P, t, p);
#pragma unroll
      for (int e = 0; e < 2; e++) S[r * CT::LD + 8 * t + 2 * me.j + e] = pack(S, p[e].re, p[e].im);
    }
    link_sync<NT>(slot);
#pragma unroll
    for (int t = 0; t < NT; t++) {
      me.own(P, t, p);
      tile_cols(S, me, t, me.w, q);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        v[1] = fma((double)p[e].re, (double)q[e].re, v[1]);
        v[1] = fma(-(double)p[e].im, (double)q[e].im, v[1]);
      }
    }
    link_sync<NT>(slot);
  };

  if (mode != 2) {
    if (SUMS && mode == 1) kinetic(static_cast<const S2*>(job.Pin) + own);
    Acc W[NT];  // the staple sum S first
    zero(W);
    // lane nu fetches the neighbours of plane nu, all planes at once (D <= 16)
    const int xpmu = __ldg(nbr + (size_t)(2 * mu) * V + x);
    const int ln = min(lane, D - 1);
    const int xp = __ldg(nbr + (size_t)(2 * ln) * V + x), xm = __ldg(nbr + (size_t)(2 * ln + 1) * V + x),
              xpm = __ldg(nbr + (size_t)(2 * ln + 1) * V + xpmu);
#pragma unroll 1
    for (int nu = 0; nu < D; nu++) {
      if (nu == mu) continue;
      const int xpnu = __shfl_sync(0xffffffffu, xp, nu), xmnu = __shfl_sync(0xffffffffu, xm, nu),
                xpmu_mnu = __shfl_sync(0xffffffffu, xpm, nu);
      Acc T[NT];
      {
        const S2 *a = link(nu, xpmu), *b = link(mu, xpnu), *y = link(nu, x);
        zero(T);
        prod<NT, true, KU, FINE>(
            T, [&](int kb, Op(&o)[2]) { me.rows(a, me.w, kb, o); },
            [&](int kb, int t, Op(&o)[2]) { me.rows(b, t, kb, o); });
        prod<NT, true, NT, FINE>(
            W, [&](int kb, Op(&o)[2]) { from_acc(T, kb, o); },
            [&](int kb, int t, Op(&o)[2]) { me.rows(y, t, kb, o); });
      }
      {
        const S2 *a = link(nu, xpmu_mnu), *b = link(mu, xmnu), *y = link(nu, xmnu);
        zero(T);
        prod<NT, true, KU, FINE>(
            T,
            [&](int kb, Op(&o)[2]) {
              me.cols(a, kb, me.w, o);
              o[0].im = -o[0].im;
              o[1].im = -o[1].im;
            },
            [&](int kb, int t, Op(&o)[2]) { me.rows(b, t, kb, o); });
        prod<NT, false, NT, FINE>(
            W, [&](int kb, Op(&o)[2]) { from_acc(T, kb, o); },
            [&](int kb, int t, Op(&o)[2]) { me.cols(y, kb, t, o); });
      }
    }
    tile_rows(S, me, W);
    link_sync<NT>(slot);
    zero(W);
    prod<NT, false, KU, FINE>(
        W, [&](int kb, Op(&o)[2]) { me.rows(Ux, me.w, kb, o); },
        [&](int kb, int t, Op(&o)[2]) { tile_cols(S, me, kb, t, o); });
    link_sync<NT>(slot);
    tile_rows(S, me, W);
    link_sync<NT>(slot);
    // kick with the traceless anti-hermitian part of W: z = W_cr
    const int N = me.N();
    R trim = R(0);
    for (int k = 0; k < N; k++) trim += S[k * (CT::LD + 1)].y;
    trim = trim / R(N);
    const R ek = (R)(kick_scale * job.kick), ed = (R)job.dt;
    const S2* P = static_cast<const S2*>(job.Pin) + own;
    S2* Po = static_cast<S2*>(job.Pout) + own;
#pragma unroll
    for (int t = 0; t < NT; t++) {
      Op z[2];
      tile_cols(S, me, t, me.w, z);
      Op p[2];
      me.own(P, t, p);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int c = 8 * t + 2 * me.j + e;
        const R fr = r == c ? W[t].im[e] - trim : R(0.5) * (W[t].im[e] + z[e].im);
        const R fi = r == c ? R(0) : R(-0.5) * (W[t].re[e] - z[e].re);
        p[e].re = round_to(P, fma(-ek, fr, p[e].re));
        p[e].im = round_to(P, fma(-ek, fi, p[e].im));
        X[t].re[e] = -ed * p[e].im;
        X[t].im[e] = ed * p[e].re;
      }
      me.put(Po, t, p);
    }
    if (SUMS) {
#pragma unroll
      for (int t = 0; t < NT; t++)
#pragma unroll
        for (int e = 0; e < 2; e++) v[0] += r == 8 * t + 2 * me.j + e ? (double)W[t].re[e] : 0.0;
    }
    link_sync<NT>(slot);
    if (SUMS && mode == 0) kinetic(Po);
    if (mode == 0) return;
  } else {
    const S2* P = static_cast<const S2*>(job.Pin) + own;
    S2* Po = static_cast<S2*>(job.Pout) + own;
    const R ed = (R)job.dt;
#pragma unroll
    for (int t = 0; t < NT; t++) {
      Op p[2];
      me.rows(P, me.w, t, p);
      me.put(Po, t, p);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        X[t].re[e] = -ed * p[e].im;
        X[t].im[e] = ed * p[e].re;
      }
    }
  }
  const int order = job.order;
  // rows of X again where keeping them costs registers: from the momenta just
  // written (or read), which this thread owns
  auto x_rows = [&](int t, Op(&o)[2]) {
    if constexpr (CT::KEEP) {
      from_acc(X, t, o);
    } else {
      const S2* P = (mode == 2 ? static_cast<const S2*>(job.Pin) : static_cast<const S2*>(job.Pout)) + own;
      const R ed = (R)job.dt;
      Op p[2];
      me.own(P, t, p);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        o[e].re = -ed * p[e].im;
        o[e].im = ed * p[e].re;
      }
    }
  };
  tile_rows(S, me, X);
  link_sync<NT>(slot);
  Acc E[NT], X2[NT];
  V2* S2t = S + CT::TILE;  // X^2, own rows only (not KEEP)
  auto tile_row = [&](const V2* tile, int kb, Op(&o)[2]) {
    const V2* p = tile + r * CT::LD + 8 * kb + 2 * me.j;
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const V2 v = p[e];
      o[e].re = v.x;
      o[e].im = v.y;
    }
  };
  zero(X2);
  prod<NT, false, KU>(
      X2,
      [&](int kb, Op(&o)[2]) {
        if constexpr (CT::KEEP)
          from_acc(X, kb, o);
        else
          tile_row(S, kb, o);
      },
      [&](int kb, int t, Op(&o)[2]) { tile_cols(S, me, kb, t, o); });
  if constexpr (!CT::KEEP) tile_rows(S2t, me, X2);
  auto x2_rows = [&](int kb, Op(&o)[2]) {
    if constexpr (CT::KEEP)
      from_acc(X2, kb, o);
    else
      tile_row(S2t, kb, o);
  };
  auto block = [&](Acc(&c)[NT], int k) {  // sum_{i<3} X^i / (k + i)!, the identity of k = 0 left out
    const R a0 = k ? (R)inv_factorial(k, order) : R(0), a1 = (R)inv_factorial(k + 1, order),
            a2 = (R)inv_factorial(k + 2, order);
#pragma unroll
    for (int t = 0; t < NT; t++) {
      Op o[2], o2[2];
      x_rows(t, o);
      x2_rows(t, o2);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        c[t].re[e] = fma(a2, o2[e].re, fma(a1, o[e].re, r == 8 * t + 2 * me.j + e ? a0 : R(0)));
        c[t].im[e] = fma(a2, o2[e].im, a1 * o[e].im);
      }
    }
  };
  int k = order - order % 3;
  if (k == 0) {
    block(E, 0);
  } else {
    {
      Acc X3[NT];
      zero(X3);
      prod<NT, false, KU>(
          X3, [&](int kb, Op(&o)[2]) { x2_rows(kb, o); },
          [&](int kb, int t, Op(&o)[2]) { tile_cols(S, me, kb, t, o); });
      link_sync<NT>(slot);
      tile_rows(S, me, X3);
      if (k == order) {  // the top block is the single term X^k / k!: joined to the next one down
        k -= 3;
        block(E, k);
        const R a = (R)inv_factorial(order, order);
#pragma unroll
        for (int t = 0; t < NT; t++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            E[t].re[e] = fma(a, X3[t].re[e], E[t].re[e]);
            E[t].im[e] = fma(a, X3[t].im[e], E[t].im[e]);
          }
      } else {
        block(E, k);
      }
    }
    link_sync<NT>(slot);
#pragma unroll 1
    while (k > 0) {
      // large matrices read the tile anew: its loads hoisted out of the loop would all spill
      if (NT > 2) asm volatile("" ::: "memory");
      k -= 3;
      Acc H[NT];
      block(H, k);
      prod<NT, false, NT>(
          H, [&](int kb, Op(&o)[2]) { from_acc(E, kb, o); },
          [&](int kb, int t, Op(&o)[2]) { tile_cols(S, me, kb, t, o); });
#pragma unroll
      for (int t = 0; t < NT; t++) E[t] = H[t];
    }
  }
  if (sizeof(S2) == 8 && job.project) {
    AccT<double> M[NT];  // always in FP64: what counts is its distance from 1
    zero(M);
    prod<NT, true, KU>(
        M, [&](int kb, OpT<double>(&o)[2]) { me.rows(Ux, me.w, kb, o); },
        [&](int kb, int t, OpT<double>(&o)[2]) { me.rows(Ux, t, kb, o); });
    float d = 0.f;  // of the squared length of row r from 1
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const bool diag = r == 8 * t + 2 * me.j + e && (FULL || r < me.n);
        M[t].re[e] -= diag ? 1.0 : 0.0;
        if (diag) d = (float)M[t].re[e];
      }
    d += __shfl_xor_sync(0xffffffffu, d, 1);
    d += __shfl_xor_sync(0xffffffffu, d, 2);
    // a row further off is left to the step on U' below
    const double half = fabsf(d) <= ROW_TOLERANCE ? 0.5 : 0.0;
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        E[t].re[e] -= (R)(half * M[t].re[e]);
        E[t].im[e] -= (R)(half * M[t].im[e]);
      }
  }
  // U' = U + (E - 1) U; FP32 sums the small product on its own
  Acc Y[NT];
  auto add_u = [&]() {
#pragma unroll
    for (int t = 0; t < NT; t++) {
      Op o[2];
      me.rows(Ux, me.w, t, o);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        Y[t].re[e] += o[e].re;
        Y[t].im[e] += o[e].im;
      }
    }
  };
  zero(Y);
  if constexpr (sizeof(R) == 8) add_u();
  prod<NT, false, NT>(
      Y, [&](int kb, Op(&o)[2]) { from_acc(E, kb, o); },
      [&](int kb, int t, Op(&o)[2]) { me.cols(Ux, kb, t, o); });
  if constexpr (sizeof(R) == 4) add_u();
  if (sizeof(S2) == 8 && job.project) {
    // rows of U' further from length 1 than rounding takes them: a Taylor sum or
    // links that are not unitary to rounding
    R n2 = R(0);
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
      for (int e = 0; e < 2; e++) n2 = fma(Y[t].re[e], Y[t].re[e], fma(Y[t].im[e], Y[t].im[e], n2));
    float n = (float)n2;
    n += __shfl_xor_sync(0xffffffffu, n, 1);
    n += __shfl_xor_sync(0xffffffffu, n, 2);
    const bool off = !(fabsf(n - 1.f) <= ROW_TOLERANCE) && (FULL || r < me.n);
    if (link_any<NT>(slot, off)) {
      tile_rows(S, me, Y);
      link_sync<NT>(slot);
      AccT<double> M[NT];
      zero(M);
      prod<NT, true, 1>(
          M,
          [&](int kb, OpT<double>(&o)[2]) {
            Op a[2];
            tile_row(S, kb, a);
#pragma unroll
            for (int e = 0; e < 2; e++) {
              o[e].re = a[e].re;
              o[e].im = a[e].im;
            }
          },
          [&](int kb, int t, OpT<double>(&o)[2]) {
            const V2* p = S + (8 * t + me.q) * CT::LD + 8 * kb + 2 * me.j;
#pragma unroll
            for (int e = 0; e < 2; e++) {
              const V2 v = p[e];
              o[e].re = v.x;
              o[e].im = v.y;
            }
          });
      Acc C[NT];
      zero(C);
#pragma unroll
      for (int t = 0; t < NT; t++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const bool diag = r == 8 * t + 2 * me.j + e && (FULL || r < me.n);
          E[t].re[e] = (R)(-0.5 * (M[t].re[e] - (diag ? 1.0 : 0.0)));
          E[t].im[e] = (R)(-0.5 * M[t].im[e]);
        }
      prod<NT, false, NT>(
          C, [&](int kb, Op(&o)[2]) { from_acc(E, kb, o); },
          [&](int kb, int t, Op(&o)[2]) { tile_cols(S, me, kb, t, o); });
#pragma unroll
      for (int t = 0; t < NT; t++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
          Y[t].re[e] += C[t].re[e];
          Y[t].im[e] += C[t].im[e];
        }
    }
  }
  grid_done();
  store_rows(static_cast<S2*>(job.U[cur ^ 1]) + own, me, Y);
}

template <int NT, bool FULL, typename S2, bool SUMS, typename R, bool TIGHT>
__global__ void __launch_bounds__(Cta<NT, R>::THREADS, TIGHT ? Cta<NT, R>::MIN_CTAS : 1)
    k_link(const __grid_constant__ Job one, const Job* __restrict__ table, const int2* __restrict__ items, int cur,
           double kick_scale, int mode) {
  grid_wait();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Job* __restrict__ jp = &one;
  int blk = blockIdx.x;
  if (table) {
    const int2 it = __ldg(items + blk);
    jp = table + it.x;
    blk = it.y;
  }
  const Job& job = *jp;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int slot = wid / NT;
  Who<NT, FULL> me;
  me.w = wid - slot * NT;
  me.q = lane >> 2;
  me.j = lane & 3;
  me.n = job.N;
  const int idx = blk * Cta<NT>::LINKS + slot;
  using CT = Cta<NT, R>;
  auto* S = reinterpret_cast<typename CT::V2*>(smem_raw) + slot * (CT::TILES * CT::TILE);
  double v[2] = {0.0, 0.0};
  // whole links: no barrier of a link is left waiting
  if (idx < job.V * job.D) update_link<NT, FULL, S2, SUMS, R>(job, idx, me, slot, cur, kick_scale, mode, S, v);
  if constexpr (SUMS) {
    misc::block_sum<2>(v);
    if (threadIdx.x == 0) {
      double* p = job.pairs + 2 * ((size_t)blk + (mode == 0 ? job.ctas : 0));
      p[0] = v[0];
      p[1] = v[1];
    }
  }
}

// Plaquette sums, NT warps per site: Re sum_ij (AB)_ij conj((DC)_ij) of every
// plane, A = U_mu(x), B = U_nu(x+mu), D = U_nu(x), C = U_mu(x+nu); the block's
// temporal and spatial sums go to plaq_partial[2 blk], [2 blk + 1].
// Two products a plane at the FP64 MMA rate, where a thread per site (NC < 16)
// or four threads per row (above) did them on the FMA pipe from uncoalesced
// loads: SU(8) 10^4 1222 -> 41 us, SU(16) 6^4 687 -> 47, SU(32) 8^4 5627 -> 422,
// SU(64) 4x8x16 2554 -> 310 (the products alone 13, 14, 350 and 175).
template <int NT, bool FULL, typename S2>
__global__ void __launch_bounds__(Cta<NT>::PLAQ_THREADS)
    k_plaq(const __grid_constant__ Job one, const Job* __restrict__ table, const int2* __restrict__ items, int cur) {
  constexpr int KU = NT <= 4 ? NT : 1;
  const Job* __restrict__ jp = &one;
  int blk = blockIdx.x;
  if (table) {
    const int2 it = __ldg(items + blk);
    jp = table + it.x;
    blk = it.y;
  }
  const Job& job = *jp;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int slot = wid / NT;
  const int V = job.V, D = job.D;
  Who<NT, FULL> me;
  me.w = wid - slot * NT;
  me.q = lane >> 2;
  me.j = lane & 3;
  me.n = job.N;
  const int x = blk * Cta<NT>::SITES + slot;
  const size_t NN = FULL ? (size_t)64 * NT * NT : (size_t)me.n * me.n;
  const S2* __restrict__ U = static_cast<const S2*>(job.U[cur]);
  const int* __restrict__ nbr = job.nbr;
  auto link = [&](int d, int s) { return U + ((size_t)d * V + s) * NN; };
  double v[2] = {0.0, 0.0};
  if (x < V && x >= job.r0 && (job.r1 == 0 || x < job.r1)) {
#pragma unroll 1
    for (int mu = 0; mu < D; mu++) {
      const int xpmu = __ldg(nbr + (size_t)(2 * mu) * V + x);
#pragma unroll 1
      for (int nu = mu + 1; nu < D; nu++) {
        const int xpnu = __ldg(nbr + (size_t)(2 * nu) * V + x);
        const S2 *a = link(mu, x), *b = link(nu, xpmu), *d = link(nu, x), *c = link(mu, xpnu);
        Acc AB[NT], DC[NT];
        zero(AB);
        zero(DC);
        prod<NT, false, KU>(
            AB, [&](int kb, Op(&o)[2]) { me.rows(a, me.w, kb, o); },
            [&](int kb, int t, Op(&o)[2]) { me.cols(b, kb, t, o); });
        prod<NT, false, KU>(
            DC, [&](int kb, Op(&o)[2]) { me.rows(d, me.w, kb, o); },
            [&](int kb, int t, Op(&o)[2]) { me.cols(c, kb, t, o); });
        double tr = 0.0;
#pragma unroll
        for (int t = 0; t < NT; t++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            tr = fma(AB[t].re[e], DC[t].re[e], tr);
            tr = fma(AB[t].im[e], DC[t].im[e], tr);
          }
        v[mu == 0 ? 0 : 1] += (me.w == 0 && lane == 0 ? 1.0 : 0.0) - tr / me.N();
      }
    }
  }
  misc::block_sum<2>(v);
  if (!table) {
    misc::publish<2>(v, job.plaq_partial, job.out, job.ticket);
  } else if (threadIdx.x == 0) {
    job.plaq_partial[2 * (size_t)blk + 0] = v[0];
    job.plaq_partial[2 * (size_t)blk + 1] = v[1];
  }
}

// Kinetic sums sum ReTr(P P) and, with Pin2, sum ReTr((P + P2)^2) / 4: a warp takes 8 x 8 tiles of a link's matrix, each
// with its mirror tile in the column pattern (whole sectors, where element pairs
// read a row length apart took 365 us for SU(64) 4x8x16 on 24 CTAs);
// KIN_TILES tiles per CTA, whole links; three sums per CTA and their totals for
// one lattice, kin_partial[blk] in a batch.
constexpr int KIN_TILES = 64;
__host__ __device__ inline int kin_links(int N) {
  const int nt = (N + 7) / 8;
  return KIN_TILES / (nt * nt) > 0 ? KIN_TILES / (nt * nt) : 1;
}
template <typename S2>
__global__ void __launch_bounds__(misc::RED_THREADS)
    k_kinetic(const __grid_constant__ Job one, const Job* __restrict__ table, const int2* __restrict__ items) {
  const Job* __restrict__ jp = &one;
  int blk = blockIdx.x;
  if (table) {
    const int2 it = __ldg(items + blk);
    jp = table + it.x;
    blk = it.y;
  }
  const Job& job = *jp;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int N = job.N, nt = (N + 7) / 8;
  const long nl = (long)job.V * job.D;
  const long l0 = (long)blk * kin_links(N);
  const int links = (int)min((long)kin_links(N), nl - l0);
  Who<8, false> me;
  me.w = 0;
  me.q = lane >> 2;
  me.j = lane & 3;
  me.n = N;
  double v[2] = {0.0, 0.0};
  for (int f = wid; f < links * nt * nt; f += misc::RED_THREADS / 32) {
    const long l = l0 + f / (nt * nt);
    const int t = f % (nt * nt), ti = t / nt, tj = t - ti * nt;
    const int s = (int)(l % job.V);
    if (!(s >= job.r0 && (job.r1 == 0 || s < job.r1))) continue;
    const S2* P = static_cast<const S2*>(job.Pin) + (size_t)l * N * N;
    Op p[2], q[2];
    me.rows(P, ti, tj, p);
    me.cols(P, tj, ti, q);
#pragma unroll
    for (int e = 0; e < 2; e++) {
      v[0] = fma(p[e].re, q[e].re, v[0]);
      v[0] = fma(-p[e].im, q[e].im, v[0]);
    }
    if (job.Pin2) {
      const S2* P2 = static_cast<const S2*>(job.Pin2) + (size_t)l * N * N;
      Op p2[2], q2[2];
      me.rows(P2, ti, tj, p2);
      me.cols(P2, tj, ti, q2);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        v[1] = fma(p[e].re + p2[e].re, q[e].re + q2[e].re, v[1]);
        v[1] = fma(-(p[e].im + p2[e].im), q[e].im + q2[e].im, v[1]);
      }
    }
  }
  misc::block_sum<2>(v);
  if (!table) {
    const double w[3] = {v[0], 0.25 * v[1], 0.0};
    misc::publish<3>(w, job.kin_partial, job.out, job.ticket);
  } else if (threadIdx.x == 0) {
    job.kin_partial[blk] = v[0];
  }
}

// UViol (sun.cpp:441-471): sum ReTr((U U^dag - 1)^2), the matrix Hermitian, so
// the sum of its squared moduli; SITES links per CTA.
template <int NT, bool FULL, typename S2>
__global__ void __launch_bounds__(Cta<NT>::PLAQ_THREADS) k_uviol(const __grid_constant__ Job job) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int slot = wid / NT;
  Who<NT, FULL> me;
  me.w = wid - slot * NT;
  me.q = lane >> 2;
  me.j = lane & 3;
  me.n = job.N;
  const long l = (long)blockIdx.x * Cta<NT>::SITES + slot;
  const int s = (int)(l % job.V);
  double v[1] = {0.0};
  if (l < (long)job.V * job.D && s >= job.r0 && (job.r1 == 0 || s < job.r1)) {
    const S2* u = static_cast<const S2*>(job.U[0]) + (size_t)l * me.N() * me.N();
    Acc M[NT];
    zero(M);
    prod<NT, true, (NT <= 4 ? NT : 1)>(
        M, [&](int kb, Op(&o)[2]) { me.rows(u, me.w, kb, o); },
        [&](int kb, int t, Op(&o)[2]) { me.rows(u, t, kb, o); });
    const int r = 8 * me.w + me.q;
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const double re = M[t].re[e] - (r == 8 * t + 2 * me.j + e && r < me.N() ? 1.0 : 0.0);
        v[0] = fma(re, re, v[0]);
        v[0] = fma(M[t].im[e], M[t].im[e], v[0]);
      }
  }
  misc::block_sum<1>(v);
  const double w[3] = {0.0, 0.0, v[0]};
  misc::publish<3>(w, job.kin_partial, job.out, job.ticket);
}

// Gauss law: sum over the links of Pi - U^dag Pi U (lines.cuh), NT warps per
// group, each group's links accumulated in its warps' registers with a grid
// stride; the group's matrix goes to kin_partial[g * 2 NC^2 + 2 e + {0, 1}].
template <int NT, bool FULL, typename S2>
__global__ void __launch_bounds__(Cta<NT>::PLAQ_THREADS) k_gauss(const __grid_constant__ Job job, int ngroups) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int slot = wid / NT;
  Who<NT, FULL> me;
  me.w = wid - slot * NT;
  me.q = lane >> 2;
  me.j = lane & 3;
  me.n = job.N;
  const int g = blockIdx.x * Cta<NT>::SITES + slot;
  if (g >= ngroups) return;
  const int N = me.N();
  const long nl = (long)job.V * job.D;
  Acc G[NT];
  zero(G);
  for (long l = g; l < nl; l += ngroups) {
    const S2* u = static_cast<const S2*>(job.U[0]) + (size_t)l * N * N;
    const S2* p = static_cast<const S2*>(job.Pin) + (size_t)l * N * N;
    Acc T[NT];
    zero(T);
    prod<NT, false, (NT <= 4 ? NT : 1)>(
        T,
        [&](int kb, Op(&o)[2]) {  // -U^dag
          me.cols(u, kb, me.w, o);
          o[0].re = -o[0].re;
          o[1].re = -o[1].re;
        },
        [&](int kb, int t, Op(&o)[2]) { me.cols(p, kb, t, o); });
    prod<NT, false, NT>(
        G, [&](int kb, Op(&o)[2]) { from_acc(T, kb, o); },
        [&](int kb, int t, Op(&o)[2]) { me.cols(u, kb, t, o); });
#pragma unroll
    for (int t = 0; t < NT; t++) {
      Op o[2];
      me.rows(p, me.w, t, o);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        G[t].re[e] += o[e].re;
        G[t].im[e] += o[e].im;
      }
    }
  }
  double2* out = reinterpret_cast<double2*>(job.kin_partial) + (size_t)g * N * N;
#pragma unroll
  for (int t = 0; t < NT; t++) {
    const int r = 8 * me.w + me.q, c = 8 * t + 2 * me.j;
#pragma unroll
    for (int e = 0; e < 2; e++)
      if (FULL || (r < N && c + e < N)) out[r * N + c + e] = make_double2(G[t].re[e], G[t].im[e]);
  }
}

// Closed lines (LineSet of lines.cuh), NT warps per line: the running product
// is each warp's accumulator rows, so a link of the line is one product with no
// barrier.  ev null: out[q] = |Tr W_q| / NC; else the eigenvalues of W_q by one
// warp from shared memory (eig.cuh).
template <int NT, bool FULL, typename S2>
__global__ void __launch_bounds__(32 * NT) k_lines(const __grid_constant__ Lat L, const S2* __restrict__ U,
                                                   const __grid_constant__ LineSet ls, double* __restrict__ out,
                                                   double2* __restrict__ ev, int* __restrict__ fail) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  Who<NT, FULL> me;
  me.w = threadIdx.x >> 5;
  me.q = lane >> 2;
  me.j = lane & 3;
  me.n = L.N;
  const int N = me.N();
  int start;
  const int dir = line_of(ls, blockIdx.x, &start);
  const S2* u = U + ((size_t)dir * L.V + start) * N * N;
  const size_t step = (size_t)L.stride[dir] * N * N;
  Acc W[NT];
#pragma unroll
  for (int t = 0; t < NT; t++) {
    Op o[2];
    me.rows(u, me.w, t, o);
#pragma unroll
    for (int e = 0; e < 2; e++) {
      W[t].re[e] = o[e].re;
      W[t].im[e] = o[e].im;
    }
  }
  for (int k = 1; k < L.n[dir]; k++) {
    u += step;
    Acc T[NT];
    zero(T);
    prod<NT, false, NT>(
        T, [&](int kb, Op(&o)[2]) { from_acc(W, kb, o); },
        [&](int kb, int t, Op(&o)[2]) { me.cols(u, kb, t, o); });
#pragma unroll
    for (int t = 0; t < NT; t++) W[t] = T[t];
  }
  const int r = 8 * me.w + me.q;
  if (ev) {
    cpx<double>* H = reinterpret_cast<cpx<double>*>(smem_raw);
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int c = 8 * t + 2 * me.j + e;
        if (r < N && c < N) H[r * N + c] = mkc<double>(W[t].re[e], W[t].im[e]);
      }
    __syncthreads();
    if (threadIdx.x < 32) {
      cpx<double>* v = H + N * N;
      cpx<double>* e = v + N;
      eig::hessenberg_qr(H, N, v, e, fail);
      __syncwarp();
      for (int i = lane; i < N; i += 32) ev[(size_t)blockIdx.x * N + i] = make_double2(e[i].re, e[i].im);
    }
    return;
  }
  double v[2] = {0.0, 0.0};
#pragma unroll
  for (int t = 0; t < NT; t++)
#pragma unroll
    for (int e = 0; e < 2; e++)
      if (r == 8 * t + 2 * me.j + e && r < N) {
        v[0] += W[t].re[e];
        v[1] += W[t].im[e];
      }
  misc::block_sum<2>(v);
  if (threadIdx.x == 0) out[blockIdx.x] = hypot(v[0], v[1]) / N;
}

}  // namespace m64
}  // namespace askja
