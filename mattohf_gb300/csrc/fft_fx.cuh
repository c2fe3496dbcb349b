// Complex FFT in 64-bit fixed point for the exchange's pair transforms.
//
// GB300 issues about 1.8 FP64 operations per clock and SM, but 32 multiply-adds
// 32 x 32 + 64 -> 64 bits (mad.wide) and 67 additions of 64 bits (measured
// with independent chains).  A pair transform needs no exponent range: its
// values are bounded by the norms of the two orbitals.  So pair densities,
// transforms, kernel products and sums run on 64-bit integers, scaled so that
// no value can reach 2^61.  That keeps 8 more bits than an FP64 significand
// under the largest value, which covers the rounding of the longest sums.
//
// Numbers.  A value v stands for v / 2^60 (a twiddle, a kernel factor) or for
// an orbital-like quantity with a scale of its own (k_fock_fx.cu).  Products
// take both factors as limbs, v = h 2^30 + l with 0 <= l < 2^30:
//     h h' + ((h l' + l h') >> 30) + 1.
// The product l l' is not formed; the 1 makes up for its mean and for the
// truncation, so that the rounding has no bias (a bias of half a place in
// every pair density would add up to 2^-53 of the transform's largest value).
// With |v| < 2^61 the limbs fit 32 bits and the sums of a complex product 64.
//
// The multiply-adds are written as mad.wide because the compiler makes a full
// 64 x 64 product of the same expression in C++ (32 instead of 12 multiplies
// per complex product, counted with ncu).
//
// Transform.  A Stockham transform over T lanes of E values with equal first
// and last radix, so that input and output use the same register positions
//     pos(tl, e) = tl + T (e / R0) + (N / R0) (e % R0),
// and one piece of code serves both directions: the backward transform of z
// is conj(forward(conj z)), and the caller's kernel product conjugates.  The
// pair loop is thus about 2000 instructions with E = 8, which matters: with
// E = 16 and both directions unrolled (8000 instructions) the warps waited
// two issue slots for instructions for every one they issued.
#pragma once
#include <cuda_runtime.h>

namespace mattohf {
namespace fx {

using i64 = long long;

struct alignas(16) cx {  // complex fixed-point number
  i64 x, y;
};
struct alignas(16) lc {  // complex number in limbs
  int xh, xl, yh, yl;
};

constexpr int kLimb = 30;
constexpr int kOne = 60;  // log2 of the fixed-point one of twiddles and kernels

__device__ __forceinline__ int hi_limb(i64 v) { return (int)(v >> kLimb); }
__device__ __forceinline__ int lo_limb(i64 v) { return (int)v & ((1 << kLimb) - 1); }
__device__ __forceinline__ lc limbs(cx a) { return lc{hi_limb(a.x), lo_limb(a.x), hi_limb(a.y), lo_limb(a.y)}; }
// a b + c and a b, 32 x 32 (+ 64) -> 64 bits
__device__ __forceinline__ i64 mw(int a, int b, i64 c) {
  i64 d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}
__device__ __forceinline__ i64 mw(int a, int b) {
  i64 d;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(d) : "r"(a), "r"(b));
  return d;
}
// -v - 1 for a number in limbs, low limb again in [0, 2^30).  The products below
// use it for -v: the factors it is applied to are 2^60 for 1, so the change is
// below the last place of a 60-bit factor.
__device__ __forceinline__ int neg_hi(int h) { return ~h; }
__device__ __forceinline__ int neg_lo(int l) { return l ^ ((1 << kLimb) - 1); }

__device__ __forceinline__ cx add(cx a, cx b) { return cx{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ cx sub(cx a, cx b) { return cx{a.x - b.x, a.y - b.y}; }

// Each component below drops two low products of mean 1/4 and truncates the
// middle sum (mean 1/2): the + 1 makes the mean error zero.  A rounding
// constant in the first multiply-add would cost two register moves a chain.
__device__ __forceinline__ i64 finish(i64 hh, i64 mid) { return hh + (mid >> kLimb) + 1; }
// a * b, nb = (neg_hi(b.yh), neg_lo(b.yl))
__device__ __forceinline__ cx cmul(lc a, lc b, int2 nb) {
  const i64 mr = mw(a.xh, b.xl, mw(a.xl, b.xh, mw(a.yh, nb.y, mw(a.yl, nb.x))));
  const i64 mi = mw(a.xh, b.yl, mw(a.xl, b.yh, mw(a.yh, b.xl, mw(a.yl, b.xh))));
  return cx{finish(mw(a.xh, b.xh, mw(a.yh, nb.x)), mr), finish(mw(a.xh, b.yh, mw(a.yh, b.xh)), mi)};
}
__device__ __forceinline__ cx cmul(lc a, lc b) { return cmul(a, b, make_int2(neg_hi(b.yh), neg_lo(b.yl))); }
// a * conj(b)
__device__ __forceinline__ cx cmulc(lc a, lc b) {
  const int nyh = neg_hi(b.yh), nyl = neg_lo(b.yl);
  const i64 mr = mw(a.xh, b.xl, mw(a.xl, b.xh, mw(a.yh, b.yl, mw(a.yl, b.yh))));
  const i64 mi = mw(a.xh, nyl, mw(a.xl, nyh, mw(a.yh, b.xl, mw(a.yl, b.xh))));
  return cx{finish(mw(a.xh, b.xh, mw(a.yh, b.yh)), mr), finish(mw(a.xh, nyh, mw(a.yh, b.xh)), mi)};
}
// Limbs of a real factor with the low limb in [2^29, 3 2^29): the one dropped
// low product of rmul then has mean 1/2 as well.
__host__ __device__ __forceinline__ int2 real_limbs(i64 v) {
  const i64 o = 1ll << (kLimb - 1), l = ((v - o) & ((1ll << kLimb) - 1)) + o;
  return make_int2((int)((v - l) >> kLimb), (int)l);
}
// a * k for a real factor k in real_limbs
__device__ __forceinline__ i64 rmul(i64 a, int2 k) {
  const int ah = hi_limb(a), al = lo_limb(a);
  return finish(mw(ah, k.x), mw(ah, k.y, mw(al, k.x)));
}

// sqrt(1/2) times 2^60, nearest integer, in limbs (its low limb is within 0.6 % of
// the mean that rmul wants)
constexpr int kC8h = 759250124, kC8l = 1067312712;

__device__ __forceinline__ i64 rmul_c8(i64 a) { return rmul(a, make_int2(kC8h, kC8l)); }

// Forward transforms (exp(-2 pi i n k / R)) of R values in place.
template <int R> struct Dft;
template <> struct Dft<2> {
  __device__ __forceinline__ static void run(cx* x) {
    const cx a = x[0];
    x[0] = add(a, x[1]);
    x[1] = sub(a, x[1]);
  }
};
template <> struct Dft<4> {
  __device__ __forceinline__ static void run(cx& x0, cx& x1, cx& x2, cx& x3) {
    const cx e0 = add(x0, x2), e1 = sub(x0, x2), e2 = add(x1, x3), e3 = sub(x1, x3);
    x0 = add(e0, e2);
    x2 = sub(e0, e2);
    x1 = cx{e1.x + e3.y, e1.y - e3.x};
    x3 = cx{e1.x - e3.y, e1.y + e3.x};
  }
  __device__ __forceinline__ static void run(cx* x) { run(x[0], x[1], x[2], x[3]); }
};
template <> struct Dft<8> {
  __device__ __forceinline__ static void run(cx* x) {
    cx a0 = x[0], a1 = x[2], a2 = x[4], a3 = x[6], b0 = x[1], b1 = x[3], b2 = x[5], b3 = x[7];
    Dft<4>::run(a0, a1, a2, a3);
    Dft<4>::run(b0, b1, b2, b3);
    // b1 (1 - i) / sqrt 2 and, up to the sign, b3 (-1 - i) / sqrt 2
    const cx t1{rmul_c8(b1.x + b1.y), rmul_c8(b1.y - b1.x)};
    const cx t3{rmul_c8(b3.y - b3.x), rmul_c8(b3.x + b3.y)};
    x[0] = add(a0, b0);
    x[4] = sub(a0, b0);
    x[1] = add(a1, t1);
    x[5] = sub(a1, t1);
    x[2] = cx{a2.x + b2.y, a2.y - b2.x};
    x[6] = cx{a2.x - b2.y, a2.y + b2.x};
    x[3] = cx{a3.x + t3.x, a3.y - t3.y};
    x[7] = cx{a3.x - t3.x, a3.y + t3.y};
  }
};

// Radices (first = last; R1 = 1: two passes) and lanes.  V = 1: where few
// transforms run at a time, 64 points on 16 lanes (half the chain of a lane).
template <int N, int V = 0> struct Plan : Plan<N, 0> {};
template <> struct Plan<16, 0> { static constexpr int R0 = 4, R1 = 1, T = 4; };
template <> struct Plan<32, 0> { static constexpr int R0 = 4, R1 = 2, T = 8; };
template <> struct Plan<64, 0> { static constexpr int R0 = 8, R1 = 1, T = 8; };
template <> struct Plan<128, 0> { static constexpr int R0 = 4, R1 = 8, T = 16; };
template <> struct Plan<256, 0> { static constexpr int R0 = 8, R1 = 4, T = 32; };
template <> struct Plan<512, 0> { static constexpr int R0 = 8, R1 = 8, T = 64; };
template <> struct Plan<64, 1> { static constexpr int R0 = 4, R1 = 4, T = 16; };

template <int N, int V = 0> struct Team {
  static constexpr int R0 = Plan<N, V>::R0, R1 = Plan<N, V>::R1, T = Plan<N, V>::T;
  static constexpr int E = N / T, STRIDE = N / R0;
  __device__ __forceinline__ static int pos(int tl, int e) { return tl + T * (e / R0) + STRIDE * (e % R0); }
  // register slot of lane 0 that holds the self-aliased frequency N/2
  static constexpr int kNyquistSlot = R0 / 2;
  // twiddle table: middle pass [R1][R0] of W_(R0 R1), then last pass [R0][N/R0] of W_N
  static constexpr int kTwLast = R1 > 1 ? R0 * R1 : 0;
  static constexpr int kTwCount = kTwLast + N;
};

// Slot of element i in the team buffer (fft_slot of fft.cuh: conflict-free
// stores of the first pass, unit-stride accesses stay so).
__device__ __forceinline__ int slot(int i) { return i ^ ((i >> 3) & 7); }

// A team of 64 lanes is two warps: it meets at named barrier 1 + team.
// ALONE: the team is the only one of its warp (lanes 0 .. T - 1).
template <int T, bool ALONE = false>
__device__ __forceinline__ void team_sync(int team) {
  if constexpr (T > 32) asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(T) : "memory");
  else if constexpr (ALONE && T < 32) __syncwarp((1u << T) - 1);
  else __syncwarp();
}

// Forward transform of x in place (slots pos); twn: the negated imaginary parts
// of the twiddles, as neg_hi and neg_lo.
template <int N, bool ALONE = false, int V = 0>
__device__ __forceinline__ void forward(cx (&x)[Team<N, V>::E], cx* buf, const lc* __restrict__ tw,
                                        const int2* __restrict__ twn, int tl, int team) {
  using TM = Team<N, V>;
  constexpr int R0 = TM::R0, R1 = TM::R1, T = TM::T, E = TM::E;
#pragma unroll
  for (int p = 0; p < E / R0; ++p) Dft<R0>::run(&x[p * R0]);
  team_sync<T, ALONE>(team);
#pragma unroll
  for (int p = 0; p < E / R0; ++p)
#pragma unroll
    for (int r = 0; r < R0; ++r) buf[slot((tl + T * p) * R0 + r)] = x[p * R0 + r];
  team_sync<T, ALONE>(team);
  if constexpr (R1 > 1) {
    constexpr int NB = N / R1;
#pragma unroll
    for (int p = 0; p < E / R1; ++p) {
      const int j = tl + T * p, k = j % R0;
      cx* y = &x[p * R1];
#pragma unroll
      for (int r = 0; r < R1; ++r) y[r] = buf[slot(j + r * NB)];
#pragma unroll
      for (int r = 1; r < R1; ++r) y[r] = cmul(limbs(y[r]), tw[r * R0 + k], twn[r * R0 + k]);
      Dft<R1>::run(y);
    }
    team_sync<T, ALONE>(team);
#pragma unroll
    for (int p = 0; p < E / R1; ++p) {
      const int j = tl + T * p, base = (j / R0) * (R0 * R1) + j % R0;
#pragma unroll
      for (int r = 0; r < R1; ++r) buf[slot(base + r * R0)] = x[p * R1 + r];
    }
    team_sync<T, ALONE>(team);
  }
#pragma unroll
  for (int p = 0; p < E / R0; ++p) {
    const int j = tl + T * p;
    cx* y = &x[p * R0];
#pragma unroll
    for (int r = 0; r < R0; ++r) y[r] = buf[slot(j + r * TM::STRIDE)];
#pragma unroll
    for (int r = 1; r < R0; ++r) {
      const int i = TM::kTwLast + r * TM::STRIDE + j;
      y[r] = cmul(limbs(y[r]), tw[i], twn[i]);
    }
    Dft<R0>::run(y);
  }
}

}  // namespace fx
}  // namespace mattohf
