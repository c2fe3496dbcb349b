// Between FP64 and the 64-bit fixed point of fft_fx.cuh: sizes, scales, conversions.
#pragma once
#include "fft_fx.cuh"

namespace mattohf {

using fx::cx;
using fx::i64;
using fx::lc;

// Sizes are taken from the high words of the doubles, in integer and FP32 work
// only: an FP64 pass over 65536 orbital values took 5.4 us, four fifths of it
// for two multiply-adds an element at 1.8 a clock and SM.
__device__ __forceinline__ float fx_mantissa(int h, int e) {  // |component| with high word h in units of 2^(e - 1023)
  const int x = (h >> 20) - e + 127;
  return x > 0 && h >= 0x100000 ? __int_as_float((x << 23) | ((h & 0xfffff) << 3)) : 0.0f;
}
// A size: x = high word of the largest |component|, y = the squared norm as a key
// that orders like it: 13 bits of binary exponent (biased by 2 * 1023), 18 of mantissa.
__device__ __forceinline__ int2 fx_size(int m, float s) {
  const int b = __float_as_int(s);
  return make_int2(m, m < 0x100000 ? 0 : (2 * (m >> 20) + (b >> 23) - 127) << 18 | ((b >> 5) & 0x3ffff));
}
__device__ __forceinline__ int2 fx_larger(int2 a, int2 b) { return make_int2(max(a.x, b.x), max(a.y, b.y)); }

// Size of one column, by a warp.
__device__ __forceinline__ int2 fx_column_size(const double2* __restrict__ p, int N, int lane) {
  int m = 0;
  for (int i = lane; i < N; i += 32) {
    const double2 z = p[i];
    m = max(m, max(__double2hiint(z.x) & 0x7fffffff, __double2hiint(z.y) & 0x7fffffff));
  }
  m = __reduce_max_sync(0xffffffffu, m);
  const int e = m >> 20;
  float s = 0.0f;
  for (int i = lane; i < N; i += 32) {
    const double2 z = p[i];
    const float x = fx_mantissa(__double2hiint(z.x) & 0x7fffffff, e), y = fx_mantissa(__double2hiint(z.y) & 0x7fffffff, e);
    s = fmaf(x, x, fmaf(y, y, s));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return fx_size(m, s);
}

// A short scale c 2^k, c in {8 .. 15}.  Conversions and scales below are integer
// and FP32 work: one FP64 instruction after another takes 64 cycles a warp, and
// with FP64 square roots and divisions a conversion launch took 14 us for 1536
// values.
struct Scale {
  int c, k;  // c = 0: not a number
};
__device__ __forceinline__ Scale fx_short_scale(float m, int e) {  // largest one that is not above m 2^e, m normal
  const int b = __float_as_int(m);
  return Scale{8 | ((b >> 20) & 7), (b >> 23) - 127 + e - 3};
}

// round(v c 2^k) for |v c 2^k| < 2^62: every bit of v counts
__device__ __forceinline__ i64 fx_convert(double v, Scale s) {
  const int hi = __double2hiint(v), ex = (hi >> 20) & 0x7ff;
  const unsigned long long m =
      ((unsigned long long)((hi & 0xfffff) | (ex ? 0x100000 : 0)) << 32 | (unsigned)__double2loint(v)) * (unsigned)s.c;
  const int sh = 1075 - (ex ? ex : 1) - s.k;  // value = m 2^-sh, m < 2^57
  const i64 r = sh > 58 ? 0 : sh > 0 ? (i64)((m + (1ull << (sh - 1))) >> sh) : (i64)(m << min(-sh, 8));
  return hi < 0 ? -r : r;
}

// bounds of the converted orbitals, with a margin for the FP32 arithmetic:
// 2^60.2 for the norm, 2^58.4 for a component (2^58.9 for a modulus)
constexpr float kNorm = 1.3241e18f, kPeak = 3.803e17f;

// s of a set of size z (largest component, largest squared norm; both short of the
// true ones by less than 2^-17).  Not a number when the set holds a value that is
// not finite; for a set of zeros (or
// denormal numbers), so large that every result scales back to zero.  peak: the
// bound of a component, n: further factor under the norm's.
__device__ __forceinline__ Scale fx_scale(int2 z, float peak, float n) {
  const int e = z.x >> 20;
  if (e >= 2047) return Scale{0, 0};
  if (z.x < 0x100000) return Scale{8, 2000};
  // norm^2 = g 2^(2 (e - 1023)); the key's exponent is within a few units of 2 e
  const float g = __int_as_float(((z.y >> 18) - 2 * e + 127) << 23 | (z.y & 0x3ffff) << 5);
  return fx_short_scale(fminf(kNorm * rsqrtf(g * n), peak / fx_mantissa(z.x, e)) * (1.0f - 1.0f / 16384.0f), 1023 - e);
}

__device__ __forceinline__ double pow2(int e) {  // 2^e, 0 or infinity outside the normal range
  return e > 1023 ? __longlong_as_double(0x7ff0000000000000ll) : e < -1022 ? 0.0 : __hiloint2double((e + 1023) << 20, 0);
}

// v 2^e for any e, to denormal numbers.  Not inlined: what is rare stays a branch, not
// an FP64 product of every value.
static __device__ __noinline__ double fx_times_pow2(double v, int e) { return v * pow2(e / 2) * pow2(e - e / 2); }

// 2^180 / (s^2 sd sk) as factor + correction: the product of the short factors
// is exact, its reciprocal is good to twice the precision.  Where a sum of 2^62 times the
// factor may leave the normal range downwards, both are 2^kTiny larger and negative
// (exchange_value takes that back).
constexpr int kTiny = 512;
__device__ __forceinline__ double2 fx_output_scale(Scale s, Scale sd, Scale sk) {
  if (s.c == 0 || sd.c == 0) return make_double2(__longlong_as_double(0x7ff8000000000000ll), 0.0);
  const int q = s.c * s.c * sd.c * sk.c;  // below 2^16
  const double dq = (double)q;
  double r = (double)(1.0f / (float)q);
  r = fma(fma(-r, dq, 1.0), r, r);
  r = fma(fma(-r, dq, 1.0), r, r);
  const double lo = fma(-r, dq, 1.0) * r;
  const int e0 = 180 - 2 * s.k - sd.k - sk.k, e = e0 < -800 ? e0 + kTiny : e0, h = e / 2;
  const double p = e0 < -800 ? -pow2(h) : pow2(h), p2 = pow2(e - h);
  return make_double2(r * p * p2, lo * p * p2);
}

// Scale of N values of size z (fx_block_size) that a transform takes: every partial sum is below sqrt(N) |v|_2 <= 2^60.2.  A power
// of two, so that scaling back is exact.
__device__ __forceinline__ Scale fx_fft_scale(int2 z, int N) {
  Scale s = fx_scale(z, 1e30f, (float)N);
  if (s.c) s.c = 8;
  return s;
}
// Back from such a scale: times 2^-(k + 3), which need not be a normal number, by the
// exponent field in integer work
struct Unscale {
  int e;
  bool ok;
  __device__ __forceinline__ double operator()(i64 v) const {
    const double d = (double)v;
    const int hi = __double2hiint(d), x = ((hi >> 20) & 0x7ff) + e;
    if (ok && hi != 0 && x > 0 && x < 0x7ff) return __hiloint2double(hi + (e << 20), __double2loint(d));
    return fx_times_pow2(ok ? d : __longlong_as_double(0x7ff8000000000000ll), e);
  }
};
__device__ __forceinline__ Unscale fx_unscale(Scale s) { return Unscale{-(s.k + 3), s.c != 0}; }

// Size of the values that a CTA's threads hold; red: two words per warp.  Two barriers.
template <int PER, int NWARP>
__device__ __forceinline__ int2 fx_block_size(const double2 (&v)[PER], int* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int m = 0;
#pragma unroll
  for (int p = 0; p < PER; ++p)
    m = max(m, max(__double2hiint(v[p].x) & 0x7fffffff, __double2hiint(v[p].y) & 0x7fffffff));
  m = __reduce_max_sync(0xffffffffu, m);
  if (lane == 0) red[warp] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < NWARP; ++w) m = max(m, red[w]);
  const int e = m >> 20;
  float s = 0.0f;
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    const float x = fx_mantissa(__double2hiint(v[p].x) & 0x7fffffff, e), y = fx_mantissa(__double2hiint(v[p].y) & 0x7fffffff, e);
    s = fmaf(x, x, fmaf(y, y, s));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) red[NWARP + warp] = __float_as_int(s);
  __syncthreads();
  s = 0.0f;
#pragma unroll
  for (int w = 0; w < NWARP; ++w) s += __int_as_float(red[NWARP + w]);
  return fx_size(m, s);
}

}  // namespace mattohf
