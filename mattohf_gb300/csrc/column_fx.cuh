// One column per CTA: fixed-point transforms on the CTA's first team, FP64 work
// spread over all its threads.
#pragma once
#include "fx_convert.cuh"
#include "internal.h"

namespace mattohf {

// Fixed xor-shuffle tree over the 32 lanes of a warp (deterministic order).
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Twiddles in shared memory (fixed point), loaded by the whole CTA.
template <int N>
struct FxTwiddles {
  lc w[fx::Team<N>::kTwCount];
  int2 n[fx::Team<N>::kTwCount];
  __device__ __forceinline__ void load(const lc* __restrict__ tw) {
    for (int i = threadIdx.x; i < fx::Team<N>::kTwCount; i += blockDim.x) {
      const lc v = tw[i];
      w[i] = v;
      n[i] = make_int2(fx::neg_hi(v.yh), fx::neg_lo(v.yl));
    }
  }
};

// Transform of buf (N fixed-point values) in place by the CTA's first team; every
// thread calls it, with buf complete, and finds it complete.
template <int N>
__device__ __forceinline__ void fx_block_forward(cx* buf, const FxTwiddles<N>& tw) {
  using TM = fx::Team<N>;
  __syncthreads();
  const int tl = threadIdx.x;
  if (tl < TM::T) {
    cx x[TM::E];
#pragma unroll
    for (int e = 0; e < TM::E; ++e) x[e] = buf[TM::pos(tl, e)];
    fx::forward<N, true>(x, buf, tw.w, tw.n, tl, 0);
    fx::team_sync<TM::T, true>(0);
#pragma unroll
    for (int e = 0; e < TM::E; ++e) buf[TM::pos(tl, e)] = x[e];
  }
  __syncthreads();
}

// Threads of a CTA that holds one column of N values, and values per thread.
template <int N>
struct ColumnCta {
  static constexpr int TH = N < 32 ? 32 : N > 128 ? 128 : N;
  static constexpr int PER = N > TH ? N / TH : 1;
  static constexpr int NW = TH / 32;
};

// Value of an exchange source.
__device__ __forceinline__ double2 exchange_value(const ExSource& s, int col, int q, int N) {
  if (s.f != nullptr) return s.f[(size_t)col * N + q];
  const double2 f = s.scale[col];
  const unsigned long long* p;
  size_t stride;
  if (s.dm != nullptr) {
    stride = s.dm_nk;
    p = s.dm + 4 * ((size_t)q * s.dm_nb + col % s.dm_nb) * stride + col / s.dm_nb;
  } else {
    stride = N;
    p = s.acc + (size_t)col * 4 * N + q;
  }
  const i64 hx = (i64)p[0], lx = (i64)p[stride], hy = (i64)p[2 * stride], ly = (i64)p[3 * stride];
  double x, y;
  // one conversion where the sums fit 64 bits (they can only outgrow them when
  // very many equal localised orbitals add up)
  if (((hx + (1ll << 29)) >> 30) == 0 && ((hy + (1ll << 29)) >> 30) == 0) {
    x = (double)((hx << 32) + lx);
    y = (double)((hy << 32) + ly);
  } else {
    x = fma((double)hx, 4294967296.0, (double)lx);
    y = fma((double)hy, 4294967296.0, (double)ly);
  }
  x = fma(x, f.x, x * f.y);
  y = fma(y, f.x, y * f.y);
  if (__double2hiint(f.x) < 0) {  // fx_output_scale: 2^kTiny too large
    x = fx_times_pow2(-x, -kTiny);
    y = fx_times_pow2(-y, -kTiny);
  }
  if (s.pexp != nullptr) {
    const int e = -s.pexp[q];
    x = fx_times_pow2(x, e);
    y = fx_times_pow2(y, e);
  }
  return make_double2(x, y);
}
// Sum over a CTA, result in every thread of warp 0 (fixed order).
template <int NW>
__device__ __forceinline__ double block_sum(double v, double* red) {
  v = warp_sum(v);
  if constexpr (NW == 1) return v;
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = red[0];
#pragma unroll
  for (int w = 1; w < NW; ++w) v += red[w];
  __syncthreads();
  return v;
}

}  // namespace mattohf
