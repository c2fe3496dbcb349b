// Fock exchange (src/Functions.f90:237-261) through the density matrix, for many
// orbitals per grid point.
//
// The sum over source orbitals is taken first.  With D_k(x, x') = sum_j u_kj(x)
// conj(u_kj(x')) over the occupied bands and v_d(r) = sum_G kern_d(G) e^{i G r},
//     (VF w)_k(x) = sum_x' W_k(x, x') w_k(x'),
//     W_k(x, x') = sum_k' D_k'(x, x') v_{k-k'}(x - x'):
// for each pair of grid points a convolution over the k-points, done by transforms
// of length L >= 2 NK over zero-padded k (linear, since the kernel's self-aliased
// frequency makes it not quite periodic in k).  D and W are Hermitian in (x, x'), so
// half of the pairs are formed.  All in 64-bit fixed point (fft_fx.cuh).
//
// Work, in 32 x 32 + 64-bit multiply-adds: N^2/2 NK (12 NBocc + 114) for W and
// N^2 NK 12 nbw for the product, against (NK NBocc)^2/2 87 N (w = u) or
// NK^2 NBocc nbw 75 N of the pair kernels (k_fock_fx.cu), whose work grows with
// the square of the bands.  Where the line lies: see fock_dm_wins.
//
// Scales.  u^ = u s with s^2 n(x) <= 2^119.4 for n(x) = sum |u_kj(x)|^2, so
// sum_k |D^_k| <= 2^59.4; the kernel's transform
// is scaled so that its absolute sum over t is below 2^60 for every r, so |W^| <=
// 2^59.4; w^ = w s_w with components up to 2^57.4 (moduli to 2^57.9), so the kDmTerms = 32
// products / 2^60 of a sum stay below 2^62.3 and are then added to two words in global memory.
#include "fx_convert.cuh"
#include "internal.h"

namespace mattohf {

constexpr float kDmPeak = 1.9e17f;  // 2^57.4

// ---------------------------------------------------------------------------
// Kernel tables, once per context: v_d(r) by a transform over G of each kern_d,
// then over d of each r.
// ---------------------------------------------------------------------------
template <int N>
__global__ void __launch_bounds__(fx::Team<N>::T < 32 ? 32 : fx::Team<N>::T) k_dm_vdr(const int2* __restrict__ kern,
                                                                                   const lc* __restrict__ tw,
                                                                                   cx* __restrict__ v) {
  using TM = fx::Team<N>;
  __shared__ lc tw_s[TM::kTwCount];
  __shared__ int2 twn_s[TM::kTwCount];
  __shared__ cx buf[N];
  for (int i = threadIdx.x; i < TM::kTwCount; i += blockDim.x) {
    const lc w = tw[i];
    tw_s[i] = w;
    twn_s[i] = make_int2(fx::neg_hi(w.yh), fx::neg_lo(w.yl));
  }
  __syncthreads();
  const int tl = threadIdx.x;
  if (tl >= TM::T) return;
  cx x[TM::E];
#pragma unroll
  for (int e = 0; e < TM::E; ++e) {
    const int2 k = kern[(size_t)blockIdx.x * N + TM::pos(tl, e)];
    x[e] = cx{((i64)k.x << fx::kLimb) + k.y, 0};
  }
  fx::forward<N, true>(x, buf, tw_s, twn_s, tl, 0);
#pragma unroll
  for (int e = 0; e < TM::E; ++e) v[(size_t)blockIdx.x * N + TM::pos(tl, e)] = cx{x[e].x, -x[e].y};  // backward
}

// raw[r][t] = sum_d v_d(r) exp(-2 pi i d t / L) / 2^shift, with the sum taken in 128
// bits (a transform of the shifted values would round at 2^shift times this place;
// the products, up to 2^120, lose ten bits so that the sum of all fits)
__global__ void k_dm_table(const cx* __restrict__ v, int N, int NK, int L, int shift, const cx* __restrict__ roots,
                           cx* __restrict__ raw) {
  constexpr int kDrop = 10;
  const int t = threadIdx.x, r = blockIdx.x;
  for (int q = t; q < L; q += blockDim.x) {
    __int128 sx = 0, sy = 0;
    for (int d = -NK + 1; d < NK; ++d) {
      const cx z = v[(size_t)(d + NK - 1) * N + r], w = roots[(((long long)d * q) % L + L) % L];
      sx += ((__int128)z.x * w.x - (__int128)z.y * w.y) >> kDrop;
      sy += ((__int128)z.x * w.y + (__int128)z.y * w.x) >> kDrop;
    }
    const int s = fx::kOne + shift - kDrop;
    const __int128 h = (__int128)1 << (s - 1);
    raw[(size_t)r * L + q] = cx{(i64)((sx + h) >> s), (i64)((sy + h) >> s)};
  }
}

// largest sum over t of |raw| / 2^20
__global__ void __launch_bounds__(32) k_dm_maxsum(const cx* __restrict__ raw, int L, int* maxsum) {
  float s = 0.0f;
  for (int t = threadIdx.x; t < L; t += 32) {
    const cx z = raw[(size_t)blockIdx.x * L + t];
    const float a = (float)(z.x >> 20), b = (float)(z.y >> 20);
    s += sqrtf(a * a + b * b);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (threadIdx.x == 0) atomicMax(maxsum, __float_as_int(s));  // positive floats order like integers
}

// out = raw c 2^k in limbs with sum_t |out| <= 2^60 for every r.  *scale: (c, k - shift
// + log2 L), what W^ carries beyond the scales of u^ and of the kernel table (the
// transforms over k are not normalised).
__global__ void k_dm_scale(const cx* __restrict__ raw, int n, int shift, int log2L, const int* __restrict__ maxsum,
                           lc* __restrict__ out, int2* scale) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const float m = __int_as_float(*maxsum);  // sum of |raw| / 2^20
  const Scale s = m > 0.0f ? fx_short_scale(1.09e12f / m, 0) : Scale{8, -3};  // 2^40 (1 - 9e-3): 2^60 / 2^20
  if (i == 0) *scale = make_int2(s.c, s.k - shift + log2L);
  if (i >= n) return;
  // raw c 2^k, k <= 0 as a rule: in 128 bits
  const cx z = raw[i];
  auto mul = [&](i64 a) -> i64 {
    const __int128 p = (__int128)a * s.c;
    return s.k >= 0 ? (i64)(p << s.k) : (i64)((p + ((__int128)1 << (-s.k - 1))) >> -s.k);
  };
  out[i] = fx::limbs(cx{mul(z.x), mul(z.y)});
}

// ---------------------------------------------------------------------------
// Largest density n(x) = sum |u_kj(x)|^2 over the grid, in FP32 and in units of the
// largest component's exponent, to *a.nmax (as bits; zeroed by k_dm_build).  The
// sum of the columns' largest squares would do for a bound, but is 8 to 10 times
// larger for smooth orbitals, and W would lose as many places (bound 1.3e-16 off at
// 128 / 16 / 8, this 0.8e-16).  A CTA takes eight points, 4.6 us at 256 / 64 / 4 and
// 9.3 at 512 / 128 / 8 (with 32 points, too few CTAs to cover the loads: 13.5 and 40).
// ---------------------------------------------------------------------------
__device__ __forceinline__ int dm_largest(const int2* __restrict__ sizes, int M, int* red) {
  int m = 0;
  for (int c = threadIdx.x; c < M; c += blockDim.x) m = max(m, sizes[c].x);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  for (int w = 0; w < (int)blockDim.x / 32; ++w) m = max(m, red[w]);
  return m;
}

__global__ void __launch_bounds__(512) k_dm_density(FockDmArgs a, int N) {
  __shared__ int red[16];
  __shared__ float part[16][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, x = blockIdx.x * 8 + (lane & 7);
  const int M = a.nk * a.nbocc, e = dm_largest(a.sizes, M, red) >> 20;
  float s = 0.0f;
#pragma unroll 4
  for (int c = threadIdx.x >> 3; c < M; c += 64) {
    const double2 z = a.u.p[(size_t)(c / a.nbocc) * a.u.kstride + (size_t)(c % a.nbocc) * N + x];
    const float p = fx_mantissa(__double2hiint(z.x) & 0x7fffffff, e), q = fx_mantissa(__double2hiint(z.y) & 0x7fffffff, e);
    s = fmaf(p, p, fmaf(q, q, s));
  }
  s += __shfl_xor_sync(0xffffffffu, s, 8);
  s += __shfl_xor_sync(0xffffffffu, s, 16);
  if (lane < 8) part[warp][lane] = s;
  __syncthreads();
  if (warp > 0) return;
  s = 0.0f;
  if (lane < 8)
    for (int w = 0; w < 16; ++w) s += part[w][lane];
  const int m = __reduce_max_sync(0xffffffffu, __float_as_int(s));  // floats of one sign order like integers
  if (lane == 0) atomicMax(a.nmax, m);
}

// ---------------------------------------------------------------------------
// Orbitals and functions w to fixed point, k fastest: ut[x][j][k] (k < L/2, the
// columns past NK stay zero), wt[x][i][k].  A CTA takes eight k-points of one band,
// so that it writes 128 bytes in a row; 64 grid points, since with all points of a
// band to a CTA the 64 CTAs of 256 / 64 / 4 waited for memory (14 us, now 8).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_dm_convert(FockDmArgs a, int N, int nbu) {
  __shared__ int red[4];
  __shared__ Scale sw[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int M = a.nk * a.nbocc, k0 = blockIdx.x * 8;
  const bool row = (int)blockIdx.y >= nbu;
  const int b = row ? blockIdx.y - nbu : blockIdx.y;
  const Block& src = row ? a.w : a.u;
  const bool same = a.w.p == a.u.p && a.w.kstride == a.u.kstride && nbu > 0;  // sizes are those of w's first bands
  const int m = dm_largest(a.sizes, M, red);
  // n(x) s^2 <= 2^119.4: the sums over a band's pairs keep a bit for their middle words
  const int2 us = nbu == 0 ? *a.uscale : make_int2(0, 0);  // no orbitals to convert: W's scale
  const Scale su = nbu == 0 ? Scale{us.x, us.y} : fx_scale(fx_size(m, __int_as_float(*a.nmax) * 1.0002f), 1e30f, 2.0f);
  if (row) {
    for (int j = warp; j < 8 && k0 + j < a.nk; j += 4) {
      const double2* p = src.p + (size_t)(k0 + j) * src.kstride + (size_t)b * N;
      const int2 z = same && b < a.nbocc ? a.sizes[(k0 + j) * a.nbocc + b] : fx_column_size(p, N, lane);
      if (lane == 0) sw[j] = fx_scale(z, kDmPeak, 1e-6f);
    }
    __syncthreads();
  }
  const int j = tid & 7, k = k0 + j;
  if (k < a.nk) {
    const Scale s = row ? sw[j] : su;
    const bool ok = s.c != 0;
    const double2* p = src.p + (size_t)k * src.kstride + (size_t)b * N;
    lc* o = row ? a.wt + (size_t)b * a.nk + k : a.ut + (size_t)b * a.lh + k;
    const size_t stride = row ? (size_t)a.w.nb * a.nk : (size_t)a.nbocc * a.lh;
#pragma unroll 4
    for (int x = blockIdx.z * 64 + (tid >> 3); x < min(N, ((int)blockIdx.z + 1) * 64); x += 16) {
      const double2 z = p[x];
      o[x * stride] = ok ? fx::limbs(cx{fx_convert(z.x, s), fx_convert(z.y, s)}) : lc{0, 0, 0, 0};
    }
  }
  // this CTA's share of the sums to zero
  const size_t nacc = (size_t)N * a.w.nb * 4 * a.nk, ncta = (size_t)gridDim.x * gridDim.y * gridDim.z;
  const size_t per = (nacc + ncta - 1) / ncta, z0 = per * (((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x);
  for (size_t i = z0 + tid; i < z0 + per && i < nacc; i += 128) a.acc[i] = 0;
  if (blockIdx.z > 0) return;
  if (!row) {
    if (tid == 0 && b == 0 && k0 == 0) *a.uscale = make_int2(su.c, su.k);
    return;
  }
  if (tid >= 8 || k >= a.nk) return;
  // F = F^ 2^180 / (su^2 s_w s_k s_t): u^ twice, w^, the kernel table's scale and its transform's
  const double2 f = fx_output_scale(su, sw[j], Scale{a.kscale->x, a.kscale->y});  // 2^180 / (su^2 s s_k)
  const double ct = (double)a.tscale->x;
  double r = (double)(1.0f / (float)a.tscale->x);
  r = fma(fma(-r, ct, 1.0), r, r);
  r = fma(fma(-r, ct, 1.0), r, r);
  const double rl = fma(-r, ct, 1.0) * r;
  const double q = pow2(-a.tscale->y);
  a.wscale[(size_t)k * a.w.nb + b] = make_double2(f.x * r * q, (fma(f.x, r, -(f.x * r)) + fma(f.x, rl, f.y * r)) * q);
}

// ---------------------------------------------------------------------------
// W for pairs x <= x': team w of a CTA has row x = R tile + w and visits the
// columns x' of the CTA's chunk together with the other teams, which so read the
// same orbital values.  W[x][x' - x] (k fastest) in limbs.
//
// Bound by the multiply-adds of the two transforms and of D (37 us of them at 256 /
// 64 / 4, 380 at 512 / 128 / 8; 78 and 698 us taken) and by the barriers between the
// passes of a team of 16 or 32 lanes.
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ size_t dm_row(int x, int N) { return (size_t)x * N - (size_t)x * (x - 1) / 2 - x; }

template <int L>
__global__ void __launch_bounds__(kDmThreads, 2) k_dm_build(FockDmArgs a, int N, int chunk) {
  using TM = fx::Team<L>;
  constexpr int E = TM::E, T = TM::T, R0 = TM::R0, R = kDmThreads / T;
  extern __shared__ int4 sm_dm[];
  lc* tw_s = reinterpret_cast<lc*>(sm_dm);                 // kTwCount
  cx* bufs = reinterpret_cast<cx*>(sm_dm + TM::kTwCount);  // R * L
  int2* twn_s = reinterpret_cast<int2*>(bufs + R * L);     // kTwCount
  const int tl = threadIdx.x % T, team = threadIdx.x / T;
  const int x0 = blockIdx.x * R, x = x0 + team;
  const int xb = max(x0, (int)blockIdx.y * chunk), xe = min(N, ((int)blockIdx.y + 1) * chunk);
  if (xb >= xe) return;
  for (int i = threadIdx.x; i < TM::kTwCount; i += kDmThreads) {
    const lc w = a.twL[i];
    tw_s[i] = w;
    twn_s[i] = make_int2(fx::neg_hi(w.yh), fx::neg_lo(w.yl));
  }
  __syncthreads();
  cx* buf = bufs + team * L;
  const lc* ux = a.ut + (size_t)min(x, N - 1) * a.nbocc * a.lh;
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *a.nmax = 0;  // for the next apply
  for (int xp = xb; xp < xe; ++xp) {
    const lc* up = a.ut + (size_t)xp * a.nbocc * a.lh;
    cx z[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      z[e] = cx{0, 0};
      if (e % R0 < R0 / 2) {  // k < L / 2
        const int k = TM::pos(tl, e);
        for (int j0 = 0; j0 < a.nbocc; j0 += 8) {
          // u(x) conj(u(x')) over up to eight bands, rounded once: half a place and the
          // mean of the dropped low products (real part: two of 1/4 per band)
          const int j1 = min(a.nbocc, j0 + 8);
          i64 hr = 0, hi = 0, mr = (i64)(j1 - j0 + 1) << (fx::kLimb - 1), mi = 1ll << (fx::kLimb - 1);
          for (int j = j0; j < j1; ++j) {
            const lc p = ux[j * a.lh + k], q = up[j * a.lh + k];
            const int nyh = -q.yh, nyl = -q.yl;
            hr = fx::mw(p.xh, q.xh, fx::mw(p.yh, q.yh, hr));
            mr = fx::mw(p.xh, q.xl, fx::mw(p.xl, q.xh, fx::mw(p.yh, q.yl, fx::mw(p.yl, q.yh, mr))));
            hi = fx::mw(p.yh, q.xh, fx::mw(p.xh, nyh, hi));
            mi = fx::mw(p.yh, q.xl, fx::mw(p.yl, q.xh, fx::mw(p.xh, nyl, fx::mw(p.xl, nyh, mi))));
          }
          z[e] = fx::add(z[e], cx{hr + (mr >> fx::kLimb), hi + (mi >> fx::kLimb)});
        }
      }
    }
    const lc* vt = a.table + (size_t)((x - xp + N) % N) * L;
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      fx::forward<L>(z, buf, tw_s, twn_s, tl, team);
      if (h == 0) {
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const cx y = fx::cmul(fx::limbs(z[e]), vt[TM::pos(tl, e)]);
          z[e] = cx{y.x, -y.y};
        }
      }
    }
    if (x <= xp && x < N) {
      lc* o = a.W + (dm_row(x, N) + xp) * a.nk;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int k = TM::pos(tl, e);
        if (e % R0 < R0 / 2 && k < a.nk) o[k] = fx::limbs(cx{z[e].x, -z[e].y});
      }
    }
  }
}

// ---------------------------------------------------------------------------
// F(x) = sum_x' W(x, x') w(x'): a thread has one k, R rows x and BW bands, a CTA one
// chunk of x'.  Sums go to 64-bit atomics after kDmTerms terms.
//
// Bound by the 32 x 32 + 64-bit multiply-adds (12 a term; 22 us of them at 256 / 64 /
// 4, 44 us taken) and by what loads and few warps leave open: a row of W is read once
// for BW bands, a value of w once for R rows.  256 / 64 / 4 and 512 / 128 / 8, us:
// BW x R = 4 x 2 at 128 registers 44 / 596, at 102 (spills) 54 / 646, 4 x 1 46 / 647,
// 2 x 2 48 / 678, 2 x 4 46 / 634, 1 x 4 54 / 777; 8 x 2 1148 at the second.
// ---------------------------------------------------------------------------
template <int BW, int R, int MINB>
__global__ void __launch_bounds__(128, MINB) k_dm_apply(FockDmArgs a, int N, int chunk) {
  const int nbg = (a.w.nb + BW - 1) / BW, t = (blockIdx.x / nbg) * 128 + threadIdx.x;
  const int k = t % a.nk, x0 = t / a.nk * R;
  const int b0 = (blockIdx.x % nbg) * BW, nb = min(BW, a.w.nb - b0);
  if (x0 >= N) return;
  const int xe = min(N, ((int)blockIdx.y + 1) * chunk);
#pragma unroll 1
  for (int xb = blockIdx.y * chunk; xb < xe; xb += kDmTerms) {
    cx acc[R][BW];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int b = 0; b < BW; ++b) acc[r][b] = cx{0, 0};
    const int xq = min(xe, xb + kDmTerms);
#pragma unroll 1
    for (int xp = xb; xp < xq; ++xp) {
      lc w[BW], W[R];
      int2 nW[R];
      const lc* wp = a.wt + ((size_t)xp * a.w.nb + b0) * a.nk + k;
#pragma unroll
      for (int b = 0; b < BW; ++b) w[b] = b < nb ? wp[(size_t)b * a.nk] : lc{0, 0, 0, 0};
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int x = x0 + r, lo = min(x, xp);
        const lc v = a.W[(dm_row(lo, N) + (x + xp - lo)) * a.nk + k];
        const int nyh = fx::neg_hi(v.yh), nyl = fx::neg_lo(v.yl);
        const bool up = x <= xp;  // below the diagonal: conjugate
        W[r] = lc{v.xh, v.xl, up ? v.yh : nyh, up ? v.yl : nyl};
        nW[r] = up ? make_int2(nyh, nyl) : make_int2(v.yh, v.yl);
      }
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int b = 0; b < BW; ++b) acc[r][b] = fx::add(acc[r][b], fx::cmul(w[b], W[r], nW[r]));
    }
    // words [x high, x low, y high, y low][k]
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int b = 0; b < BW; ++b) {
        if (b >= nb) continue;
        unsigned long long* o = a.acc + 4 * ((size_t)(x0 + r) * a.w.nb + b0 + b) * a.nk + k;
        atomicAdd(o, (unsigned long long)(acc[r][b].x >> 32));
        atomicAdd(o + a.nk, (unsigned long long)(unsigned)acc[r][b].x);
        atomicAdd(o + 2 * a.nk, (unsigned long long)(acc[r][b].y >> 32));
        atomicAdd(o + 3 * a.nk, (unsigned long long)(unsigned)acc[r][b].y);
      }
  }
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
int dm_length(int NK) {
  int L = 16;
  while (L < 2 * NK) L *= 2;
  return L;
}

template <int N>
static cudaError_t dm_vdr_impl(const int2* kern, const lc* tw, cx* v, int nd, cudaStream_t s) {
  k_dm_vdr<N><<<nd, fx::Team<N>::T < 32 ? 32 : fx::Team<N>::T, 0, s>>>(kern, tw, v);
  return cudaGetLastError();
}
#define MATTOHF_DISPATCH(NG, CALL)                 \
  switch (NG) {                                    \
    case 16: return CALL(16);                      \
    case 32: return CALL(32);                      \
    case 64: return CALL(64);                      \
    case 128: return CALL(128);                    \
    case 256: return CALL(256);                    \
    case 512: return CALL(512);                    \
    default: return cudaErrorInvalidValue;         \
  }

static cudaError_t dm_vdr(int N, const int2* kern, const lc* tw, cx* v, int nd, cudaStream_t s) {
#define CALL(n) dm_vdr_impl<n>(kern, tw, v, nd, s)
  MATTOHF_DISPATCH(N, CALL)
#undef CALL
}
cudaError_t launch_dm_table(int N, int NK, const int2* kern, const fx::lc* twN, const fx::cx* roots, fx::cx* v, fx::cx* raw,
                            int* maxsum, fx::lc* table, int2* scale, cudaStream_t s) {
  const int L = dm_length(NK);
  int log2L = 4;
  while ((1 << log2L) < L) ++log2L;
  int shift = 1;
  while ((1 << shift) < 2 * NK) ++shift;  // |v_d| <= 2^60, 2 NK - 1 of them
  cudaError_t e = cudaMemsetAsync(maxsum, 0, sizeof(int), s);
  if (e == cudaSuccess) e = dm_vdr(N, kern, twN, v, 2 * NK - 1, s);
  if (e != cudaSuccess) return e;
  k_dm_table<<<N, L < 256 ? L : 256, 0, s>>>(v, N, NK, L, shift, roots, raw);
  k_dm_maxsum<<<N, 32, 0, s>>>(raw, L, maxsum);
  k_dm_scale<<<(N * L + 255) / 256, 256, 0, s>>>(raw, N * L, shift, log2L, maxsum, table, scale);
  return cudaGetLastError();
}

cudaError_t launch_dm_convert(int NG, const FockDmArgs& a, bool have_orbitals, cudaStream_t s) {
  if (!have_orbitals) k_dm_density<<<NG / 8, 512, 0, s>>>(a, NG);
  const int nbu = have_orbitals ? 0 : a.nbocc;
  k_dm_convert<<<dim3((a.nk + 7) / 8, nbu + a.w.nb, (NG + 63) / 64), 128, 0, s>>>(a, NG, nbu);
  return cudaGetLastError();
}

template <int L>
static constexpr size_t dm_smem() { return 24 * (size_t)fx::Team<L>::kTwCount + 16 * (size_t)L * (kDmThreads / fx::Team<L>::T); }

template <int L>
static cudaError_t dm_build_impl(int N, const FockDmArgs& a, int nsm, cudaStream_t s) {
  constexpr int R = kDmThreads / fx::Team<L>::T;
  const int tiles = (N + R - 1) / R;
  // chunks of x' so that the half triangle has about 16 CTAs per SM
  int nch = (32 * nsm + tiles - 1) / tiles;
  nch = nch < 1 ? 1 : nch > N / 4 ? (N / 4 > 0 ? N / 4 : 1) : nch;
  const int chunk = (N + nch - 1) / nch;
  k_dm_build<L><<<dim3(tiles, (N + chunk - 1) / chunk), kDmThreads, dm_smem<L>(), s>>>(a, N, chunk);
  return cudaGetLastError();
}

cudaError_t launch_dm_build(int NG, const FockDmArgs& a, int nsm, cudaStream_t s) {
#define CALL(n) dm_build_impl<n>(NG, a, nsm, s)
  MATTOHF_DISPATCH(2 * a.lh, CALL)
#undef CALL
}

template <int BW, int R, int MINB>
static cudaError_t dm_apply_impl(int NG, const FockDmArgs& a, int nsm, cudaStream_t s) {
  const int gx = (NG / R * a.nk + 127) / 128 * ((a.w.nb + BW - 1) / BW);
  // about 16 CTAs per SM, in chunks of 16 terms or more
  int nch = (16 * nsm + gx - 1) / gx;
  const int most = NG / (kDmTerms / 2);
  nch = nch < 1 ? 1 : nch > most ? most : nch;
  const int chunk = (NG + nch - 1) / nch;
  k_dm_apply<BW, R, MINB><<<dim3(gx, (NG + chunk - 1) / chunk), 128, 0, s>>>(a, NG, chunk);
  return cudaGetLastError();
}
cudaError_t launch_dm_apply(int NG, const FockDmArgs& a, int nsm, cudaStream_t s) {
  const int nb = a.w.nb;
  if (nb == 1) return dm_apply_impl<1, 4, 6>(NG, a, nsm, s);
  if (nb == 2) return dm_apply_impl<2, 4, 4>(NG, a, nsm, s);
  // groups of four bands, or of three where that leaves fewer places empty
  if ((nb + 2) / 3 * 3 < (nb + 3) / 4 * 4) return dm_apply_impl<3, 2, 4>(NG, a, nsm, s);
  return dm_apply_impl<4, 2, 4>(NG, a, nsm, s);
}

template <int L>
static cudaError_t dm_configure() {
  return cudaFuncSetAttribute(k_dm_build<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dm_smem<L>());
}
cudaError_t configure_dm_kernels() {
  cudaError_t e;
  if ((e = dm_configure<16>()) != cudaSuccess) return e;
  if ((e = dm_configure<32>()) != cudaSuccess) return e;
  if ((e = dm_configure<64>()) != cudaSuccess) return e;
  if ((e = dm_configure<128>()) != cudaSuccess) return e;
  if ((e = dm_configure<256>()) != cudaSuccess) return e;
  return dm_configure<512>();
}

}  // namespace mattohf
