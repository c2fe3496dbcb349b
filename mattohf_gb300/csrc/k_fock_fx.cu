// Fock exchange (src/Functions.f90:237-261) with 64-bit fixed-point pair
// transforms (fft_fx.cuh).
//
// Scales.  Orbitals are converted once per apply to u^ = u s 2^d with one
// scale s for all of them (k_fx_sizes, k_fx_convert): a short factor times a
// power of two, so that u^ keeps every bit of the components from 2^-6 of the
// largest on and 2^-59 of the largest at the others, with
//     |u^|_2 <= 2^60.2      (a pair density's absolute sum stays below 2^60.4, and
//                            so does |phi^|, the kernel's being at most 2^60)
//     each component of u^ <= 2^58.4, its modulus <= 2^58.9.
// A term phi^ u^ / 2^60 is at most 2^59.3, all of which may fall on one component of the
// sum: kFxTerms = 12 of them stay below 2^62.9 and the 8 of a tile below 2^62.3 (16, as
// counted with 2^58.4 and |phi^| <= 2^60, reached 1.19 times 2^63 with equal functions
// that are flat on a few points).
// d = 0 except for an orbital whose norm is half the largest one or less: d then
// brings it to the upper half, and a term that it enters twice is shifted back by 2 d
// (its components may pass 2^58.4, as a modulus up to 2^60.2; 2 d >= 2 makes up for it).
// The kernel table is K^ = kern s_k with sum_G |K^(G)| <= 2^60 for every k - k'.
// A pair's chain is then
//     p^ = u_a^ conj(u_b^) / 2^60,  phi^ = IFFT(K^ FFT(p^) / 2^60),
//     F_a^ += phi^ u_b^ / 2^60,     F = F^ 2^180 / (s^3 s_k 2^d_a),
// every sum exact in integers, so the order of summation does not matter.
// Orbitals that are not finite give NaN.
//
// What bounds it and what it measured.  k_fock_sym_fx at NG = 256, NK = 64,
// Nocc = 4 (32896 pairs): 165 us, against 918 us of the same pairs in FP64 (89 % FP64
// pipe).  It issues about 390 instructions per point and pair, 87 of them
// 32 x 32 + 64-bit multiply-adds at half the rate of the others; at NK = 32 (51 us, tiles
// of 2) the heavy FMA pipe that has these is 55 % busy, the ALU 44 %, the issue slots
// 48 %.  Two CTAs of 128 threads a SM at least (a register limit for four of them spills:
// 183 us).
// Error of one apply against long double, same table, smooth orthonormal
// orbitals, here / FP64: NG = 64 0.7e-16 / 1.2e-16, NG = 256 1.0e-16 / 1.8e-16,
// NG = 512 1.3e-16 / 1.9e-16.
//
// Sums over tiles and chunks go to 64-bit atomics in global memory (29 us by
// themselves at that size, mostly beside the pair loop) instead of 68 MB of
// partials and a reduction launch (13 + 24 us).
#include <algorithm>

#include "fx_convert.cuh"
#include "internal.h"

namespace mattohf {

__device__ __forceinline__ const double2* fx_column(const Block& u, int nb, int col, int N) {
  return u.p + (size_t)(col / nb) * u.kstride + (size_t)(col % nb) * N;
}

// One column to fixed point, by a CTA of 128 threads: column i < M of the orbitals
// (one scale for all), or column i - M of the rows (a scale of its own).  The
// orbitals' sizes are in a.sizes, or (scan: few orbitals) taken here.
__device__ __forceinline__ void fx_convert_body(const FockFxArgs& a, const FockFxRows& r, int N, int i, bool scan) {
  constexpr int PER = 4;  // N <= 512
  __shared__ int2 red[4], own_s;
  __shared__ int redr[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int M = a.nk * a.nbocc;
  const bool row = i >= M;
  const int col = row ? i - M : i;
  const double2* p = row ? fx_column(r.w, r.w.nb, col, N) : fx_column(a.u, a.nbocc, col, N);
  double2 v[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) v[j] = tid + 128 * j < N ? p[tid + 128 * j] : make_double2(0.0, 0.0);
  int2 g = make_int2(0, 0), own = make_int2(0, 0);
  if (scan) {
    for (int c = warp; c < M; c += 4) {
      const int2 z = fx_column_size(fx_column(a.u, a.nbocc, c, N), N, lane);
      g = fx_larger(g, z);
      if (c == i && lane == 0) {
        own_s = z;
        a.sizes[c] = z;
      }
    }
  } else {
    for (int c = tid; c < M; c += 128) g = fx_larger(g, a.sizes[c]);
    g = make_int2(__reduce_max_sync(0xffffffffu, g.x), __reduce_max_sync(0xffffffffu, g.y));
    if (!row && tid == 0) own_s = a.sizes[col];
  }
  if (lane == 0) red[warp] = g;
  if (row) own = fx_block_size<PER, 4>(v, redr);  // has barriers
  else __syncthreads();
  g = fx_larger(fx_larger(red[0], red[1]), fx_larger(red[2], red[3]));
  if (!row) own = own_s;
  // with a scale per point the sums' terms are uprod's, and u^ is bounded by its norm alone
  Scale s = fx_scale(g, a.pexp != nullptr ? 1e30f : kPeak, 1.0f);
  s.k -= a.halve;
  Scale sd = s;
  int d = 0;
  if (row) {
    sd = fx_scale(own, 1e30f, 1.0f);
  } else if (a.lift && own.y > 0) {
    // a column with half the largest norm or less is lifted by 2^d to the upper half: the
    // largest d with own^2 4^d up to the largest square (keys order like these)
    d = min(1000, (g.y - own.y) >> 19);
    sd.k += d;
  }
  const bool ok = sd.c != 0;
  lc* o = (row ? r.wfx : a.ufx) + (size_t)col * N;
#pragma unroll
  for (int j = 0; j < PER; ++j)
    if (tid + 128 * j < N) o[tid + 128 * j] = ok ? fx::limbs(cx{fx_convert(v[j].x, sd), fx_convert(v[j].y, sd)}) : lc{0, 0, 0, 0};
  unsigned long long* acc = row ? r.acc : a.acc;
  if (acc != nullptr)
    for (int j = tid; j < 4 * N; j += 128) acc[(size_t)col * 4 * N + j] = 0;
  if (tid != 0) return;
  const Scale sk{a.kscale->x, a.kscale->y};
  if (row) {
    r.wscale[col] = fx_output_scale(s, sd, sk);
    return;
  }
  if (a.shift) a.shift[col] = d;
  if (col == 0) *a.uscale = make_int2(s.c, s.k);
  if (a.fscale) {
    // a column of zeros has a sum of zero; the roundings of its terms do not count
    a.fscale[col] = own.y > 0 || s.c == 0 ? fx_output_scale(s, sd, sk) : make_double2(0.0, 0.0);
  }
}

__global__ void __launch_bounds__(128) k_fx_sizes(FockFxArgs a, int N) {
  const int col = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (col >= a.nk * a.nbocc) return;
  const int2 z = fx_column_size(fx_column(a.u, a.nbocc, col, N), N, threadIdx.x & 31);
  if ((threadIdx.x & 31) == 0) a.sizes[col] = z;
}
__global__ void __launch_bounds__(128) k_fx_convert(FockFxArgs a, FockFxRows r, int N, int first, int scan) {
  fx_convert_body(a, r, N, first + blockIdx.x, scan);
}
// two sets at once (blockIdx.y): the adjoint's v and mu
__global__ void __launch_bounds__(128) k_fx_sizes2(FockFxArgs a, FockFxArgs b, int N) {
  const FockFxArgs& c = blockIdx.y ? b : a;
  const int col = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (col >= c.nk * c.nbocc) return;
  const int2 z = fx_column_size(fx_column(c.u, c.nbocc, col, N), N, threadIdx.x & 31);
  if ((threadIdx.x & 31) == 0) c.sizes[col] = z;
}
__global__ void __launch_bounds__(128) k_fx_convert2(FockFxArgs a, FockFxArgs b, int N) {
  fx_convert_body(blockIdx.y ? b : a, FockFxRows{}, N, blockIdx.x, false);
}
// element prefix: pre[r] = sum over earlier runs of M_r * N
__global__ void __launch_bounds__(128) k_fx_sizes_batch(const FockFxArgs* __restrict__ args,
                                                        const int* __restrict__ pre, int nruns, int N) {
  const int c = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (c * N >= pre[nruns]) return;
  const int r = find_run(pre, nruns, c * N), col = c - pre[r] / N;
  const int2 z = fx_column_size(fx_column(args[r].u, args[r].nbocc, col, N), N, threadIdx.x & 31);
  if ((threadIdx.x & 31) == 0) args[r].sizes[col] = z;
}
__global__ void __launch_bounds__(128) k_fx_convert_batch(const FockFxArgs* __restrict__ args,
                                                          const int* __restrict__ pre, int nruns, int N) {
  const int r = find_run(pre, nruns, blockIdx.x * N);
  fx_convert_body(args[r], FockFxRows{}, N, blockIdx.x - pre[r] / N, false);
}

// The exchange by itself (mattohf_fock) is accurate at every grid point, as with FP64
// values, where h[u] w has the kinetic transform's error of one size everywhere.  A
// pair's density may have one scale, its transform mixing all points; but the product
// phi_ab(x) u_b(x) then loses what |u_b(x)| is below the peak (a Gaussian's value of 1e-8
// of it came out 5e-11 off).  So it takes the orbitals again, with a scale 2^pexp(x)
// that brings the largest of |u_b(x)| 2^-d_b over b (the size of its term: phi_ab^
// carries 2^d_b) to 2^57 or more.  A CTA takes eight points; it reads the orbitals twice.
__global__ void __launch_bounds__(512) k_fx_points(FockFxArgs a, int N) {
  __shared__ int part[16][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, x = blockIdx.x * 8 + (lane & 7);
  const int M = a.nk * a.nbocc;
  const Scale s{a.uscale->x, a.uscale->y};
  constexpr int kNone = -8192;
  int m = kNone;
  for (int c = threadIdx.x >> 3; c < M; c += 64) {
    const double2 z = fx_column(a.u, a.nbocc, c, N)[x];
    const int e = max((__double2hiint(z.x) & 0x7fffffff) >> 20, (__double2hiint(z.y) & 0x7fffffff) >> 20);
    if (z.x != 0.0 || z.y != 0.0) m = max(m, max(e, 1) - a.shift[c]);
  }
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 8));
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 16));
  if (lane < 8) part[warp][lane] = m;
  __syncthreads();
  for (int w = 0; w < 16; ++w) m = max(m, part[w][lane & 7]);
  // a component with exponent field e is below 2^(e - 1022), s below 2^(k + 4); where all
  // are zero (2^-2000 = 0), so is the sum of the products' roundings
  const int pe = s.c == 0 ? 0 : m == kNone ? 2000 : min(1000, 1076 - s.k - m);
  if (warp == 0 && lane < 8) a.pexp[x] = pe;
  for (int c = threadIdx.x >> 3; c < M; c += 64) {
    const double2 z = fx_column(a.u, a.nbocc, c, N)[x];
    const Scale sx{s.c, s.k + pe - a.shift[c]};
    a.uprod[(size_t)c * N + x] = s.c ? fx::limbs(cx{fx_convert(z.x, sx), fx_convert(z.y, sx)}) : lc{0, 0, 0, 0};
  }
}

// t / 2^s for s > 0, rounded (a floor would be biased by half a place per term)
__device__ __forceinline__ cx fx_shift(cx t, int s) {
  s = min(s, 62);
  const i64 r = 1ll << (s - 1);
  return cx{(t.x + r) >> s, (t.y + r) >> s};
}

// Adds a 64-bit partial sum to a column's accumulators, as its high and low words:
// planes [4][N] of x high, x low, y high, y low.  Exact, so in any order.
__device__ __forceinline__ void fx_accumulate(unsigned long long* acc, int N, int q, cx v) {
  atomicAdd(acc + q, (unsigned long long)(v.x >> 32));
  atomicAdd(acc + N + q, (unsigned long long)(unsigned)v.x);
  atomicAdd(acc + 2 * N + q, (unsigned long long)(v.y >> 32));
  atomicAdd(acc + 3 * N + q, (unsigned long long)(unsigned)v.y);
}

// x: pair density in, conj(its potential) out; returns the density's transform at
// the self-aliased frequency N/2.
template <int N>
__device__ __forceinline__ cx potential(cx (&x)[fx::Team<N>::E], const int2* __restrict__ kab, cx* buf,
                                        const lc* tw_s, const int2* twn_s, int tl, int team) {
  using TM = fx::Team<N>;
  constexpr int E = TM::E, T = TM::T;
  cx rn{0, 0};
  // forward transform, kernel product, backward transform of the conjugate
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    fx::forward<N>(x, buf, tw_s, twn_s, tl, team);
    if (h == 0) {
      rn = x[TM::kNyquistSlot];  // in the team's lane 0
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int2 k = __ldg(kab + TM::pos(tl, e));
        x[e] = cx{fx::rmul(x[e].x, k), -fx::rmul(x[e].y, k)};
      }
    }
  }
  if constexpr (T > 32) {  // the team's two warps share lane 0's value through the buffer
    fx::team_sync<T>(team);
    if (tl == 0) buf[0] = rn;
    fx::team_sync<T>(team);
    return buf[0];
  } else {
    const int lane0 = (threadIdx.x & 31) / T * T;
    return cx{__shfl_sync(0xffffffffu, rn.x, lane0), __shfl_sync(0xffffffffu, rn.y, lane0)};
  }
}
// the same for the density of the pair (a, b): x = conj(phi_ab)
template <int N>
__device__ __forceinline__ cx pair_potential(cx (&x)[fx::Team<N>::E], const lc* __restrict__ ua,
                                             const lc* __restrict__ ub, const int2* __restrict__ kab, cx* buf,
                                             const lc* tw_s, const int2* twn_s, int tl, int team) {
  using TM = fx::Team<N>;
#pragma unroll
  for (int e = 0; e < TM::E; ++e) {
    const int q = TM::pos(tl, e);
    x[e] = fx::cmulc(ua[q], ub[q]);
  }
  return potential<N>(x, kab, buf, tw_s, twn_s, tl, team);
}

// Twiddles to shared memory: tw_s, and the negated imaginary parts to twn_s.
template <int N>
__device__ __forceinline__ void load_twiddles(const lc* __restrict__ tw, lc* tw_s, int2* twn_s) {
  for (int i = threadIdx.x; i < fx::Team<N>::kTwCount; i += blockDim.x) {
    const lc w = tw[i];
    tw_s[i] = w;
    twn_s[i] = make_int2(fx::neg_hi(w.yh), fx::neg_lo(w.yl));
  }
}

// ---------------------------------------------------------------------------
// Symmetric exchange (w == u, occupied pairs).  A CTA has a tile pair (ti <= tj) of
// S orbitals each: team w owns row a = i S + w in registers and in round r visits
// column b = j S + (w + r) % S, whose accumulator in shared memory has one
// writer per round.
// ---------------------------------------------------------------------------
template <int N>
__device__ __forceinline__ void fock_sym_fx_body(const FockFxArgs& a, const int tile) {
  using TM = fx::Team<N>;
  constexpr int E = TM::E, T = TM::T;
  const int S = a.S;
  const int nteam = blockDim.x / T;
  extern __shared__ int4 sm_fx[];
  lc* tw_s = reinterpret_cast<lc*>(sm_fx);                 // kTwCount
  cx* bufs = reinterpret_cast<cx*>(sm_fx + TM::kTwCount);  // nteam * N
  cx* cacc = bufs + nteam * N;                             // S * N
  const int tid = threadIdx.x, tl = tid % T, tw_ = tid / T;
  cx* buf = bufs + tw_ * N;
  int2* twn_s = reinterpret_cast<int2*>(cacc + S * N);  // kTwCount
  load_twiddles<N>(a.tw, tw_s, twn_s);
  for (int i = tid; i < S * N; i += blockDim.x) cacc[i] = cx{0, 0};
  int ti = 0, rem = tile;
  while (rem >= a.T - ti) { rem -= a.T - ti; ++ti; }
  const int tj = ti + rem;
  const int M = a.nk * a.nbocc;
  const int ia = ti * S + tw_;
  const bool va = tw_ < S && ia < M;
  const int oa = va ? ia : 0;
  const int ka = oa / a.nbocc;
  const lc *ua = a.ufx + (size_t)oa * N, *uam = a.uprod + (size_t)oa * N;
  const bool points = a.pexp != nullptr;  // the orbitals' 2^d are in uprod
  const int sa = points ? 0 : 2 * a.shift[oa];
  cx racc[E];
#pragma unroll
  for (int e = 0; e < E; ++e) racc[e] = cx{0, 0};
  __syncthreads();
  const bool diag = (ti == tj);
  const int nrounds = diag ? (S / 2 + 1) : S;
  for (int r = 0; r < nrounds; ++r) {
    const int lb = (tw_ + r) % S;
    const int ib = tj * S + lb;
    bool valid = va && ib < M;
    if (diag && (S % 2 == 0) && r == S / 2 && tw_ >= S / 2) valid = false;  // counted by the partner
    const bool self = diag && r == 0;
    const int ob = ib < M ? ib : 0;
    const int kb = ob / a.nbocc;
    const lc *ub = a.ufx + (size_t)ob * N, *ubm = a.uprod + (size_t)ob * N;
    const int2* kab = a.kern + (size_t)(ka - kb + a.nk - 1) * N;
    cx x[E];
    const cx rn = pair_potential<N>(x, ua, ub, kab, buf, tw_s, twn_s, tl, tw_);
    if (valid) {
      const int sb = points ? 0 : 2 * a.shift[ob];
      // phi u_b = conj(x) u_b
      if (sb == 0) {
#pragma unroll
        for (int e = 0; e < E; ++e) racc[e] = fx::add(racc[e], fx::cmulc(ubm[TM::pos(tl, e)], fx::limbs(x[e])));
      } else {
#pragma unroll
        for (int e = 0; e < E; ++e)
          racc[e] = fx::add(racc[e], fx_shift(fx::cmulc(ubm[TM::pos(tl, e)], fx::limbs(x[e])), sb));
      }
      if (!self) {
        // phi_ba = conj(phi_ab + c (-1)^x), c = (K_ba - K_ab)(N/2) R_ab(N/2)
        const int2 kba = __ldg(a.kern + (size_t)(kb - ka + a.nk - 1) * N + N / 2), kn = __ldg(kab + N / 2);
        cx c{fx::rmul(rn.x, kba) - fx::rmul(rn.x, kn), fx::rmul(rn.y, kn) - fx::rmul(rn.y, kba)};
        if (tl & 1) c = cx{-c.x, -c.y};  // T and N/R0 are even: the sign is the lane's
        cx* col = cacc + lb * N;
        if (sa == 0) {
#pragma unroll
          for (int e = 0; e < E; ++e) {
            const int q = TM::pos(tl, e);
            col[q] = fx::add(col[q], fx::cmul(fx::limbs(fx::add(x[e], c)), uam[q]));
          }
        } else {
#pragma unroll
          for (int e = 0; e < E; ++e) {
            const int q = TM::pos(tl, e);
            col[q] = fx::add(col[q], fx_shift(fx::cmul(fx::limbs(fx::add(x[e], c)), uam[q]), sa));
          }
        }
      }
    }
    __syncthreads();
  }
  if (va) {
    unsigned long long* dst = a.acc + (size_t)ia * 4 * N;
#pragma unroll
    for (int e = 0; e < E; ++e) fx_accumulate(dst, N, TM::pos(tl, e), racc[e]);
  }
  for (int i = tid; i < S * N; i += blockDim.x) {
    const int ib = tj * S + i / N;
    if (ib < M) fx_accumulate(a.acc + (size_t)ib * 4 * N, N, i % N, cacc[i]);
  }
}

// threads of a CTA with the largest tile
template <int N>
constexpr int sym_fx_threads() {
  return kFxMaxTile * fx::Team<N>::T < 32 ? 32 : kFxMaxTile * fx::Team<N>::T > 256 ? 256 : kFxMaxTile * fx::Team<N>::T;
}

template <int N>
__global__ void __launch_bounds__(sym_fx_threads<N>(), 2) k_fock_sym_fx(FockFxArgs a) { fock_sym_fx_body<N>(a, blockIdx.x); }

template <int N>
__global__ void __launch_bounds__(sym_fx_threads<N>(), 2) k_fock_sym_fx_batch(const FockFxArgs* __restrict__ args,
                                                                           const int* __restrict__ pre, int nruns) {
  const int r = find_run(pre, nruns, blockIdx.x);
  fock_sym_fx_body<N>(args[r], blockIdx.x - pre[r]);
}

// ---------------------------------------------------------------------------
// Exchange on other functions w (Krylov blocks, empty bands, a rank's rows):
// F_w = sum over all occupied b of phi_wb u_b, no symmetry.  Each column of w
// has a scale of its own (|w^|_2 <= 2^60.2), since it enters every term once.
// A CTA takes kRowsThreads / T columns, one per team, against one chunk of the
// sources, which all its teams read together.
// ---------------------------------------------------------------------------
template <int N>
constexpr int rows_fx_teams() { return kRowsThreads / fx::Team<N>::T; }

template <int N>
__global__ void __launch_bounds__(kRowsThreads, 2) k_fock_fx(FockFxArgs a, FockFxRows r) {
  using TM = fx::Team<N>;
  constexpr int E = TM::E, T = TM::T, R = kRowsThreads / TM::T;
  extern __shared__ int4 sm_fx[];
  lc* tw_s = reinterpret_cast<lc*>(sm_fx);                      // kTwCount
  cx* bufs = reinterpret_cast<cx*>(sm_fx + TM::kTwCount);       // R * N
  int2* twn_s = reinterpret_cast<int2*>(bufs + R * N);          // kTwCount
  const int tl = threadIdx.x % T, team = threadIdx.x / T;
  cx* buf = bufs + team * N;
  load_twiddles<N>(a.tw, tw_s, twn_s);
  __syncthreads();
  const int col = (blockIdx.x / r.nchunks) * R + team, chunk = blockIdx.x % r.nchunks;
  const bool valid = col < r.ncols;
  const int c = valid ? col : 0;
  const int kr = c / r.w.nb;
  const lc* wa = r.wfx + (size_t)c * N;
  unsigned long long* dst = r.acc + (size_t)c * 4 * N;
  const int p0 = chunk * r.chunk, p1 = min(a.nk * a.nbocc, p0 + r.chunk);
  cx acc[E];
#pragma unroll
  for (int e = 0; e < E; ++e) acc[e] = cx{0, 0};
  for (int p = p0; p < p1; ++p) {
    if (p != p0 && (p - p0) % kFxTerms == 0) {  // before the accumulators could overflow
#pragma unroll
      for (int e = 0; e < E; ++e) {
        if (valid) fx_accumulate(dst, N, TM::pos(tl, e), acc[e]);
        acc[e] = cx{0, 0};
      }
    }
    const lc *ub = a.ufx + (size_t)p * N, *ubm = a.uprod + (size_t)p * N;
    const int2* kab = a.kern + (size_t)(kr - p / a.nbocc + a.nk - 1) * N;
    cx x[E];
    pair_potential<N>(x, wa, ub, kab, buf, tw_s, twn_s, tl, team);
    const int sb = a.pexp != nullptr ? 0 : 2 * a.shift[p];
    if (sb == 0) {
#pragma unroll
      for (int e = 0; e < E; ++e) acc[e] = fx::add(acc[e], fx::cmulc(ubm[TM::pos(tl, e)], fx::limbs(x[e])));
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e)
        acc[e] = fx::add(acc[e], fx_shift(fx::cmulc(ubm[TM::pos(tl, e)], fx::limbs(x[e])), sb));
    }
  }
  if (!valid) return;
#pragma unroll
  for (int e = 0; e < E; ++e) fx_accumulate(dst, N, TM::pos(tl, e), acc[e]);
}

// ---------------------------------------------------------------------------
// Adjoint of the exchange (k_adjoint.cu has the formulas): tile pairs as
// k_fock_sym_fx, two transform pairs per pair of orbitals.  v and mu have one
// scale each, without lifting small columns: the two pair densities of the second
// pass are subtracted, and a gradient takes absolute errors.  The factor i is left
// to the combine.  Bounded like the forward kernel; a gradient over 3 steps at
// NG = 256, NK = 32, Nocc = 4 went from 10.3 to 5.1 ms with it and the column-wise
// combine (13.1 ms with the forward exchange in FP64 as well).
// ---------------------------------------------------------------------------
template <int N>
__global__ void __launch_bounds__(sym_fx_threads<N>(), 2) k_fock_adj_fx(FockAdjFxArgs a) {
  using TM = fx::Team<N>;
  constexpr int E = TM::E, T = TM::T;
  const int S = a.S;
  const int nteam = blockDim.x / T;
  extern __shared__ int4 sm_fx[];
  lc* tw_s = reinterpret_cast<lc*>(sm_fx);                 // kTwCount
  cx* bufs = reinterpret_cast<cx*>(sm_fx + TM::kTwCount);  // nteam * N
  cx* cacc = bufs + nteam * N;                             // S * N
  const int tid = threadIdx.x, tl = tid % T, tw_ = tid / T;
  cx* buf = bufs + tw_ * N;
  int2* twn_s = reinterpret_cast<int2*>(cacc + S * N);  // kTwCount
  load_twiddles<N>(a.tw, tw_s, twn_s);
  if (blockIdx.x == 0) {
    const double2 f = fx_output_scale(Scale{a.vscale->x, a.vscale->y}, Scale{a.muscale->x, a.muscale->y},
                                      Scale{a.kscale->x, a.kscale->y});
    for (int i = tid; i < a.nk * a.nbocc; i += blockDim.x) a.fscale[i] = f;
  }
  for (int i = tid; i < S * N; i += blockDim.x) cacc[i] = cx{0, 0};
  int ti = 0, rem = blockIdx.x;
  while (rem >= a.T - ti) { rem -= a.T - ti; ++ti; }
  const int tj = ti + rem;
  const int M = a.nk * a.nbocc;
  const int ia = ti * S + tw_;
  const bool va = tw_ < S && ia < M;
  const int oa = va ? ia : 0;
  const int ka = oa / a.nbocc;
  const lc* vA = a.v + (size_t)oa * N;
  const lc* mA = a.mu + (size_t)oa * N;
  cx racc[E];
#pragma unroll
  for (int e = 0; e < E; ++e) racc[e] = cx{0, 0};
  __syncthreads();
  const bool diag = (ti == tj);
  const int nrounds = diag ? (S / 2 + 1) : S;
  for (int r = 0; r < nrounds; ++r) {
    const int lb = (tw_ + r) % S;
    const int ib = tj * S + lb;
    bool valid = va && ib < M;
    if (diag && (S % 2 == 0) && r == S / 2 && tw_ >= S / 2) valid = false;
    const bool self = diag && r == 0;
    const int ob = ib < M ? ib : 0;
    const int kb = ob / a.nbocc;
    const lc* vB = a.v + (size_t)ob * N;
    const lc* mB = a.mu + (size_t)ob * N;
    const int2* kab = a.kern + (size_t)(ka - kb + a.nk - 1) * N;
    const int2 kba = __ldg(a.kern + (size_t)(kb - ka + a.nk - 1) * N + N / 2), kn = __ldg(kab + N / 2);
    cx* col = cacc + lb * N;
    cx x[E];
    // ---- pass A: x = conj(phi_ab), c = dk conj(R_ab) (-1)^m;
    //      out_a += conj(x + c) mu_b, out_b += x mu_a (on the diagonal out_a += x mu_a)
    {
      const cx rn = pair_potential<N>(x, vA, vB, kab, buf, tw_s, twn_s, tl, tw_);
      if (valid) {
        if (self) {
#pragma unroll
          for (int e = 0; e < E; ++e) racc[e] = fx::add(racc[e], fx::cmul(fx::limbs(x[e]), mA[TM::pos(tl, e)]));
        } else {
          cx c{fx::rmul(rn.x, kba) - fx::rmul(rn.x, kn), fx::rmul(rn.y, kn) - fx::rmul(rn.y, kba)};
          if (tl & 1) c = cx{-c.x, -c.y};
#pragma unroll
          for (int e = 0; e < E; ++e) {
            const int q = TM::pos(tl, e);
            racc[e] = fx::add(racc[e], fx::cmulc(mB[q], fx::limbs(fx::add(x[e], c))));
            col[q] = fx::add(col[q], fx::cmul(fx::limbs(x[e]), mA[q]));
          }
        }
      }
    }
    // ---- pass B: x = conj(Phi_ab[mu_a conj(v_b) - v_a conj(mu_b)]),
    //      n2 = sum_m (-1)^m v_a conj(mu_b); conj(y) = x - dk conj(n2) (-1)^m;
    //      out_a += v_b y, out_b -= v_a conj(y)
    cx n2{0, 0};
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int q = TM::pos(tl, e);
      const cx t = fx::cmulc(vA[q], mB[q]);
      x[e] = fx::sub(fx::cmulc(mA[q], vB[q]), t);
      n2 = fx::add(n2, t);
    }
    if (tl & 1) n2 = cx{-n2.x, -n2.y};
#pragma unroll
    for (int o = (T < 32 ? T : 32) / 2; o > 0; o >>= 1) {
      n2.x += __shfl_xor_sync(0xffffffffu, n2.x, o);
      n2.y += __shfl_xor_sync(0xffffffffu, n2.y, o);
    }
    if constexpr (T > 32) {
      fx::team_sync<T>(tw_);
      if ((tl & 31) == 0) buf[tl >> 5] = n2;
      fx::team_sync<T>(tw_);
      n2 = fx::add(buf[0], buf[1]);
    }
    potential<N>(x, kab, buf, tw_s, twn_s, tl, tw_);
    if (valid) {
      cx c{fx::rmul(n2.x, kn) - fx::rmul(n2.x, kba), fx::rmul(n2.y, kba) - fx::rmul(n2.y, kn)};  // -dk conj(n2)
      if (tl & 1) c = cx{-c.x, -c.y};
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int q = TM::pos(tl, e);
        const lc y = fx::limbs(fx::add(x[e], c));
        racc[e] = fx::add(racc[e], fx::cmulc(vB[q], y));
        if (!self) col[q] = fx::sub(col[q], fx::cmul(y, vA[q]));
      }
    }
    __syncthreads();
  }
  if (va) {
    unsigned long long* dst = a.acc + (size_t)ia * 4 * N;
#pragma unroll
    for (int e = 0; e < E; ++e) fx_accumulate(dst, N, TM::pos(tl, e), racc[e]);
  }
  for (int i = tid; i < S * N; i += blockDim.x) {
    const int ib = tj * S + i / N;
    if (ib < M) fx_accumulate(a.acc + (size_t)ib * 4 * N, N, i % N, cacc[i]);
  }
}

// Kernel table: K^ = kern s_k, with s_k the largest short factor that keeps
// sum_G |K^(G)| below 2^60 for every k - k'.
__global__ void __launch_bounds__(1024) k_fx_kern_scale(const double* __restrict__ kern, int nd, int N, int2* kscale) {
  __shared__ double red[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double m = 0.0;
  for (int d = warp; d < nd; d += 32) {
    double s = 0.0;
    for (int i = lane; i < N; i += 32) s += fabs(kern[(size_t)d * N + i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    m = fmax(m, s);
  }
  if (lane == 0) red[warp] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 32; ++w) m = fmax(m, red[w]);
    // 2^60 (1 - 2e-5) / m
    int e = 0;
    const float f = m > 1e-280 ? (float)(2.0 * frexp(1.1529e18 / m, &e)) : 1.0f;
    const Scale s = m > 1e-280 ? fx_short_scale(f * (1.0f - 1.0f / 65536.0f), e - 1) : Scale{8, -3};
    *kscale = make_int2(s.c, s.k);
  }
}
__global__ void k_fx_kern(const double* __restrict__ kern, int n, const int2* __restrict__ kscale, int2* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const i64 v = fx_convert(kern[i], Scale{kscale->x, kscale->y});
  out[i] = fx::real_limbs(v);
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
template <int N>
static void sym_fx_shape(int S, int* threads, size_t* smem) {
  using TM = fx::Team<N>;
  *threads = (S * TM::T + 31) / 32 * 32;
  *smem = 24 * (size_t)TM::kTwCount + 16 * (size_t)N * (*threads / TM::T + S);
}

template <int N>
static cudaError_t fock_sym_fx_impl(const FockFxArgs& a, cudaStream_t s) {
  const int tiles = a.T * (a.T + 1) / 2;
  if (tiles == 0) return cudaSuccess;
  int threads;
  size_t smem;
  sym_fx_shape<N>(a.S, &threads, &smem);
  k_fock_sym_fx<N><<<tiles, threads, smem, s>>>(a);
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

// after launch_fx_convert
cudaError_t launch_fock_sym_fx(int NG, const FockFxArgs& a, cudaStream_t s) {
#define CALL(n) fock_sym_fx_impl<n>(a, s)
  MATTOHF_DISPATCH(NG, CALL)
#undef CALL
}

template <int N>
static cudaError_t fock_sym_fx_batch_impl(const FockFxArgs* d_args, const int* d_tile_pre, int nruns, int S,
                                          int total_tiles, const int* d_elem_pre, int total_elems, cudaStream_t s) {
  int threads;
  size_t smem;
  sym_fx_shape<N>(S, &threads, &smem);
  k_fx_convert_batch<<<total_elems / N, 128, 0, s>>>(d_args, d_elem_pre, nruns, N);
  k_fock_sym_fx_batch<N><<<total_tiles, threads, smem, s>>>(d_args, d_tile_pre, nruns);
  return cudaGetLastError();
}

cudaError_t launch_fock_sym_fx_batch(int NG, const FockFxArgs* d_args, const int* d_tile_pre, int nruns, int S,
                                     int total_tiles, const int* d_elem_pre, int total_elems, cudaStream_t s) {
  if (total_tiles <= 0) return cudaSuccess;
#define CALL(n) fock_sym_fx_batch_impl<n>(d_args, d_tile_pre, nruns, S, total_tiles, d_elem_pre, total_elems, s)
  MATTOHF_DISPATCH(NG, CALL)
#undef CALL
}

cudaError_t launch_fx_sizes(int NG, const FockFxArgs& a, cudaStream_t s) {
  k_fx_sizes<<<(a.nk * a.nbocc + 3) / 4, 128, 0, s>>>(a, NG);
  return cudaGetLastError();
}
cudaError_t launch_fx_sizes_batch(int NG, const FockFxArgs* d_args, const int* d_elem_pre, int nruns, int total_elems,
                                  cudaStream_t s) {
  if (total_elems <= 0) return cudaSuccess;
  k_fx_sizes_batch<<<(total_elems / NG + 3) / 4, 128, 0, s>>>(d_args, d_elem_pre, nruns, NG);
  return cudaGetLastError();
}

cudaError_t launch_fx_convert(int NG, const FockFxArgs& a, const FockFxRows* r, bool have_sizes, bool have_orbitals,
                              cudaStream_t s) {
  const int M = a.nk * a.nbocc;
  // up to 16 orbitals every CTA takes all the sizes itself: a launch less
  const bool scan = !have_sizes && !have_orbitals && M <= 16;
  if (!have_sizes && !have_orbitals && !scan) {
    const cudaError_t e = launch_fx_sizes(NG, a, s);
    if (e != cudaSuccess) return e;
  }
  const int n = (have_orbitals ? 0 : M) + (r ? r->ncols : 0);
  if (n == 0) return cudaSuccess;
  k_fx_convert<<<n, 128, 0, s>>>(a, r ? *r : FockFxRows{}, NG, have_orbitals ? M : 0, scan);
  return cudaGetLastError();
}

cudaError_t launch_fx_points(int NG, const FockFxArgs& a, cudaStream_t s) {
  k_fx_points<<<NG / 8, 512, 0, s>>>(a, NG);
  return cudaGetLastError();
}

template <int N>
static constexpr size_t rows_fx_smem() {
  return 24 * (size_t)fx::Team<N>::kTwCount + 16 * (size_t)N * rows_fx_teams<N>();
}

template <int N>
static cudaError_t fock_fx_impl(const FockFxArgs& a, const FockFxRows& r, cudaStream_t s) {
  constexpr int R = rows_fx_teams<N>();
  k_fock_fx<N><<<(r.ncols + R - 1) / R * r.nchunks, kRowsThreads, rows_fx_smem<N>(), s>>>(a, r);
  return cudaGetLastError();
}

cudaError_t launch_fock_fx(int NG, const FockFxArgs& a, const FockFxRows& r, cudaStream_t s) {
  if (r.ncols <= 0) return cudaSuccess;
#define CALL(n) fock_fx_impl<n>(a, r, s)
  MATTOHF_DISPATCH(NG, CALL)
#undef CALL
}

// Chunks of the sources for ncols columns: enough CTAs to fill the device's
// SMs several times over.
void fx_rows_split(int NG, int ncols, int npairs, int nsm, int fixed, int* nchunks, int* chunk) {
  int nch = fixed;
  if (nch <= 0) {
    const int groups = (ncols + fx_rows_teams(NG) - 1) / fx_rows_teams(NG);
    nch = (std::max(1, nsm) * kRowsCtasPerSm + groups - 1) / groups;
  }
  nch = std::max(1, std::min(nch, npairs));
  const int ch = (npairs + nch - 1) / nch;
  *chunk = ch;
  *nchunks = (npairs + ch - 1) / ch;
}

int fx_rows_teams(int NG) {
  switch (NG) {
    case 16: return rows_fx_teams<16>();
    case 32: return rows_fx_teams<32>();
    case 64: return rows_fx_teams<64>();
    case 128: return rows_fx_teams<128>();
    case 256: return rows_fx_teams<256>();
    default: return rows_fx_teams<512>();
  }
}

template <int N>
static cudaError_t fock_adj_fx_impl(const FockAdjFxArgs& a, cudaStream_t s) {
  int threads;
  size_t smem;
  sym_fx_shape<N>(a.S, &threads, &smem);
  k_fock_adj_fx<N><<<a.T * (a.T + 1) / 2, threads, smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_fx_convert2(int NG, const FockFxArgs& a, const FockFxArgs& b, cudaStream_t s) {
  const int M = a.nk * a.nbocc;
  k_fx_sizes2<<<dim3((M + 3) / 4, 2), 128, 0, s>>>(a, b, NG);
  k_fx_convert2<<<dim3(M, 2), 128, 0, s>>>(a, b, NG);
  return cudaGetLastError();
}

cudaError_t launch_fock_adj_fx(int NG, const FockAdjFxArgs& a, cudaStream_t s) {
  if (a.T <= 0) return cudaSuccess;
#define CALL(n) fock_adj_fx_impl<n>(a, s)
  MATTOHF_DISPATCH(NG, CALL)
#undef CALL
}

cudaError_t launch_fx_kern(const double* kern, int nd, int NG, int2* kscale, int2* out, cudaStream_t s) {
  k_fx_kern_scale<<<1, 1024, 0, s>>>(kern, nd, NG, kscale);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_fx_kern<<<(nd * NG + 255) / 256, 256, 0, s>>>(kern, nd * NG, kscale, out);
  return cudaGetLastError();
}

// The first eighth of the circle gives the others: where long double has 113 bits
// in software, a context of 256 points spent 0.3 ms on 544 sines.
std::vector<longlong2> fx_roots(int N) {
  std::vector<longlong2> c(N / 8 + 1), r(N);  // (cos, sin) of 2 pi j / N
  const long double step = 2.0L * acosl(-1.0L) / (long double)N;
  for (int j = 0; j <= N / 8; ++j)
    c[j] = make_longlong2(llrintl(ldexpl(cosl(step * j), fx::kOne)), llrintl(ldexpl(sinl(step * j), fx::kOne)));
  for (int t = 0; t < N; ++t) {
    const int q = t / (N / 4), j = t % (N / 4);
    const longlong2 z = j <= N / 8 ? c[j] : make_longlong2(c[N / 4 - j].y, c[N / 4 - j].x);
    r[t] = q == 0 ? make_longlong2(z.x, -z.y) : q == 1 ? make_longlong2(-z.y, -z.x) : q == 2 ? make_longlong2(-z.x, z.y) : make_longlong2(z.y, z.x);
  }
  return r;
}

template <int N, int V = 0>
static int fx_twiddles(int4* out) {
  using TM = fx::Team<N, V>;
  if (!out) return TM::kTwCount;
  const std::vector<longlong2> roots = fx_roots(N);
  int n = 0;
  auto put = [&](int num, int den) {
    const longlong2 z = roots[num % den * (N / den)];
    const long long m = (1ll << fx::kLimb) - 1;
    out[n++] = make_int4((int)(z.x >> fx::kLimb), (int)(z.x & m), (int)(z.y >> fx::kLimb), (int)(z.y & m));
  };
  if (TM::R1 > 1)
    for (int r = 0; r < TM::R1; ++r)
      for (int k = 0; k < TM::R0; ++k) put(r * k, TM::R0 * TM::R1);
  for (int r = 0; r < TM::R0; ++r)
    for (int j = 0; j < TM::STRIDE; ++j) put(r * j, N);
  return n;
}

int fx_twiddle_table(int NG, int4* out, bool latency) {
  if (latency && NG == 64) return fx_twiddles<64, 1>(out);
  switch (NG) {
    case 16: return fx_twiddles<16>(out);
    case 32: return fx_twiddles<32>(out);
    case 64: return fx_twiddles<64>(out);
    case 128: return fx_twiddles<128>(out);
    case 256: return fx_twiddles<256>(out);
    case 512: return fx_twiddles<512>(out);
    default: return 0;
  }
}

template <int N>
static cudaError_t configure_fx_impl() {
  int threads;
  size_t smem;
  sym_fx_shape<N>(sym_fx_threads<N>() / fx::Team<N>::T, &threads, &smem);
  const cudaError_t e = cudaFuncSetAttribute(k_fock_sym_fx<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const cudaError_t e1 = cudaFuncSetAttribute(k_fock_adj_fx<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e1 != cudaSuccess) return e1;
  const cudaError_t e2 =
      cudaFuncSetAttribute(k_fock_fx<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rows_fx_smem<N>());
  if (e2 != cudaSuccess) return e2;
  return cudaFuncSetAttribute(k_fock_sym_fx_batch<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

cudaError_t configure_fx_kernels() {
  cudaError_t e;
  if ((e = configure_fx_impl<16>()) != cudaSuccess) return e;
  if ((e = configure_fx_impl<32>()) != cudaSuccess) return e;
  if ((e = configure_fx_impl<64>()) != cudaSuccess) return e;
  if ((e = configure_fx_impl<128>()) != cudaSuccess) return e;
  if ((e = configure_fx_impl<256>()) != cudaSuccess) return e;
  return configure_fx_impl<512>();
}

}  // namespace mattohf
