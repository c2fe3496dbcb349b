// Fused RK4 stage for small problems in 64-bit fixed point: k_small.cu's work, where
// that kernel is bound by the FP64 pipe (an SM's rate is one instruction per 19 cycles).
//
// Differences.  The pairs, the kinetic term and the Hartree potential are transformed
// in fixed point (fft_fx.cuh); the density is summed by the pair teams, which hold the
// orbitals in fixed point, and pushed to the column's first CTA (a second cluster
// barrier phase); FP64 remains in the Parseval sums, the sums over CTAs and the update.
//
// One FP64 instruction becomes 12 to 20 integer ones, which a warp runs once a launch
// and so fetches cold: with few orbitals k_small.cu stays faster.  us per RK4 step
// at NG / NK / bands, FP64 against this: 16/4/2 24 34, 32/16/2 29 37, 64/8/2 29 37;
// 64/8/4 86 44, 128/8/2 71 65, 256/4/2 79 70, 256/8/2 83 77 (separate launches: 61, 68, 83,
// 85 from 64/8/4 on).  Hence from 64 points and M NG = 2048 on (small_stage_fx).
#include "fx_convert.cuh"
#include "small_stage.cuh"

namespace mattohf {

template <int N>
struct SmallFxLayout {
  using TM = fx::Team<N, 1>;
  static constexpr int PW = 32 / TM::T;
  static constexpr int NTEAM = kSmallWarps * PW;
  // tw, bufs[NTEAM][N], K[N] (16 bytes each); negated twiddles; vH[N] (fixed point);
  // rho[N], vh[N]; then what the cluster's CTAs push to this one: for its share of
  // the grid points the P exchange partials (at most 2N + 2 kSmallMaxCtas doubles),
  // vH and T_A w (N and 2N doubles), and to the first CTA the densities [P][N]
  static constexpr int RECV_F = kSmallRecvF<N>;
  static constexpr size_t bytes = 16 * ((size_t)N * (NTEAM + 1) + TM::kTwCount) + 8 * (size_t)TM::kTwCount +
                                  sizeof(double) * (RECV_F + (size_t)N * (6 + kSmallMaxCtas));
  // the adjoint's variant also stages its stage-store copy (N double2)
  static constexpr size_t bytes_adj = bytes + sizeof(double2) * (size_t)N;
};

// Size of a team's values (fx_size); every lane of the warp calls it.
template <int T, int E>
__device__ __forceinline__ int2 team_size(const double2 (&v)[E]) {
  int m = 0;
#pragma unroll
  for (int e = 0; e < E; ++e) m = max(m, max(__double2hiint(v[e].x) & 0x7fffffff, __double2hiint(v[e].y) & 0x7fffffff));
#pragma unroll
  for (int o = T / 2; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  const int ex = m >> 20;
  float s = 0.0f;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const float x = fx_mantissa(__double2hiint(v[e].x) & 0x7fffffff, ex), y = fx_mantissa(__double2hiint(v[e].y) & 0x7fffffff, ex);
    s = fmaf(x, x, fmaf(y, y, s));
  }
#pragma unroll
  for (int o = T / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return fx_size(m, s);
}
// Scales are powers of two here, so that nothing has to be divided by them.
__device__ __forceinline__ Scale binary_scale(Scale s) { return Scale{s.c ? 8 : 0, s.k}; }

// x <- conj(x k 2^-g) 2^r for the real factors k 2^-g (real_limbs; 2^58 <= |k| < 2^60 or
// zero, 0 <= g <= kMaxShift), ready for the way back, with r from the product's norm:
// its N values' partial sums stay below 2^60.5 whatever the factors' range (a kinetic
// energy's is 2^12 and more between the frequencies that carry a function and the
// largest).  The factors being normalised, the rounding of a product to a place is
// no larger than what the transform has left in x.  Returns r.
constexpr int kMaxShift = 100;
template <int N, int T, int E>
__device__ __forceinline__ int multiply_back(cx (&x)[E], const int2 (&k)[E], const int (&g)[E]) {
  constexpr int kLog2N = N == 64 ? 6 : N == 128 ? 7 : 8;
  float s = 0.0f;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    x[e] = cx{fx::rmul(x[e].x, k[e]), -fx::rmul(x[e].y, k[e])};
    const float f = __int_as_float((127 - g[e]) << 23), p = __ll2float_rn(x[e].x) * f, q = __ll2float_rn(x[e].y) * f;
    s = fmaf(p, p, fmaf(q, q, s));
  }
#pragma unroll
  for (int o = T / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  // N s < 2^(log2 N + e + 1) for the exponent e of s; at most 2^120
  const int r = min(29, max(-8, (119 - kLog2N - ((__float_as_int(s) >> 23) - 127)) >> 1));
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int q = r - g[e], left = max(q, 0), right = min(62, max(-q, 0));
    const i64 half = (1ll << right) >> 1;
    x[e] = cx{((x[e].x << left) + half) >> right, ((x[e].y << left) + half) >> right};
  }
  return r;
}

// v 2^e in integer work; v is normal or zero
__device__ __forceinline__ double shift_exponent(double v, int e) {
  const int hi = __double2hiint(v), x = ((hi >> 20) & 0x7ff) + e;
  if (x <= 0 || ((hi >> 20) & 0x7ff) == 0) return 0.0;
  if (x >= 0x7ff) return __hiloint2double((hi & 0x80000000) | 0x7ff00000, 0);
  return __hiloint2double(hi + (e << 20), __double2loint(v));
}
// an integer times 2^e, or no number
__device__ __forceinline__ double fx_to_double(i64 v, int e, bool ok) {
  return ok ? shift_exponent((double)v, e) : __longlong_as_double(0x7ff8000000000000ll);
}

template <int N, bool ADJ>
__global__ void __launch_bounds__(kSmallThreads) k_small_stage_fx(SmallStageArgs a) {
  using TM = fx::Team<N, 1>;
  constexpr int E = TM::E, T = TM::T, PW = 32 / T;
  constexpr int NTEAM = SmallFxLayout<N>::NTEAM;
  constexpr int kLog2N = N == 64 ? 6 : N == 128 ? 7 : 8;
  namespace cg = cooperative_groups;
  extern __shared__ int4 sm_small[];
  lc* tw_s = reinterpret_cast<lc*>(sm_small);                   // kTwCount
  cx* bufs = reinterpret_cast<cx*>(sm_small + TM::kTwCount);    // NTEAM * N
  cx* Ki_s = bufs + NTEAM * N;                                  // N: T_A w (the column's first CTA)
  int2* twn_s = reinterpret_cast<int2*>(Ki_s + N);              // kTwCount
  i64* vhi_s = reinterpret_cast<i64*>(twn_s + TM::kTwCount);    // N: vH
  double* rho_s = reinterpret_cast<double*>(vhi_s + N);
  double* vh_s = rho_s + N;
  double* recvF = vh_s + N;                             // [P][2 per]: the partials of this CTA's points
  double* recvR = recvF + SmallFxLayout<N>::RECV_F + 3 * N;  // behind vH and T_A w at its points;                      // [kSmallMaxCtas][N]: densities (the first CTA)
  double2* st_s = reinterpret_cast<double2*>(recvR + kSmallMaxCtas * N);  // [per]: staged stage-store copy (ADJ)
  __shared__ int2 size_s[kSmallWarps];
  __shared__ int2 escale_s[3];               // exponent and validity of: exchange, vH, T_A w
  __shared__ double2 kinv_s;                 // 1 / c of the kernel table's scale, and its error
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tl = lane % T, team = warp * PW + lane / T;
  cx* buf = bufs + team * N;
  const int ncols = a.nk * a.nb;
  const int c = blockIdx.x / a.P;          // output column (k, b)
  const int chunk = blockIdx.x % a.P;      // rank in the column's cluster
  const int kr = c / a.nb, ib = c % a.nb;
  const int M = a.nk * a.nbocc;
  // This CTA's exchange pairs.  With more than one CTA per column the first
  // CTA takes none: its warps carry the density, the kinetic and Hartree
  // transforms and the Parseval sums, and the other CTAs split the pairs
  // evenly on all eight warps.  A single CTA runs them on warps 0-5.
  const int p0 = (a.P == 1 || chunk == 0) ? 0 : (M * (chunk - 1)) / (a.P - 1);
  const int p1 = a.P == 1 ? M : chunk == 0 ? 0 : (M * chunk) / (a.P - 1);
  const int workers = a.P == 1 ? kSmallWarps - 2 : chunk == 0 ? 0 : kSmallWarps;  // pair warps 0 .. workers-1
  const int worker_teams = workers * PW;
  const bool occupied = ib < a.nbocc;
  const bool obs = a.mode == 0 || a.mode == 4;
  const double2* wcol = a.u + (size_t)c * N;

  for (int i = tid; i < TM::kTwCount; i += kSmallThreads) {
    const lc w = a.tw_fx[i];
    tw_s[i] = w;
    twn_s[i] = make_int2(fx::neg_hi(w.yh), fx::neg_lo(w.yl));
  }
  if (tid == 0) {
    const double d = (double)a.kscale->x;
    double r = (double)(1.0f / (float)a.kscale->x);
    r = fma(fma(-r, d, 1.0), r, r);
    r = fma(fma(-r, d, 1.0), r, r);
    kinv_s = make_double2(r, fma(-r, d, 1.0) * r);
    escale_s[0] = make_int2(0, 1);
  }
  const bool hartree = chunk == 0 && warp == kSmallWarps - 1;
  int2 vg[E];  // the Hartree warp: vCG 2^kv = vg 2^-gg, vg < 2^60
  int gg[E], kv = 0;
  if (hartree) {
    int m = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) m = max(m, __double2hiint(a.vCG[TM::pos(tl, e)]) & 0x7fffffff);
    kv = 1082 - max(1, __reduce_max_sync(0xffffffffu, m) >> 20);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const double v = a.vCG[TM::pos(tl, e)];
      gg[e] = min(kMaxShift, 1082 - kv - max(1, (__double2hiint(v) & 0x7fffffff) >> 20));
      vg[e] = fx::real_limbs(fx_convert(v, Scale{8, kv - 3 + gg[e]}));
    }
  }
  __syncthreads();
  // Launched as a programmatic dependent of the previous stage: everything
  // above reads only constant tables.  Wait for the previous grid to complete
  // (and its writes to be visible) before touching the state or the scratch,
  // then let the next stage's grid start its own prologue.  Both are no-ops
  // without a programmatic dependency.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  // every CTA of the cluster has started once this barrier phase completes;
  // it is waited for only before the first store to another CTA's memory
  asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
  if (a.it_out && blockIdx.x == 0 && tid == 0) *a.it_out = *a.it + a.it_inc;
  if (ADJ) small_stage_in<N>(a, wcol, st_s);
  // Density: every CTA sums |u|^2 over its pairs' orbitals, which its pair teams
  // hold in fixed point with one scale for the CTA, and pushes the sum to the
  // column's first CTA.  The cluster's second barrier phase completes when all have.
  const int n = p1 - p0;
  const bool one_round = n <= worker_teams, worker = warp < workers;
  double2 uv[E], wv[E];
  lc ul[E];
  Scale su{0, 0}, sw{0, 0};
  auto load_pair = [&](int p) {
    const double2* ucol = a.u + ((size_t)(p / a.nbocc) * a.nb + p % a.nbocc) * N;
#pragma unroll
    for (int e = 0; e < E; ++e) uv[e] = ucol[TM::pos(tl, e)];
  };
  auto convert_pair = [&]() {
#pragma unroll
    for (int e = 0; e < E; ++e) ul[e] = fx::limbs(cx{fx_convert(uv[e].x, su), fx_convert(uv[e].y, su)});
  };
  if (worker) {
    int2 zu = make_int2(0, 0);
    // warp-uniform trip counts: every team of a warp runs the same rounds
    for (int base = p0 + warp * PW; base < p1; base += worker_teams) {
      load_pair(min(base + lane / T, p1 - 1));
      zu = fx_larger(zu, team_size<T>(uv));
    }
#pragma unroll
    for (int o = 16; o >= T; o >>= 1)
      zu = fx_larger(zu, make_int2(__shfl_xor_sync(0xffffffffu, zu.x, o), __shfl_xor_sync(0xffffffffu, zu.y, o)));
    if (lane == 0) size_s[warp] = zu;
#pragma unroll
    for (int e = 0; e < E; ++e) wv[e] = wcol[TM::pos(tl, e)];
    sw = binary_scale(fx_scale(team_size<T>(wv), 1e30f, 1.0f));
    asm volatile("bar.sync 4, %0;" ::"r"(32 * workers) : "memory");
    for (int w = 0; w < workers; ++w) zu = fx_larger(zu, size_s[w]);
    // sums of n terms, at most 2^59.3 each at the full peak (k_fock_fx.cu), below 2^62.9
    su = binary_scale(fx_scale(zu, kPeak * fminf(1.0f, (float)kFxTerms / (float)n), 1.0f));
    i64 rr[E];
#pragma unroll
    for (int e = 0; e < E; ++e) rr[e] = 0;
    for (int base = p0 + warp * PW; base < p1; base += worker_teams) {
      if (!one_round) load_pair(min(base + lane / T, p1 - 1));
      convert_pair();
      if (base + lane / T < p1) {
#pragma unroll
        for (int e = 0; e < E; ++e) rr[e] += fx::cmulc(ul[e], ul[e]).x;
      }
    }
#pragma unroll
    for (int e = 0; e < E; ++e) buf[TM::pos(tl, e)].x = rr[e];
    if (tid == 0) escale_s[0] = make_int2(171 - 2 * su.k - sw.k - a.kscale->y, su.c != 0 && sw.c != 0);
    asm volatile("bar.sync 4, %0;" ::"r"(32 * workers) : "memory");
  }
  asm volatile("barrier.cluster.wait;" ::: "memory");
  if (worker) {
    double* dst = cg::this_cluster().map_shared_rank(recvR, 0) + (chunk > 0 ? chunk - 1 : 0) * N;
    const int act = min(worker_teams, n);
    for (int q = tid; q < N; q += 32 * workers) {
      i64 s = 0;
      for (int t2 = 0; t2 < act; ++t2) s += bufs[(size_t)t2 * N + q].x;
      dst[q] = fx_to_double(s, 54 - 2 * su.k, su.c != 0);  // 2^60 / su^2
    }
    asm volatile("bar.sync 4, %0;" ::"r"(32 * workers) : "memory");
  }
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  // The first CTA adds the densities on warps 0, 1, 4 and 5 (a single CTA: on the
  // Hartree warp).
  const bool adds = chunk == 0 && a.P > 1 && (warp & 2) == 0;
  const bool waited = adds || hartree;
  if (waited) asm volatile("barrier.cluster.wait;" ::: "memory");
  if (adds) {
    for (int q = (warp < 2 ? warp : warp - 2) * 32 + lane; q < N; q += 128) {
      double r = recvR[q];
      for (int j = 1; j < a.P - 1; ++j) r += recvR[j * N + q];
      rho_s[q] = a.occ * r;
    }
    asm volatile("bar.sync 1, 160;" ::: "memory");
  }
  // Ekin and Je of the input column at the previous step's field (Parseval)
  auto parseval = [&](const cx (&X)[E], Scale s) {
    const int itn = *a.it;
    const double Ao = (itn >= 1 && a.Aobs) ? a.Aobs[itn - 1] : 0.0;
    const double kAx = a.kx[kr] + Ao, kA2 = kAx * kAx;
    const Unscale un = fx_unscale(s);
    double ek = 0.0, je = 0.0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const double G = a.Gx[TM::pos(tl, e)], xr = un(X[e].x), xi = un(X[e].y);
      const double m2 = xr * xr + xi * xi;
      ek += 0.5 * (G * G + 2.0 * G * kAx + kA2) * m2;
      je += (G + a.kx[kr] + Ao) * m2;
    }
#pragma unroll
    for (int o = T / 2; o > 0; o >>= 1) {
      ek += __shfl_xor_sync(0xffffffffu, ek, o);
      je += __shfl_xor_sync(0xffffffffu, je, o);
    }
    if (lane == 0) {
      a.colbuf[(size_t)c * 4] = ek / (double)N;
      a.colbuf[(size_t)c * 4 + 1] = je / (double)N;
    }
  };
  // the column's transform
  auto column_forward = [&](cx (&X)[E]) {
#pragma unroll
    for (int e = 0; e < E; ++e) wv[e] = wcol[TM::pos(tl, e)];
    const Scale s = fx_fft_scale(team_size<T>(wv), N);
#pragma unroll
    for (int e = 0; e < E; ++e) X[e] = cx{fx_convert(wv[e].x, s), fx_convert(wv[e].y, s)};
    fx::forward<N, false, 1>(X, buf, tw_s, twn_s, tl, team);
    return s;
  };
  if (hartree) {
    // vH (F:147-162)
    if (a.P == 1) {
      for (int q = lane; q < N; q += 32) rho_s[q] = a.occ * recvR[q];
      __syncwarp();
    } else {
      asm volatile("bar.sync 1, 160;" ::: "memory");
    }
#pragma unroll
    for (int e = 0; e < E; ++e) wv[e] = make_double2(rho_s[TM::pos(tl, e)], 0.0);
    const Scale s = fx_fft_scale(team_size<T>(wv), N);
    cx x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) x[e] = cx{fx_convert(wv[e].x, s), 0};
    fx::forward<N, false, 1>(x, buf, tw_s, twn_s, tl, team);
    const int r = multiply_back<N, T>(x, vg, gg);
    fx::forward<N, false, 1>(x, buf, tw_s, twn_s, tl, team);
    if (lane < T) {
#pragma unroll
      for (int e = 0; e < E; ++e) vhi_s[TM::pos(tl, e)] = x[e].x;
    }
    if (lane == 0) escale_s[1] = make_int2(57 - kLog2N - s.k - kv - r, s.c != 0);
  } else if (chunk == 0 && warp == kSmallWarps - 2) {
    // kinetic term T_A w of column c at the stage field (F:212-234): (G + k + A)^2 / 2
    // by integer squares, and, for stage 0 and the closing pass, Ekin and Je on the
    // same forward transform
    cx x[E];
    const Scale s = column_forward(x);
    if (obs && !(a.mode == 0 && a.P > 1)) parseval(x, s);
    if (a.mode != 4) {
      const double kA = a.kx[kr] + afield_value(a.af);
      int m = __double2hiint(kA) & 0x7fffffff;
#pragma unroll
      for (int e = 0; e < E; ++e) m = max(m, __double2hiint(a.Gx[TM::pos(tl, e)]) & 0x7fffffff);
      m = max(1, __reduce_max_sync(0xffffffffu, m) >> 20);
      const Scale st{8, 1077 - m};  // |G|, |k + A| < 2^(m - 1022): their sum below 2^59
      const i64 kf = fx_convert(kA, st);
      // every factor with an exponent of its own: with one for all, those of the low
      // frequencies, which carry the orbital, were off by 2^-57 of the largest (3e-14
      // Hartree at NG = 256 and a cell of 10), the same way in every step
      int2 t2[E];
      int g[E];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        i64 t = fx_convert(a.Gx[TM::pos(tl, e)], st) + kf;
        const int h = min(29, max(0, __clzll(t < 0 ? -t : t) - 4));  // to 2^59 and more
        t <<= h;
        g[e] = 2 * h;
        t2[e] = fx::real_limbs(fx::rmul(t, fx::real_limbs(t)));
      }
      const int r = multiply_back<N, T>(x, t2, g);
      fx::forward<N, false, 1>(x, buf, tw_s, twn_s, tl, team);
      if (lane < T) {
#pragma unroll
        for (int e = 0; e < E; ++e) Ki_s[TM::pos(tl, e)] = cx{x[e].x, -x[e].y};
      }
      // 2^120 / (2 N s st^2)
      if (lane == 0) escale_s[2] = make_int2(110 - kLog2N - s.k - 2 * st.k - r, s.c != 0 && m < 0x7ff);
    }
  } else if (chunk == 0 && a.P > 1 && warp == 3 && a.mode == 0) {
    // beside the kinetic warp's transforms
    cx x[E];
    const Scale s = column_forward(x);
    parseval(x, s);
  } else if (worker && a.hf && (a.mode != 4 || occupied)) {
    // this CTA's exchange pairs of column c, one pair per team per round
    lc wl[E];
    cx acc[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      wl[e] = fx::limbs(cx{fx_convert(wv[e].x, sw), fx_convert(wv[e].y, sw)});
      acc[e] = cx{0, 0};
    }
    for (int base = p0 + warp * PW; base < p1; base += worker_teams) {
      const int p = min(base + lane / T, p1 - 1);
      if (!one_round) {
        load_pair(p);
        convert_pair();
      }
      const int2* kern = a.kern_fx + (size_t)(kr - p / a.nbocc + a.nk - 1) * N;
      // the pair's kernel row, loaded while the forward transform runs
      int2 kf[E];
      cx x[E];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        kf[e] = __ldg(kern + TM::pos(tl, e));
        x[e] = fx::cmulc(wl[e], ul[e]);
      }
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        fx::forward<N, false, 1>(x, buf, tw_s, twn_s, tl, team);
        if (h == 0) {
#pragma unroll
          for (int e = 0; e < E; ++e) x[e] = cx{fx::rmul(x[e].x, kf[e]), -fx::rmul(x[e].y, kf[e])};
        }
      }
      if (base + lane / T < p1) {
#pragma unroll
        for (int e = 0; e < E; ++e) acc[e] = fx::add(acc[e], fx::cmulc(ul[e], fx::limbs(x[e])));
      }
    }
    __syncwarp();
#pragma unroll
    for (int e = 0; e < E; ++e) buf[TM::pos(tl, e)] = acc[e];
  }
  // stage 1: the observables of the previous step's state, from the column
  // buffer and the density stage 0 left (stage 0 completed before this grid
  // passed griddepcontrol.wait), on an idle warp of column 0's first CTA
  if (a.mode == 1 && c == 0 && chunk == 0 && warp == (a.P > 1 ? 2 : kSmallWarps - 1))
    small_finalize(a, a.obs_dens, a.obs_dens + N, N);
  const int act = (a.hf && (a.mode != 4 || occupied)) ? min(worker_teams, n) : 0;
  small_finish<N, ADJ>(
      a, wcol, recvF, st_s, rho_s, vh_s,
      [&] {
        if (!waited) asm volatile("barrier.cluster.wait;" ::: "memory");
      },
      [&](int i) {
        const i64* bd = reinterpret_cast<const i64*>(bufs);
        i64 sum = 0;
        for (int t2 = 0; t2 < act; ++t2) sum += bd[(size_t)t2 * 2 * N + i];
        if (act <= 0) return 0.0;
        const int2 es = escale_s[0];
        const double2 ki = kinv_s;
        const double x = (double)sum;
        return es.y ? shift_exponent(fma(x, ki.x, x * ki.y), es.x) : __longlong_as_double(0x7ff8000000000000ll);
      },
      [&](int per, double* recvV, double* recvK) {
        const int2 ev = escale_s[1], ek = escale_s[2];
        for (int q = tid; q < N; q += kSmallThreads) {
          const double vh = fx_to_double(vhi_s[q], ev.x, ev.y);
          vh_s[q] = vh;
          if (a.mode == 0 && c == 0) {
            // the density and vH of this stage input (the previous step's state)
            // for its observables, which stage 1 completes off this critical path
            a.obs_dens[q] = rho_s[q];
            a.obs_dens[N + q] = vh;
          }
          cg::this_cluster().map_shared_rank(recvV, q / per)[q % per] = vh;
        }
        if (a.mode == 4) return;
        const i64* kd = reinterpret_cast<const i64*>(Ki_s);
        for (int i = tid; i < 2 * N; i += kSmallThreads) {
          const int q = i >> 1, owner = q / per;
          cg::this_cluster().map_shared_rank(recvK, owner)[2 * (q - owner * per) + (i & 1)] = fx_to_double(kd[i], ek.x, ek.y);
        }
      });
}

template <int N, bool ADJ>
static cudaError_t small_fx_impl(const SmallStageArgs& a, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.nk * a.nb * a.P);
  cfg.blockDim = dim3(kSmallThreads);
  cfg.dynamicSmemBytes = ADJ ? SmallFxLayout<N>::bytes_adj : SmallFxLayout<N>::bytes;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;  // one cluster per output column
  attr[1].val.clusterDim.x = a.P;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, k_small_stage_fx<N, ADJ>, a);
}

template <int N>
static cudaError_t small_fx_configure() {
  cudaError_t e = cudaFuncSetAttribute(k_small_stage_fx<N, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)SmallFxLayout<N>::bytes_adj);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_small_stage_fx<N, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)SmallFxLayout<N>::bytes);
}

bool small_stage_fx(int NG, int M) { return NG >= 64 && M * NG >= 2048; }

cudaError_t launch_small_stage_fx(int NG, const SmallStageArgs& a, cudaStream_t s) {
  if (a.P < 1 || a.P > kSmallMaxCtas) return cudaErrorInvalidValue;
  const bool adj = a.store != nullptr || a.ckpt != nullptr;
  switch (NG) {
    case 64: return adj ? small_fx_impl<64, true>(a, s) : small_fx_impl<64, false>(a, s);
    case 128: return adj ? small_fx_impl<128, true>(a, s) : small_fx_impl<128, false>(a, s);
    case 256: return adj ? small_fx_impl<256, true>(a, s) : small_fx_impl<256, false>(a, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t configure_small_fx_kernels() {
  cudaError_t e;
  if ((e = small_fx_configure<64>()) != cudaSuccess) return e;
  if ((e = small_fx_configure<128>()) != cudaSuccess) return e;
  return small_fx_configure<256>();
}

}  // namespace mattohf
