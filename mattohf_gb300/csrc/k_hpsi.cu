// Hamiltonian-apply kernels: density + Hartree, Fock pair transforms, and the
// per-column combine (kinetic + local + exchange + RK4 / observable epilogues).
//
// Reference: src/Functions.f90 ubkwbk_hwbk (F:187-209), ubk_tubk (F:212-234),
// ubk_dns (F:55-71), dns_vH (F:147-162), ubkwbk_vFwbk (F:237-261), ubk_Ekin
// (F:94-119), ubk_Ex (F:165-183), ubk_Je (F:289-318); RK4 stages from
// src/RT_calculation.f90:154-173.
#include "fft.cuh"
#include "column_fx.cuh"
#include "internal.h"

namespace mattohf {

// ---------------------------------------------------------------------------
// Density (F:55-71) and Hartree potential (F:147-162), one CTA.
// ---------------------------------------------------------------------------
// Stage 1: partial densities of kDensChunks chunks of columns (fewer for few
// columns).  A CTA takes one chunk at 64 grid points, a quarter of the chunk per
// group of 64 threads: FP64 instructions of a warp come 64 cycles apart, so the
// columns of a thread are what the launch's time goes by.
__host__ __device__ __forceinline__ int dens_chunks(int ncol) {
  const int n = (ncol + 4 * kDensSub - 1) / (4 * kDensSub);
  return n < 1 ? 1 : n > kDensChunks ? kDensChunks : n;
}
__device__ __forceinline__ void dens_partial_body(const DensArgs& a, int N, int chunk, int group) {
  __shared__ double part_s[kDensSub][64], sig_s[kDensSub][64];
  const int ncol = a.nk * a.u.nb, nch = dens_chunks(ncol);
  if (chunk >= nch) return;
  const int per = (ncol + nch * kDensSub - 1) / (nch * kDensSub);
  const int pt = threadIdx.x & 63, sub = threadIdx.x >> 6;
  const int ig = group * 64 + pt;
  const int c0 = (chunk * kDensSub + sub) * per, c1 = min(ncol, c0 + per);
  double s = 0.0, t = 0.0;
  if (ig < N) {
    if (a.mu == nullptr) {
#pragma unroll 4
      for (int c = c0; c < c1; ++c) {
        const int ik = c / a.u.nb, ib = c % a.u.nb;
        const double occ = ib < a.nbocc ? a.occ : 0.0;
        const double2 z = a.u.p[(size_t)ik * a.u.kstride + (size_t)ib * N + ig];
        s += fma(occ * z.x, z.x, (occ * z.y) * z.y);
      }
    } else {
#pragma unroll 4
      for (int c = c0; c < c1; ++c) {   // the adjoint's: all bands are occupied
        const int ik = c / a.u.nb, ib = c % a.u.nb;
        const size_t o = (size_t)ik * a.u.kstride + (size_t)ib * N + ig;
        const double2 z = a.u.p[o], m = a.mu[o];
        s += fma(a.occ * z.x, z.x, (a.occ * z.y) * z.y);
        t += fma(m.x, z.y, -(m.y * z.x));
      }
    }
  }
  part_s[sub][pt] = s;
  if (a.mu != nullptr) sig_s[sub][pt] = t;
  __syncthreads();
  if (sub == 0 && ig < N) {
    for (int j = 1; j < kDensSub; ++j) s += part_s[j][pt];
    a.part[(size_t)chunk * N + ig] = s;
    if (a.mu == nullptr) return;
    for (int j = 1; j < kDensSub; ++j) t += sig_s[j][pt];
    a.part_sig[(size_t)chunk * N + ig] = t;
  }
}

__global__ void __launch_bounds__(64 * kDensSub) k_dens_partial(DensArgs a, int N) {
  dens_partial_body(a, N, blockIdx.x, blockIdx.y);
}

__global__ void __launch_bounds__(64 * kDensSub) k_dens_partial_batch(const DensArgs* __restrict__ args, int N) {
  dens_partial_body(args[blockIdx.z], N, blockIdx.x, blockIdx.y);
}

// Stage 2 (one CTA): rho = ordered sum of the chunk partials, then the
// Hartree potential (F:147-162), vloc = vH + vion and the density scalars.
// The transforms are fixed-point (fft_fx.cuh); the product with vCG is FP64, one
// value per thread, with a new scale for the second transform.
template <int N>
__device__ __forceinline__ void density_body(const DensArgs& a) {
  constexpr int TH = N < 64 ? 64 : N, NW = TH / 32;
  __shared__ double rho_s[N];
  __shared__ double vh_s[N];
  __shared__ FxTwiddles<N> tw_s;
  __shared__ cx buf[N];
  __shared__ int red[2 * NW];
  const int tid = threadIdx.x;
  const bool in = tid < N;
  tw_s.load(a.twfx);
  double2 v[1] = {make_double2(0.0, 0.0)}, sg[1] = {make_double2(0.0, 0.0)};
  if (in) {
    const int nch = dens_chunks(a.nk * a.u.nb);
    double s = a.part[tid];
#pragma unroll 4
    for (int ch = 1; ch < nch; ++ch) s += a.part[(size_t)ch * N + tid];
    rho_s[tid] = s;
    a.rho[tid] = s;
    v[0].x = s;
    if (a.mu != nullptr) {
      s = a.part_sig[tid];
#pragma unroll 4
      for (int ch = 1; ch < nch; ++ch) s += a.part_sig[(size_t)ch * N + tid];
      sg[0].x = s;
    }
  }
  int2 z = fx_block_size<1, NW>(v, red);
  if (a.mu != nullptr) {
    // Both potentials by one transform pair: vCG is real and even, so rho + i sigma
    // goes to vH[rho] + i vH[sigma].  Each has its own scale, whatever the size of mu.
    const Scale sr = fx_fft_scale(z, 2 * N);
    __syncthreads();
    const Scale ss = fx_fft_scale(fx_block_size<1, NW>(sg, red), 2 * N);
    if (in) buf[tid] = cx{fx_convert(v[0].x, sr), fx_convert(sg[0].x, ss)};
    fx_block_forward<N>(buf, tw_s);
    const double sig = sg[0].x;
    if (in) {
      const double f = a.vCG[tid] * (1.0 / N);
      v[0] = make_double2(f * (double)buf[tid].x, -f * (double)buf[tid].y);  // conjugate: backward next
    }
    z = fx_block_size<1, NW>(v, red);
    const Scale sb = fx_fft_scale(z, N);
    if (in) buf[tid] = cx{fx_convert(v[0].x, sb), fx_convert(v[0].y, sb)};
    fx_block_forward<N>(buf, tw_s);
    if (in) {
      a.vloc[tid] = Unscale{-(sb.k + sr.k + 6), sb.c != 0 && sr.c != 0}(buf[tid].x) + a.vion[tid];
      a.psi[tid] = -Unscale{-(sb.k + ss.k + 6), sb.c != 0 && ss.c != 0}(buf[tid].y);
      a.gvion[tid] += sig;
    }
    return;
  }
  const Scale s1 = fx_fft_scale(z, N);
  if (in) buf[tid] = cx{fx_convert(v[0].x, s1), 0};
  fx_block_forward<N>(buf, tw_s);
  if (in) {
    const Unscale u = fx_unscale(s1);
    const double f = a.vCG[tid] * (1.0 / N);
    v[0] = make_double2(f * u(buf[tid].x), -f * u(buf[tid].y));  // conjugate: backward next
  }
  z = fx_block_size<1, NW>(v, red);
  const Scale s2 = fx_fft_scale(z, N);
  if (in) buf[tid] = cx{fx_convert(v[0].x, s2), fx_convert(v[0].y, s2)};
  fx_block_forward<N>(buf, tw_s);
  if (in) vh_s[tid] = fx_unscale(s2)(buf[tid].x);
  __syncthreads();
  for (int ig = tid; ig < N; ig += blockDim.x) a.vloc[ig] = vh_s[ig] + a.vion[ig];
  if (a.scal != nullptr && tid < 64) {
    // Nele, Eion, EH: lane-strided partial sums, then a fixed shuffle tree; two
    // warps (one for the first two sums)
    const int lane = tid & 31;
    double x = 0.0, y = 0.0;
    if (tid < 32) {
      for (int ig = lane; ig < N; ig += 32) {
        x += rho_s[ig];
        y += a.vion[ig] * rho_s[ig];
      }
    } else {
      for (int ig = lane; ig < N; ig += 32) x += vh_s[ig] * rho_s[ig];
    }
    x = warp_sum(x);
    y = warp_sum(y);
    if (tid == 0) {
      a.scal[0] = x * a.dvcell;
      a.scal[1] = y * a.dvcell;
    } else if (tid == 32) {
      a.scal[2] = 0.5 * x * a.dvcell;
    }
  }
}

template <int N>
__global__ void __launch_bounds__(512) k_density(DensArgs a) { density_body<N>(a); }


// one CTA per run
template <int N>
__global__ void __launch_bounds__(512) k_density_batch(const DensArgs* __restrict__ args) {
  density_body<N>(args[blockIdx.x]);
}

// ---------------------------------------------------------------------------
// Fock exchange pair kernel (F:237-261).
//
// Work item = (output column (kr, ibr), chunk of source pairs (kc, ibc)).
// Each team streams its share of the chunk's pairs:
//   x = w(kr,ibr) * conj(u(kc,ibc));  X = FFT(x);  X *= -v(G+kx(kr)-kx(kc))/(NG NK);
//   x = IFFT(X);  acc += x * u(kc,ibc)
// with w, u, acc held in registers at the team's fixed FFT slot positions.
// Teams are reduced in a fixed order and the partial column is written to
// scratch[item]; the combine kernel sums the chunks in order.  No atomics,
// bitwise-reproducible.
// ---------------------------------------------------------------------------
template <int N>
__global__ void __launch_bounds__(kThreads) k_fock(FockArgs a) {
  using TM = Team<N>;
  constexpr int E = TM::E, T = TM::T, PW = TM::PER_WARP;
  constexpr int NWARP = kThreads / 32;
  constexpr int NTEAM = NWARP * PW;
  extern __shared__ double2 sm[];
  double2* tw_s = sm;                 // N
  double2* bufs = sm + N;             // NTEAM * N
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tl = lane % T, tiw = lane / T, team = warp * PW + tiw;
  double2* buf = bufs + team * N;
  for (int i = tid; i < N; i += kThreads) tw_s[i] = a.tw[i];
  __syncthreads();

  const int item = blockIdx.x;
  const int col = item / a.nchunks, chunk = item % a.nchunks;
  const int kr = col / a.w.nb, ibr = col % a.w.nb;
  const double2* wcol = a.w.p + (size_t)kr * a.w.kstride + (size_t)ibr * N;
  // w and u columns are re-read (L1/L2) instead of held in registers
  double2 acc[E];
#pragma unroll
  for (int e = 0; e < E; ++e) acc[e] = make_double2(0.0, 0.0);
  const int npairs = a.nk * a.nbocc;
  const int p0 = chunk * a.chunk;
  const int p1 = min(npairs, p0 + a.chunk);
  // warp-uniform trip count: every team of a warp runs the same rounds
  for (int base = p0 + warp * PW; base < p1; base += NTEAM) {
    const int p = base + tiw;
    const bool valid = p < p1;
    const int pp = valid ? p : p0;
    const int kc = pp / a.nbocc, ibc = pp % a.nbocc;
    const double2* ucol = a.u.p + (size_t)kc * a.u.kstride + (size_t)ibc * N;
    const double* kern = a.kern + (size_t)(kr - kc + a.nk - 1) * N;
    double2 x[E];
    fft_team_in<N, -1>(InConjProduct<N>{wcol, ucol, tl}, x, buf, tw_s, tl);
    fft_team_in<N, +1>(InScaled<N>{x, kern, tl}, x, buf, tw_s, tl);
    if (valid) {
#pragma unroll
      for (int e = 0; e < E; ++e) acc[e] = cfma(x[e], ucol[TM::pos(tl, e)], acc[e]);
    }
  }
  // fixed-order reduction over teams
#pragma unroll
  for (int e = 0; e < E; ++e) buf[TM::pos(tl, e)] = acc[e];
  __syncthreads();
  double2* dst = a.scratch + (size_t)item * N;
  for (int i = tid; i < N; i += kThreads) {
    double2 s = bufs[i];
    for (int t = 1; t < NTEAM; ++t) s = cadd(s, bufs[t * N + i]);
    dst[i] = s;
  }
}


// Exchange term of output column (ik, ib) at grid point q; false: none.
__device__ __forceinline__ bool exchange_at(const CombineArgs& a, int ik, int ib, int q, int N, double2* f) {
  if (ib < a.nbocc && (a.occ_ex.acc != nullptr || a.occ_ex.f != nullptr)) {
    *f = exchange_value(a.occ_ex, ik * a.nbocc + ib, q, N);
    return true;
  }
  if (a.row_ex.acc == nullptr && a.row_ex.dm == nullptr) return false;
  *f = exchange_value(a.row_ex, ik * (a.w.nb - a.row_b0) + (ib - a.row_b0), q, N);
  return true;
}

// ---------------------------------------------------------------------------
// Combine: kinetic (F:212-234) + local potential (F:199-203) + exchange, then
// the mode's epilogue (RK4 stages RT:166-170, observables F:94-119, F:165-183,
// F:289-318).  One CTA per output column.
//
// FP64 is slow here in both throughput and latency (one instruction per 64
// cycles and warp), so the transforms run in fixed point on the CTA's first
// team and the FP64 work is spread over all threads, a value or a few each.
// With FP64 transforms on one warp per column a launch took 26 us at NG = 64 and
// 43 us at NG = 128.
// ---------------------------------------------------------------------------
template <int N>
__device__ __forceinline__ void combine_body(const CombineArgs& a, const int c) {
  using CC = ColumnCta<N>;
  constexpr int TH = CC::TH, PER = CC::PER, NW = CC::NW;
  __shared__ FxTwiddles<N> tw_s;
  __shared__ cx buf[N];
  __shared__ int red[2 * NW];
  __shared__ double redd[NW];
  const int tid = threadIdx.x;
  const int ik = c / a.w.nb, ib = c % a.w.nb;
  const double2* wcol = a.w.p + (size_t)ik * a.w.kstride + (size_t)ib * N;
  const bool in = tid < N;
  double2 wv[PER];
#pragma unroll
  for (int p = 0; p < PER; ++p) wv[p] = in ? wcol[tid + TH * p] : make_double2(0.0, 0.0);
  // split == 2: the kinetic part was made by the split == 1 pass (beside the
  // exchange and the density); the potential, the exchange and the epilogue remain
  const bool post = a.split == 2;
  double2 kin[PER];
  if (!post && a.mode != CM_F) {
    const double A = afield_value(a.af);
    const double kAx = a.kx[ik] + A;
    const double kA2 = kAx * kAx;
    tw_s.load(a.twfx);
    int2 z = fx_block_size<PER, NW>(wv, red);
    const Scale s1 = fx_fft_scale(z, N);
    if (in) {
#pragma unroll
      for (int p = 0; p < PER; ++p) buf[tid + TH * p] = cx{fx_convert(wv[p].x, s1), fx_convert(wv[p].y, s1)};
    }
    fx_block_forward<N>(buf, tw_s);
    const Unscale u1 = fx_unscale(s1);
    if (a.mode == CM_OBS || a.obs) {
      // Ekin and Je of this column by Parseval on FFT(u):
      //   sum_x conj(u) IFFT(f * FFT(u)) = sum_G f(G) |FFT(u)(G)|^2
      const double Ao = a.obs ? afield_value(a.af_obs) : A;
      const double kAo = a.kx[ik] + Ao, kAo2 = kAo * kAo;
      double ek = 0.0, je = 0.0, fr = 0.0, fi = 0.0;
      if (in) {
#pragma unroll
        for (int p = 0; p < PER; ++p) {
          const int q = tid + TH * p;
          const double G = a.Gx[q];
          const double xr = u1(buf[q].x), xi = u1(buf[q].y);
          const double m2 = xr * xr + xi * xi;
          ek += 0.5 * (G * G + 2.0 * G * kAo + kAo2) * m2;
          je += (G + a.kx[ik] + Ao) * m2;
          double2 f;
          if (a.mode == CM_OBS && ib < a.nbocc && exchange_at(a, ik, ib, q, N, &f)) {
            fr += wv[p].x * f.x + wv[p].y * f.y;
            fi += wv[p].x * f.y - wv[p].y * f.x;
          }
        }
      }
      ek = block_sum<NW>(ek, redd) / (double)N;
      je = block_sum<NW>(je, redd) / (double)N;
      double* cb = a.colbuf + (size_t)c * 4;
      if (tid == 0) {
        cb[0] = ek;
        cb[1] = je;
      }
      if (a.mode == CM_OBS) {
        fr = block_sum<NW>(fr, redd);
        fi = block_sum<NW>(fi, redd);
        if (tid == 0) {
          cb[2] = fr;
          cb[3] = fi;
        }
        return;
      }
    }
    // kinetic energy in FP64, then back with a new scale
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int q = tid + TH * p;
      kin[p] = make_double2(0.0, 0.0);
      if (in) {
        const double G = a.Gx[q];
        const double m = 0.5 * (G * G + 2.0 * G * kAx + kA2) * (1.0 / N);
        kin[p] = make_double2(m * u1(buf[q].x), -m * u1(buf[q].y));  // conjugate: backward next
      }
    }
    z = fx_block_size<PER, NW>(kin, red);
    const Scale s2 = fx_fft_scale(z, N);
    if (in) {
#pragma unroll
      for (int p = 0; p < PER; ++p) buf[tid + TH * p] = cx{fx_convert(kin[p].x, s2), fx_convert(kin[p].y, s2)};
    }
    fx_block_forward<N>(buf, tw_s);
    const Unscale u2 = fx_unscale(s2);
    if (in) {
#pragma unroll
      for (int p = 0; p < PER; ++p) kin[p] = make_double2(u2(buf[tid + TH * p].x), -u2(buf[tid + TH * p].y));
    }
  }
  const size_t ocol = (size_t)ik * a.w.nb * N + (size_t)ib * N;  // [NK][NB][NG]
  if (a.split == 1) {
    if (in) {
#pragma unroll
      for (int p = 0; p < PER; ++p) {
        a.hpre[ocol + tid + TH * p] = kin[p];
      }
    }
    return;
  }
  // deferred exchange energy: <w|F> of occupied columns (stage 1 of an RK4 step)
  double exr = 0.0, exi = 0.0;
  bool bad = false;
  double2 next[PER];
  const double dt6 = a.dt / 6.0;
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    next[p] = make_double2(0.0, 0.0);
    if (!in) continue;
    const int q = tid + TH * p;
    double2 h;
    if (a.mode == CM_T) {
      h = kin[p];
    } else {
      if (a.mode == CM_F) h = make_double2(0.0, 0.0);
      else {
        const double v = a.vloc[q];
        const double2 t = post ? a.hpre[ocol + q] : kin[p];
        h = make_double2(t.x + v * wv[p].x, t.y + v * wv[p].y);
      }
      double2 f;
      if (exchange_at(a, ik, ib, q, N, &f)) {
        if (a.ex_cols) {
          exr += wv[p].x * f.x + wv[p].y * f.y;
          exi += wv[p].x * f.y - wv[p].y * f.x;
        }
        h = cadd(h, f);
      }
    }
    if (a.mode == CM_H || a.mode == CM_F || a.mode == CM_T) {
      a.out.p[(size_t)ik * a.out.kstride + (size_t)ib * N + q] = h;
      bad |= !(isfinite(h.x) && isfinite(h.y));
      continue;
    }
    // RK4: k = -i h
    const double2 k = make_double2(h.y, -h.x);
    const size_t o = ocol + q;
    const double2 u0 = a.u0[o];
    double2 nx;
    if (a.mode == CM_RK0 || a.mode == CM_RK1 || a.mode == CM_RK2) {
      a.kbuf[a.mode - CM_RK0][o] = k;
      const double cdt = (a.mode == CM_RK2) ? a.dt : 0.5 * a.dt;
      nx = make_double2(u0.x + cdt * k.x, u0.y + cdt * k.y);
      a.out.p[(size_t)ik * a.out.kstride + (size_t)ib * N + q] = nx;
    } else {  // CM_RK3: ubk + (k1 + 2 k2 + 2 k3 + k4) * dt / 6
      const double2 k0 = a.kbuf[0][o], k1 = a.kbuf[1][o], k2 = a.kbuf[2][o];
      double sx = k0.x + 2.0 * k1.x, sy = k0.y + 2.0 * k1.y;
      sx = sx + 2.0 * k2.x;
      sy = sy + 2.0 * k2.y;
      sx = sx + k.x;
      sy = sy + k.y;
      nx = make_double2(fma(sx, dt6, u0.x), fma(sy, dt6, u0.y));
      a.u0[o] = nx;
    }
    next[p] = nx;
    bad |= !(isfinite(nx.x) && isfinite(nx.y));
  }
  if (a.advance != nullptr && c == 0 && tid == 0) *a.advance = *a.advance + 1;
  if (a.sizes != nullptr && ib < a.nbocc) {
    const int2 z = fx_block_size<PER, NW>(next, red);
    if (tid == 0) a.sizes[ik * a.nbocc + ib] = z;
  }
  if (a.ex_cols) {
    exr = block_sum<NW>(exr, redd);
    exi = block_sum<NW>(exi, redd);
    if (tid == 0) {
      a.colbuf[(size_t)c * 4 + 2] = exr;
      a.colbuf[(size_t)c * 4 + 3] = exi;
    }
  }
  if (bad && a.nonfinite) *a.nonfinite = 1;
}

template <int N>
__global__ void __launch_bounds__(ColumnCta<N>::TH) k_combine(CombineArgs a) {
  combine_body<N>(a, blockIdx.x);
}

// column prefix: pre[r] = sum over earlier runs of their columns
template <int N>
__global__ void __launch_bounds__(ColumnCta<N>::TH) k_combine_batch(const CombineArgs* __restrict__ args,
                                                                    const int* __restrict__ pre, int nruns) {
  const int r = find_run(pre, nruns, blockIdx.x);
  combine_body<N>(args[r], blockIdx.x - pre[r]);
}

// ---------------------------------------------------------------------------
// Observable reduction (F:74-91, F:165-183, F:289-318) in reference order.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void obs_reduce_body(const ObsReduceArgs& a, int lane) {
  if (a.advance == 3 && *a.it == 0) return;
  double ekin = 0.0, jre = 0.0, exr = 0.0;
  const int ncol = a.nk * a.nb;
  for (int c = lane; c < ncol; c += 32) {
    const int ib = c % a.nb;
    const double occ = ib < a.nbocc ? a.occ : 0.0;
    const double* cb = a.colbuf + (size_t)c * 4;
    ekin += occ * cb[0] * a.dvcell;
    jre += occ * cb[1];
    if (ib < a.nbocc && a.hf) exr += occ * cb[2] * a.dvcell;
  }
  ekin = warp_sum(ekin);
  jre = warp_sum(jre);
  exr = warp_sum(exr);
  if (lane != 0) return;
  const double Ex = a.hf ? 0.5 * exr : 0.0;
  const double Eion = a.scal[1], EH = a.scal[2], Nele = a.scal[0];
  const double Etot = ekin + Eion + EH + Ex;
  const double Je = -(jre * a.dvcell / a.vcell);
  a.out[0] = Etot;
  a.out[1] = ekin;
  a.out[2] = Eion;
  a.out[3] = EH;
  a.out[4] = Ex;
  a.out[5] = Je;
  a.out[6] = Nele;
  if (a.advance) {
    const int it = a.advance == 3 ? *a.it - 1 : *a.it;
    if (a.series_E) a.series_E[it] = Etot;
    if (a.series_J) a.series_J[it] = Je;
    if (a.series_N) a.series_N[it] = Nele;
    if (!(isfinite(Etot) && isfinite(Je) && isfinite(Nele)) && a.nonfinite) *a.nonfinite = 1;
    if (a.advance == 1) *a.it = it + 1;
  }
}

__global__ void k_obs_reduce(ObsReduceArgs a) {
  if (blockIdx.x == 0 && threadIdx.x < 32) obs_reduce_body(a, threadIdx.x);
}

// one warp per run; the step counter is advanced by k_step_advance afterwards
__global__ void k_obs_reduce_batch(const ObsReduceArgs* __restrict__ args, int nruns) {
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (r < nruns) obs_reduce_body(args[r], threadIdx.x & 31);
}

__global__ void k_step_advance(int* it) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *it = *it + 1;
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
template <int N>
static cudaError_t fock_impl(const FockArgs& a, int ncols, cudaStream_t s) {
  constexpr int NTEAM = (kThreads / 32) * Team<N>::PER_WARP;
  const size_t smem = sizeof(double2) * (size_t)N * (1 + NTEAM);
  static_assert(sizeof(double2) * N * (1 + NTEAM) <= 48 * 1024, "fits the default dynamic smem limit");
  const int items = ncols * a.nchunks;
  if (items == 0) return cudaSuccess;
  k_fock<N><<<items, kThreads, smem, s>>>(a);
  return cudaGetLastError();
}

template <int N>
static constexpr int sym_teams() { return (kThreads / 32) * Team<N>::PER_WARP; }

template <int N>
static size_t sym_smem() { return sizeof(double2) * (size_t)N * (1 + 2 * sym_teams<N>()); }

// threads and dynamic shared memory of a symmetric-exchange CTA with tile size S
template <int N>
static void sym_launch_shape(int S, int* threads, size_t* smem) {
  constexpr int PW = Team<N>::PER_WARP;
  const int warps = (S + PW - 1) / PW;
  *threads = 32 * warps;
  *smem = sizeof(double2) * (size_t)N * (1 + warps * PW + S);
}

template <int N>
static cudaError_t combine_impl(const CombineArgs& a, int ncols, cudaStream_t s) {
  if (ncols == 0) return cudaSuccess;
  k_combine<N><<<ncols, ColumnCta<N>::TH, 0, s>>>(a);
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

cudaError_t launch_density(int NG, const DensArgs& a, cudaStream_t s) {
  k_dens_partial<<<dim3(dens_chunks(a.nk * a.u.nb), (NG + 63) / 64), 64 * kDensSub, 0, s>>>(a, NG);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
#define CALL(n) (k_density<n><<<1, (n) < 64 ? 64 : (n), 0, s>>>(a), cudaGetLastError())
  MATTOHF_DISPATCH(NG, CALL)
#undef CALL
}

cudaError_t launch_fock(int NG, const FockArgs& a, int ncols, cudaStream_t s) {
#define CALL(n) fock_impl<n>(a, ncols, s)
  MATTOHF_DISPATCH(NG, CALL)
#undef CALL
}

// Largest tile size (a power of two up to the teams of a full CTA) that still
// yields enough tile pairs to occupy every one of the device's nsm SMs four
// times; small systems fall back to small tiles so their few pairs spread over
// many SMs.
int choose_sym_tile(int NG, int M, int nsm) {
  int S = fock_sym_teams(NG);
  const int want = 4 * (nsm > 0 ? nsm : 1);
  while (S > 1) {
    const int T = (M + S - 1) / S;
    if (T * (T + 1) / 2 >= want) break;
    S >>= 1;
  }
  return S;
}

cudaError_t sym_launch_params(int NG, int S, int* threads, size_t* smem) {
  switch (NG) {
    case 16: sym_launch_shape<16>(S, threads, smem); break;
    case 32: sym_launch_shape<32>(S, threads, smem); break;
    case 64: sym_launch_shape<64>(S, threads, smem); break;
    case 128: sym_launch_shape<128>(S, threads, smem); break;
    case 256: sym_launch_shape<256>(S, threads, smem); break;
    case 512: sym_launch_shape<512>(S, threads, smem); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaSuccess;
}

int fock_sym_teams(int NG) {
  switch (NG) {
    case 16: return sym_teams<16>();
    case 32: return sym_teams<32>();
    case 64: return sym_teams<64>();
    case 128: return sym_teams<128>();
    case 256: return sym_teams<256>();
    case 512: return sym_teams<512>();
    default: return 0;
  }
}

cudaError_t launch_combine(int NG, const CombineArgs& a, int ncols, cudaStream_t s) {
#define CALL(n) combine_impl<n>(a, ncols, s)
  MATTOHF_DISPATCH(NG, CALL)
#undef CALL
}

// ---- batched launchers (many independent runs per launch) ----
cudaError_t launch_density_batch(int NG, const DensArgs* d_args, int nruns, cudaStream_t s) {
  k_dens_partial_batch<<<dim3(kDensChunks, (NG + 63) / 64, nruns), 64 * kDensSub, 0, s>>>(d_args, NG);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
#define CALL(n) (k_density_batch<n><<<nruns, (n) < 64 ? 64 : (n), 0, s>>>(d_args), cudaGetLastError())
  MATTOHF_DISPATCH(NG, CALL)
#undef CALL
}

cudaError_t launch_combine_batch(int NG, const CombineArgs* d_args, const int* d_col_pre, int nruns,
                                 int total_cols, cudaStream_t s) {
  if (total_cols <= 0) return cudaSuccess;
#define CALL(n) (k_combine_batch<n><<<total_cols, ColumnCta<n>::TH, 0, s>>>(d_args, d_col_pre, nruns), cudaGetLastError())
  MATTOHF_DISPATCH(NG, CALL)
#undef CALL
}

cudaError_t launch_obs_reduce_batch(const ObsReduceArgs* d_args, int nruns, cudaStream_t s) {
  k_obs_reduce_batch<<<(nruns + 3) / 4, 128, 0, s>>>(d_args, nruns);
  return cudaGetLastError();
}

cudaError_t launch_step_advance(int* it, cudaStream_t s) {
  k_step_advance<<<1, 32, 0, s>>>(it);
  return cudaGetLastError();
}

cudaError_t launch_obs_reduce(const ObsReduceArgs& a, cudaStream_t s) {
  k_obs_reduce<<<1, 32, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace mattohf
