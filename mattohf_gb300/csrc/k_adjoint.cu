// Adjoint (reverse-mode) kernels of the RK4 real-time loop.
//
// No counterpart in the reference: the gradient of the absorbed energy or of
// the final current with respect to every sample of the vector potential.
// For the RK4 right-hand side f(v) = -i h[v](a) v of src/RT_calculation.f90:166-169
// (h from src/Functions.f90:187-209) the transposed Jacobian, for the real
// inner product <x,y> = Re sum conj(x) y, is (all bands occupied)
//   J^T mu = i h[v](a) mu                                  kinetic, local, exchange at fixed v
//          + 2 occ vH[sigma] v,  sigma = sum Im(conj(mu) v)  Hartree response
//          + i sum_j conj(phi_ji) mu_j                      exchange: dependence through the source orbital
//          + i sum_j v_j (Phi_ij[mu_i conj(v_j)] - Phi~_ji[v_i conj(mu_j)])   (the i VF mu term folded in)
// with phi_ij = Phi_ij[v_i conj(v_j)] the pair potentials of the forward step.
// Phi~_ji, the transpose of dv_j -> Phi_ij[v_i conj(dv_j)], has the multiplier
// kern_ji(-G): that is kern_ij(G) (v is even) except at the self-aliased
// Nyquist index N/2, where it stays kern_ji.  So
//   Phi~_ji[f] = Phi_ij[f] + dk_ij Nyq(f) (-1)^m,  dk_ij = kern_ji[N/2] - kern_ij[N/2],
// Nyq(f) = sum_m (-1)^m f(m) the Nyquist coefficient of the forward transform.
// k_fock_adj_fx (k_fock_fx.cu) evaluates the two exchange sums over unordered occupied pairs
// with two transform pairs per pair (pair densities v_i conj(v_j) and
// mu_i conj(v_j) - v_i conj(mu_j)), using the same conjugate-plus-Nyquist
// relation as the forward symmetric kernel.
#include "column_fx.cuh"
#include "fft.cuh"
#include "internal.h"

namespace mattohf {

__device__ __forceinline__ double2 mul_i(double2 a) { return make_double2(-a.y, a.x); }

// Adjoint combine of one RK4 stage, one CTA per column (fixed-point transforms on
// the first team, FP64 spread over the threads, as combine_body of k_hpsi.cu):
//   lu   = i (T_a + vloc) mu + i fa + 2 occ psi v
//   g_a += sum_G (G+k+a) Im(conj(FFT mu) FFT v) / N     (field gradient partial)
//   lam_u += lu ; lam_prev += c_prev * lu               (RK4 stage bookkeeping)
template <int N>
__global__ void __launch_bounds__(ColumnCta<N>::TH) k_adj_combine(AdjCombineArgs a) {
  using CC = ColumnCta<N>;
  constexpr int TH = CC::TH, PER = CC::PER, NW = CC::NW;
  __shared__ FxTwiddles<N> tw_s;
  __shared__ cx buf[N];
  __shared__ int red[2 * NW];
  __shared__ double redd[NW];
  const int tid = threadIdx.x, c = blockIdx.x;
  const int ik = c / a.nb;
  const size_t o = (size_t)c * N;
  const bool in = tid < N;
  double2 mu[PER], v[PER], lu[PER];
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    const int q = tid + TH * p;
    mu[p] = in && a.split != 2 ? a.mu[o + q] : make_double2(0.0, 0.0);
    v[p] = in ? a.v[o + q] : make_double2(0.0, 0.0);
    lu[p] = in && a.split == 2 ? a.lpre[o + q] : make_double2(0.0, 0.0);
  }
  if (a.split != 2) {
    const double A = afield_value(a.af);
    const double kAx = a.kx[ik] + A, kA2 = kAx * kAx;
    tw_s.load(a.twfx);
    int2 z = fx_block_size<PER, NW>(v, red);
    const Scale sv = fx_fft_scale(z, N);
    if (in) {
#pragma unroll
      for (int p = 0; p < PER; ++p) buf[tid + TH * p] = cx{fx_convert(v[p].x, sv), fx_convert(v[p].y, sv)};
    }
    fx_block_forward<N>(buf, tw_s);
    cx vf[PER];
#pragma unroll
    for (int p = 0; p < PER; ++p) vf[p] = in ? buf[tid + TH * p] : cx{0, 0};
    z = fx_block_size<PER, NW>(mu, red);  // its barriers also separate the reads above from the writes below
    const Scale s1 = fx_fft_scale(z, N);
    if (in) {
#pragma unroll
      for (int p = 0; p < PER; ++p) buf[tid + TH * p] = cx{fx_convert(mu[p].x, s1), fx_convert(mu[p].y, s1)};
    }
    fx_block_forward<N>(buf, tw_s);
    const Unscale u1 = fx_unscale(s1), uv = fx_unscale(sv);
    double gp = 0.0;
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      if (!in) continue;
      const int q = tid + TH * p;
      const double G = a.Gx[q];
      const double mx = u1(buf[q].x), my = u1(buf[q].y);
      gp += (G + a.kx[ik] + A) * (mx * uv(vf[p].y) - my * uv(vf[p].x));
      const double m = 0.5 * (G * G + 2.0 * G * kAx + kA2) * (1.0 / N);
      lu[p] = make_double2(m * mx, -m * my);  // conjugate: backward next
    }
    gp = block_sum<NW>(gp, redd) / (double)N;
    if (tid == 0) a.gcol[c] = gp;
    z = fx_block_size<PER, NW>(lu, red);
    const Scale s2 = fx_fft_scale(z, N);
    if (in) {
#pragma unroll
      for (int p = 0; p < PER; ++p) buf[tid + TH * p] = cx{fx_convert(lu[p].x, s2), fx_convert(lu[p].y, s2)};
    }
    fx_block_forward<N>(buf, tw_s);
    const Unscale u2 = fx_unscale(s2);
    if (!in) return;
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int q = tid + TH * p;
      const double vl = a.vloc[q];
      lu[p] = mul_i(make_double2(vl * mu[p].x + u2(buf[q].x), vl * mu[p].y - u2(buf[q].y)));
      if (a.split == 1) a.lpre[o + q] = lu[p];
    }
    if (a.split == 1) return;
  }
  if (!in) return;
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    const int q = tid + TH * p;
    double2 l = lu[p];
    if (a.fa.acc != nullptr) l = cadd(l, mul_i(exchange_value(a.fa, c, q, N)));
    const double ps = 2.0 * a.occ * a.psi[q];
    l = make_double2(fma(ps, v[p].x, l.x), fma(ps, v[p].y, l.y));
    a.lam_u[o + q] = cadd(a.lam_u[o + q], l);
    if (a.lam_prev) {
      const double2 lp = a.lam_prev[o + q];
      a.lam_prev[o + q] = make_double2(fma(a.cprev, l.x, lp.x), fma(a.cprev, l.y, lp.y));
    }
  }
}

// Sum of the per-column field-gradient partials into g[slot] (one warp, fixed order).
__global__ void k_adj_gsum(const double* __restrict__ gcol, int ncols, double* g, const int* n, int s) {
  double acc = 0.0;
  for (int i = threadIdx.x; i < ncols; i += 32) acc += gcol[i];
  acc = warp_sum(acc);
  if (threadIdx.x == 0) g[(size_t)(*n) * 4 + s] = acc;
}

// lam_k[s] = w_s lam (w = dt/6, dt/3, dt/3, dt/6); lam_u = lam.
__global__ void k_adj_init(const double2* __restrict__ lam, double2* lam_u, double2* k0, double2* k1,
                           double2* k2, double2* k3, double dt, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double2 l = lam[i];
  const double w6 = dt / 6.0, w3 = dt / 3.0;
  lam_u[i] = l;
  k0[i] = make_double2(w6 * l.x, w6 * l.y);
  k1[i] = make_double2(w3 * l.x, w3 * l.y);
  k2[i] = make_double2(w3 * l.x, w3 * l.y);
  k3[i] = make_double2(w6 * l.x, w6 * l.y);
}

// dst = store[(n - seg0) * 4 + slot]  (or the reverse with `to_store`)
__global__ void k_stage_copy(double2* dst, const double2* src, double2* store, const int* n,
                             const int* seg0, int slot, size_t elems, int to_store) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= elems) return;
  const size_t base = ((size_t)(*n - *seg0) * 4 + slot) * elems;
  if (to_store) store[base + i] = src[i];
  else dst[i] = store[base + i];
}

// checkpoint u every `every` steps: ckpt[it / every] = u when it % every == 0
// Checkpoint j holds the state at the start of segment j; segments start at
// step 0 and at every t with (t + phase) % every == 0.
__global__ void k_checkpoint(double2* ckpt, const double2* u, const int* it, int every, int phase, size_t elems) {
  const int t = *it;
  if (t != 0 && (t + phase) % every != 0) return;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < elems) ckpt[(size_t)((t + phase) / every) * elems + i] = u[i];
}

__global__ void k_counter_add(int* p, int d) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *p += d;
}

// out = scale * P_A u, P_A = IFFT((G+k+A) FFT(.)/N)  (the operator of ubk_Je, F:306-310)
template <int N>
__global__ void __launch_bounds__(kThreads) k_velocity(const double2* __restrict__ u, double2* out,
                                                       const double2* __restrict__ tw,
                                                       const double* __restrict__ Gx,
                                                       const double* __restrict__ kx, int nb, double A,
                                                       double scale, int ncols) {
  using TM = Team<N>;
  constexpr int E = TM::E, T = TM::T, PW = TM::PER_WARP;
  constexpr int NTEAM = (kThreads / 32) * PW;
  __shared__ double2 tw_s[N];
  __shared__ double2 bufs[NTEAM][N];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tl = lane % T, team = warp * PW + lane / T;
  for (int i = tid; i < N; i += kThreads) tw_s[i] = tw[i];
  __syncthreads();
  const int col0 = (blockIdx.x * (kThreads / 32) + warp) * PW;
  if (col0 >= ncols) return;
  const int col = col0 + lane / T;
  const bool valid = col < ncols;
  const int c = valid ? col : col0;
  const int ik = c / nb;
  double2 x[E];
#pragma unroll
  for (int e = 0; e < E; ++e) x[e] = u[(size_t)c * N + TM::pos(tl, e)];
  fft_team<N, -1>(x, bufs[team], tw_s, tl);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const double g = Gx[TM::pos(tl, e)] + kx[ik] + A;
    x[e] = make_double2(g * (x[e].x / (double)N), g * (x[e].y / (double)N));
  }
  fft_team<N, +1>(x, bufs[team], tw_s, tl);
  if (!valid) return;
#pragma unroll
  for (int e = 0; e < E; ++e)
    out[(size_t)c * N + TM::pos(tl, e)] = make_double2(scale * x[e].x, scale * x[e].y);
}

__global__ void k_scale2(double2* x, double s, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] = make_double2(s * x[i].x, s * x[i].y);
}

// ---------------------------------------------------------------------------
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

template <int N>
static cudaError_t adj_combine_impl(const AdjCombineArgs& a, int ncols, cudaStream_t s) {
  k_adj_combine<N><<<ncols, ColumnCta<N>::TH, 0, s>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || a.split == 2) return e;  // the field-gradient partials come from the other passes
  k_adj_gsum<<<1, 32, 0, s>>>(a.gcol, ncols, a.gstage, a.n, a.slot);
  return cudaGetLastError();
}

cudaError_t launch_adj_combine(int NG, const AdjCombineArgs& a, int ncols, cudaStream_t s) {
#define CALL(n) adj_combine_impl<n>(a, ncols, s)
  MATTOHF_DISPATCH(NG, CALL)
#undef CALL
}

cudaError_t launch_adj_init(const double2* lam, double2* lam_u, double2* const* lamk, double dt, size_t n,
                            cudaStream_t s) {
  k_adj_init<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(lam, lam_u, lamk[0], lamk[1], lamk[2], lamk[3], dt, n);
  return cudaGetLastError();
}

cudaError_t launch_stage_copy(double2* dst, const double2* src, double2* store, const int* n, const int* seg0,
                              int slot, size_t elems, int to_store, cudaStream_t s) {
  k_stage_copy<<<(unsigned)((elems + 255) / 256), 256, 0, s>>>(dst, src, store, n, seg0, slot, elems, to_store);
  return cudaGetLastError();
}

cudaError_t launch_checkpoint(double2* ckpt, const double2* u, const int* it, int every, int phase, size_t elems,
                              cudaStream_t s) {
  k_checkpoint<<<(unsigned)((elems + 255) / 256), 256, 0, s>>>(ckpt, u, it, every, phase, elems);
  return cudaGetLastError();
}

cudaError_t launch_counter_add(int* p, int d, cudaStream_t s) {
  k_counter_add<<<1, 32, 0, s>>>(p, d);
  return cudaGetLastError();
}

template <int N>
static cudaError_t velocity_impl(const double2* u, double2* out, const double2* tw, const double* Gx,
                                 const double* kx, int nb, double A, double scale, int ncols, cudaStream_t s) {
  constexpr int PER_CTA = (kThreads / 32) * Team<N>::PER_WARP;
  k_velocity<N><<<(ncols + PER_CTA - 1) / PER_CTA, kThreads, 0, s>>>(u, out, tw, Gx, kx, nb, A, scale, ncols);
  return cudaGetLastError();
}

cudaError_t launch_velocity(int NG, const double2* u, double2* out, const double2* tw, const double* Gx,
                            const double* kx, int nb, double A, double scale, int ncols, cudaStream_t s) {
#define CALL(n) velocity_impl<n>(u, out, tw, Gx, kx, nb, A, scale, ncols, s)
  MATTOHF_DISPATCH(NG, CALL)
#undef CALL
}

cudaError_t launch_scale2(double2* x, double sc, size_t n, cudaStream_t s) {
  k_scale2<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(x, sc, n);
  return cudaGetLastError();
}

// Nyquist term of the exchange-energy gradient.  Ex = 1/2 occ dvcell
// sum_ij <p_ij, Phi_ij p_ij>, p_ij = u_i conj(u_j) (src/Functions.f90:165-183).
// Varying the conj(u_j) factor brings in conj(Phi_ij[p_ij]), which equals
// Phi_ji[p_ji] except at the self-aliased Nyquist index; so the gradient is
// 2 occ dvcell h[u] u plus, for column i,
//   g_i += sc sum_j (kern_ji - kern_ij)[N/2] Nyq(p_ij) (-1)^m u_j,
// Nyq(p) = sum_m (-1)^m p(m), sc = occ dvcell.  One CTA per column i, one orbital j
// per warp at a time, so that eight chains of FP64 run side by side (with all warps on
// one j, a reduction over the CTA each, 112 us at NG = 128, NK = 16, 2 bands, now 46,
// bound by the SM's FP64 rate; an energy gradient at 256 / 32 / 4 3.12 -> 2.81 ms);
// the warps' sums are added in order.
constexpr int kNyqThreads = 256;
__global__ void __launch_bounds__(kNyqThreads) k_energy_grad_nyquist(const double2* __restrict__ u, double2* g,
                                                                      const double* __restrict__ kern, int N,
                                                                      int nk, int nb, double sc) {
  constexpr int kMaxPer = 512 / 32;    // N <= 512
  __shared__ double2 s_s[512], sum_s[512];
  const int i = blockIdx.x, ki = i / nb;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const double2* ui = u + (size_t)i * N;
  const int M = nk * nb;
  for (int m = tid; m < N; m += kNyqThreads) {
    const double sg = (m & 1) ? -1.0 : 1.0;
    s_s[m] = make_double2(sg * ui[m].x, sg * ui[m].y);
    sum_s[m] = make_double2(0.0, 0.0);
  }
  __syncthreads();
  double2 acc[kMaxPer];
#pragma unroll
  for (int r = 0; r < kMaxPer; ++r) acc[r] = make_double2(0.0, 0.0);
  for (int j = warp; j < M; j += kNyqThreads / 32) {
    const int kj = j / nb;
    if (kj == ki) continue;   // the two multipliers coincide
    const double d = kern[(size_t)(kj - ki + nk - 1) * N + N / 2] - kern[(size_t)(ki - kj + nk - 1) * N + N / 2];
    const double2* uj = u + (size_t)j * N;
    double px = 0.0, py = 0.0;
#pragma unroll
    for (int r = 0; r < kMaxPer; ++r) {
      const int m = lane + 32 * r;
      if (m < N) {
        const double2 z = uj[m], w = s_s[m];
        px = fma(w.x, z.x, fma(w.y, z.y, px));
        py = fma(w.y, z.x, fma(-w.x, z.y, py));
      }
    }
    px = warp_sum(px);
    py = warp_sum(py);
    const double2 f = make_double2(sc * d * px, sc * d * py);
#pragma unroll
    for (int r = 0; r < kMaxPer; ++r) {
      const int m = lane + 32 * r;
      if (m < N) acc[r] = cfma(f, uj[m], acc[r]);
    }
  }
  for (int w = 0; w < kNyqThreads / 32; ++w) {
    if (warp == w) {
#pragma unroll
      for (int r = 0; r < kMaxPer; ++r) {
        const int m = lane + 32 * r;
        if (m < N) sum_s[m] = cadd(sum_s[m], acc[r]);
      }
    }
    __syncthreads();
  }
  double2* gi = g + (size_t)i * N;
  for (int m = tid; m < N; m += kNyqThreads) {
    const double sg = (m & 1) ? -1.0 : 1.0;
    gi[m] = make_double2(fma(sg, sum_s[m].x, gi[m].x), fma(sg, sum_s[m].y, gi[m].y));
  }
}

cudaError_t launch_energy_grad_nyquist(const double2* u, double2* g, const double* kern, int NG, int nk, int nb,
                                       double sc, cudaStream_t s) {
  if (NG > 512) return cudaErrorInvalidValue;
  k_energy_grad_nyquist<<<nk * nb, kNyqThreads, 0, s>>>(u, g, kern, NG, nk, nb, sc);
  return cudaGetLastError();
}

}  // namespace mattohf

namespace mattohf {

// Taylor-propagator update (RT:86-88, RT:110-117): w = -i c (h0 [+ h1]) / iorder ; acc += w
__global__ void k_te_update(double2* __restrict__ w, const double2* __restrict__ h0,
                            const double2* __restrict__ h1, double c, double iorder,
                            double2* __restrict__ acc, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double2 s = h0[i];
  if (h1) s = make_double2(s.x + h1[i].x, s.y + h1[i].y);
  const double2 v = make_double2((c * s.y) / iorder, (-c * s.x) / iorder);
  w[i] = v;
  const double2 a = acc[i];
  acc[i] = make_double2(a.x + v.x, a.y + v.y);
}

// out = 0.5 * (a + b)
__global__ void k_half_sum(double2* __restrict__ out, const double2* __restrict__ a,
                           const double2* __restrict__ b, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = make_double2(0.5 * (a[i].x + b[i].x), 0.5 * (a[i].y + b[i].y));
}

cudaError_t launch_te_update(double2* w, const double2* h0, const double2* h1, double c, double iorder,
                             double2* acc, size_t n, cudaStream_t s) {
  k_te_update<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(w, h0, h1, c, iorder, acc, n);
  return cudaGetLastError();
}

cudaError_t launch_half_sum(double2* out, const double2* a, const double2* b, size_t n, cudaStream_t s) {
  k_half_sum<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(out, a, b, n);
  return cudaGetLastError();
}

}  // namespace mattohf
