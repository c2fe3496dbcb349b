// The parts of the fused fixed-point RK4 stages (k_small_fx.cu) outside the transforms:
// the observables, the staged copies for the adjoint, the exchange of partial results
// within a column's cluster and the RK4 update.  k_small.cu has the same steps written
// out in its kernel: with these functions its stages were 1.2 % slower (50 steps at
// 64 / 8 / 2: 1.005 against 0.993 of the same earlier build's time), a difference of
// register allocation.
#pragma once
#include <cooperative_groups.h>

#include "internal.h"

namespace mattohf {

constexpr int kSmallThreads = 256;
constexpr int kSmallWarps = kSmallThreads / 32;
// doubles that a CTA takes for its points' partials
template <int N> constexpr int kSmallRecvF = 2 * N + 2 * kSmallMaxCtas;

__device__ __forceinline__ double small_warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The global last CTA of an observable stage: the observables of the stage
// input (mode 0 with a previous step, mode 4) from the column buffer and this
// CTA's own density.  Run by one warp.
static __device__ void small_finalize(const SmallStageArgs& a, const double* rho_s, const double* vh_s, int N) {
  const int lane = threadIdx.x & 31;
  const int idx = *a.it - 1;
  if (idx < 0) return;
  const int ncol = a.nk * a.nb;
  double ekin = 0.0, jre = 0.0, exr = 0.0;
  for (int c = lane; c < ncol; c += 32) {
    const int ib = c % a.nb;
    const double occ = ib < a.nbocc ? a.occ : 0.0;
    const double* cb = a.colbuf + (size_t)c * 4;
    ekin += occ * __ldcg(cb) * a.dvcell;
    jre += occ * __ldcg(cb + 1);
    if (ib < a.nbocc) exr += occ * __ldcg(cb + 2) * a.dvcell;
  }
  double sn = 0.0, si = 0.0, sh = 0.0;
  for (int ig = lane; ig < N; ig += 32) {
    sn += rho_s[ig];
    si += a.vion[ig] * rho_s[ig];
    sh += vh_s[ig] * rho_s[ig];
  }
  ekin = small_warp_sum(ekin);
  jre = small_warp_sum(jre);
  exr = small_warp_sum(exr);
  sn = small_warp_sum(sn);
  si = small_warp_sum(si);
  sh = small_warp_sum(sh);
  if (lane != 0) return;
  const double Nele = sn * a.dvcell, Eion = si * a.dvcell, EH = 0.5 * sh * a.dvcell;
  const double Ex = a.hf ? 0.5 * exr : 0.0;
  const double Etot = (ekin + Eion + EH) + Ex;
  const double Je = -(jre * a.dvcell / a.vcell);
  if (a.series_E) a.series_E[idx] = Etot;
  if (a.series_J) a.series_J[idx] = Je;
  if (a.series_N) a.series_N[idx] = Nele;
  if (a.out_obs) {
    a.out_obs[0] = Etot;
    a.out_obs[1] = ekin;
    a.out_obs[2] = Eion;
    a.out_obs[3] = EH;
    a.out_obs[4] = Ex;
    a.out_obs[5] = Je;
    a.out_obs[6] = Nele;
  }
  if (!(isfinite(Etot) && isfinite(Je) && isfinite(Nele)) && a.nonfinite) *a.nonfinite = 1;
}

// checkpoint of this step's state?
__device__ __forceinline__ bool small_ckpt_step(const SmallStageArgs& a) {
  if (!a.ckpt || a.mode != 0) return false;
  const int t = *a.it;
  return t == 0 || (t + a.ckpt_phase) % a.ckpt_every == 0;
}
// The adjoint's passes: this CTA's points of the stage input, staged in shared
// memory by an asynchronous copy now and written to the stage store (recompute) or
// to a checkpoint (stage 0 of the forward pass) once the first phase is done (no
// registers held, no latency exposed).
template <int N>
__device__ __forceinline__ void small_stage_in(const SmallStageArgs& a, const double2* wcol, double2* st_s) {
  if (!a.store && !small_ckpt_step(a)) return;
  const int per = (N + a.P - 1) / a.P, q = blockIdx.x % a.P * per + threadIdx.x;
  if (threadIdx.x < per && q < N) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(st_s + threadIdx.x);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(wcol + q) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
}

// The second half of a stage.  recv: recvF [P][2 per], recvV [N], recvK [2 N];
// wait(): completes the cluster barrier phase under way; partial(i): this CTA's
// exchange partial, real component i of the column; push(per, recvV, recvK): the
// first CTA's vH (to vh_s too) and T_A w to the owners of the points.
template <int N, bool ADJ, class Wait, class Partial, class Push>
__device__ __forceinline__ void small_finish(const SmallStageArgs& a, const double2* wcol, double* recv, const double2* st_s,
                                             const double* rho_s, const double* vh_s, Wait wait, Partial partial, Push push) {
  namespace cg = cooperative_groups;
  __shared__ int last_s;
  __shared__ double red_s[2][kSmallWarps];
  __shared__ double ex_s[kSmallMaxCtas][2];  // the first CTA: every CTA's share of <w|F>
  double *recvF = recv, *recvV = recvF + kSmallRecvF<N>, *recvK = recvV + N;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ncols = a.nk * a.nb, c = blockIdx.x / a.P, chunk = blockIdx.x % a.P;
  const bool occupied = c % a.nb < a.nbocc, obs = a.mode == 0 || a.mode == 4;
  // The epilogue runs one real component per lane: lane slot idx = 2 e + cc
  // takes component cc of h = T_A w + v w + F at this CTA's element e and
  // writes the other component, dd = 1 - cc, of k = -i h and of the stage
  // output (k.x = h.y, k.y = -h.x).  A warp issues at most one FP64
  // instruction per ~64 cycles, so halving each lane's chain halves the
  // epilogue's time.  These are its inputs that no other CTA writes.
  constexpr int EPI = (2 * N + kSmallThreads - 1) / kSmallThreads;  // lane slots per thread
  const int per = (N + a.P - 1) / a.P;
  const double cdt = a.mode == 2 ? a.dt : 0.5 * a.dt;
  double wc[EPI], vi[EPI], ud[EPI], ks[EPI];
  // stage 0 and the closing pass: the w factors of this thread's components
  // in the partial sum below (component i = 2 q + cc of every point)
  double wt[EPI][2];
#pragma unroll
  for (int r = 0; r < EPI; ++r) {
    wt[r][0] = wt[r][1] = 0.0;
    const int i = tid + r * kSmallThreads;
    if (obs && i < 2 * N) {
      const double* w2 = reinterpret_cast<const double*>(wcol + (i >> 1));
      wt[r][0] = w2[i & 1];
      wt[r][1] = (i & 1) ? w2[0] : -w2[1];
    }
  }
#pragma unroll
  for (int r = 0; r < EPI; ++r) {
    wc[r] = vi[r] = ud[r] = ks[r] = 0.0;
    const int idx = tid + r * kSmallThreads, e = idx >> 1, cc = idx & 1, dd = 1 - cc;
    const int q = chunk * per + e;
    if (e < per && q < N) {
      const double* w2 = reinterpret_cast<const double*>(wcol + q);
      wc[r] = w2[cc];
      if (a.mode != 4) {
        const size_t od = 2 * ((size_t)c * N + q) + dd;
        vi[r] = a.vion[q];
        ud[r] = reinterpret_cast<const double*>(a.u0)[od];
        if (a.mode == 3) {
          // k0 + 2 k1 + 2 k2, formed before the barrier (the order of
          // ubk + (k1 + 2 k2 + 2 k3 + k4) * dt / 6, RT:165-170, is kept)
          const double k0 = reinterpret_cast<const double*>(a.kbuf[0])[od];
          const double k1 = reinterpret_cast<const double*>(a.kbuf[1])[od];
          const double k2 = reinterpret_cast<const double*>(a.kbuf[2])[od];
          ks[r] = fma(2.0, k2, fma(2.0, k1, k0));
        }
      }
    }
  }
  __syncthreads();
  if (ADJ && (a.store || small_ckpt_step(a)) && tid < per && chunk * per + tid < N) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    const size_t elems = (size_t)ncols * N, o = (size_t)c * N + chunk * per + tid;
    const int t = *a.it;
    if (a.store) a.store[((size_t)(t - *a.seg0) * 4 + a.store_slot) * elems + o] = st_s[tid];
    if (small_ckpt_step(a)) a.ckpt[(size_t)((t + a.ckpt_phase) / a.ckpt_every) * elems + o] = st_s[tid];
  }
  // This CTA's partial (pair teams in order; a team past the CTA's pair count
  // holds none), one real component per thread, pushed into the shared memory
  // of the CTA that owns the point (distributed shared memory); the first CTA
  // also pushes vH and T_A w.  After the cluster barrier every CTA finds the
  // P partials of its points in its own shared memory and does h w and the
  // RK4 update for its share of the grid, with no remote reads.
  cg::cluster_group cluster = cg::this_cluster();
  wait();
  {
    // stage 0 and the closing pass: this CTA's share of <w|F> = sum over all
    // points of conj(w) F_chunk, one real component per thread (Re gets
    // w_cc F_cc, Im gets sg w_dd F_cc with sg = +1 for cc = 1, -1 for cc = 0)
    double exr = 0.0, exi = 0.0;
#pragma unroll
    for (int r = 0; r < EPI; ++r) {
      const int i = tid + r * kSmallThreads;
      if (i >= 2 * N) continue;
      const double f = partial(i);
      const int q = i >> 1, cc = i & 1, owner = q / per, e = q - owner * per;
      cluster.map_shared_rank(recvF, owner)[chunk * 2 * per + 2 * e + cc] = f;
      if (obs) {
        exr = fma(wt[r][0], f, exr);
        exi = fma(wt[r][1], f, exi);
      }
    }
    if (obs) {
      // warp tree, then warps in order, pushed to the first CTA's slot
      exr = small_warp_sum(exr);
      exi = small_warp_sum(exi);
      if (lane == 0) {
        red_s[0][warp] = exr;
        red_s[1][warp] = exi;
      }
      __syncthreads();
      if (tid == 0) {
        double sr = red_s[0][0], si = red_s[1][0];
        for (int w2 = 1; w2 < kSmallWarps; ++w2) {
          sr += red_s[0][w2];
          si += red_s[1][w2];
        }
        double* dst = cluster.map_shared_rank(&ex_s[0][0], 0) + 2 * chunk;
        dst[0] = sr;
        dst[1] = si;
      }
    }
    if (chunk == 0) push(per, recvV, recvK);
  }
  cluster.sync();
  if (obs && chunk == 0 && tid == 0 && occupied) {
    double sr = ex_s[0][0], si = ex_s[0][1];
    for (int r = 1; r < a.P; ++r) {
      sr += ex_s[r][0];
      si += ex_s[r][1];
    }
    a.colbuf[(size_t)c * 4 + 2] = sr;
    a.colbuf[(size_t)c * 4 + 3] = si;
  }
  bool bad = false;
  // F (the P partials in chunk order) and h, from this CTA's shared memory
  double hr[EPI];
#pragma unroll
  for (int r = 0; r < EPI; ++r) {
    hr[r] = 0.0;
    const int idx = tid + r * kSmallThreads, e = idx >> 1, cc = idx & 1;
    const int q = chunk * per + e;
    if (!(e < per && q < N)) continue;
    double f = recvF[2 * e + cc];
#pragma unroll
    for (int rr = 1; rr < kSmallMaxCtas; ++rr)
      if (rr < a.P) f += recvF[rr * 2 * per + 2 * e + cc];
    if (a.mode != 4) hr[r] = fma(recvV[e] + vi[r], wc[r], recvK[2 * e + cc]) + f;
  }
#pragma unroll
  for (int r = 0; r < EPI; ++r) {
    const int idx = tid + r * kSmallThreads, e = idx >> 1, cc = idx & 1, dd = 1 - cc;
    const int q = chunk * per + e;
    if (!(e < per && q < N)) continue;
    const double scdt = cc ? cdt : -cdt;  // k_dd = sg h_cc with sg = +1 (cc = 1) or -1 (cc = 0)
    if (a.mode != 4) {
      const double h = hr[r];
      const size_t od = 2 * ((size_t)c * N + q) + dd;
      double nx;
      if (a.mode < 3) {
        nx = fma(scdt, h, ud[r]);
        reinterpret_cast<double*>(a.kbuf[a.mode])[od] = cc ? h : -h;
        reinterpret_cast<double*>(a.out)[od] = nx;
      } else {
        const double kd = cc ? h : -h;
        nx = ud[r] + (ks[r] + kd) * a.dt / 6.0;
        reinterpret_cast<double*>(a.u0)[od] = nx;  // this component only, read above by this thread
      }
      bad = bad || !isfinite(nx);
    }
  }
  if (bad && a.nonfinite) *a.nonfinite = 1;
  // No CTA touches another's shared memory after the cluster barrier, so the
  // stage is done; in the closing pass the last column to finish
  // finalizes (nothing waits on another column)
  if (a.mode != 4 || chunk != 0) return;
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    const unsigned t = atomicAdd(a.ticket, 1u);
    last_s = (t == (unsigned)ncols - 1) ? 1 : 0;
  }
  __syncthreads();
  if (last_s && warp == 0) {
    __threadfence();
    small_finalize(a, rho_s, vh_s, N);
    if (lane == 0) *a.ticket = 0u;
  }
}


}  // namespace mattohf
