"""The work that users have this framework do, as cases that can be timed.

Every case goes through the package's public Python API (``Context``,
``Batch``, ``ShardedRun``) with host arrays, as a user's program does: the
state goes in, the call runs, observables and the new state come back.

Kinds of case
  rt       real-time propagation: set the orbitals, the initial observables,
           ``rk4_run``, read the orbitals back
  hpsi     one application of the Hamiltonian, h[u] w or h[u] u
  gs       ground-state SCF iterations from a given guess
  batch    an ensemble of uneven runs advanced together
  adjoint  objective and gradient of a propagation (field samples, ion potential)
  slice    a run split over ranks by k-point, here with its one rank

Orbitals are smooth Bloch orbitals (complex normal coefficients that decay with
the plane wave's kinetic energy, orthonormal per k-point); fields are pulses of
the strengths that the benchmark uses; time steps are the largest stable ones
up to a margin.  Only gauge-invariant results of the ground state are returned
(its orbitals are fixed up to phases and rotations; the residual of a Ritz pair
is a diagnostic that is left out, being mostly rounding once converged).
"""
import math

import numpy as np
import torch

from mattohf_gb300 import Batch, Context, RunConfig

# one ion at the cell's middle, two unequal ones, three equal ones
IONS = {
    1: dict(Zeff=[2.0], alpha=[1.0], Rion=[0.5], Kion=[1]),
    2: dict(Zeff=[1.5, 0.5], alpha=[1.0, 1.0], Rion=[0.25, 0.75], Kion=[1, 2]),
    3: dict(Zeff=[1.0], alpha=[1.0], Rion=[1 / 6, 0.5, 5 / 6], Kion=[1, 1, 1]),
}


def listed():
    return [
        # the configuration that also runs on a CPU: latency of one step counts
        {"name": "rt_small", "kind": "rt", "NG": 64, "NK": 8, "NB": 2, "NBocc": 2, "acell": 10.0, "ions": 1, "nt": 50},
        # the exchange-dominated run of the benchmark
        {"name": "rt_exchange", "kind": "rt", "NG": 256, "NK": 64, "NB": 4, "NBocc": 4, "acell": 10.0, "ions": 2, "nt": 4},
        # the largest single run: one step of the finest grid and k-mesh
        {"name": "rt_large", "kind": "rt", "NG": 512, "NK": 128, "NB": 8, "NBocc": 8, "acell": 12.0, "ions": 3, "nt": 1},
        # empty bands carried along, and a k-mesh that no tile divides
        {"name": "rt_empty_bands", "kind": "rt", "NG": 128, "NK": 13, "NB": 5, "NBocc": 3, "acell": 9.0, "ions": 2, "nt": 8},
        # a single small call, as from a host program's own loop
        {"name": "hpsi_tiny", "kind": "hpsi", "NG": 32, "NK": 4, "NB": 2, "NBocc": 2, "acell": 8.0, "ions": 1, "nbw": 0},
        # h[u] w on a block of other functions, as a Krylov solver asks for
        {"name": "hpsi_block", "kind": "hpsi", "NG": 256, "NK": 64, "NB": 4, "NBocc": 4, "acell": 10.0, "ions": 2, "nbw": 8},
        # the ground state of a small cell with an empty band
        {"name": "gs_small", "kind": "gs", "NG": 64, "NK": 12, "NB": 3, "NBocc": 2, "acell": 10.0, "ions": 1, "nscf": 3, "ncg": 2},
        # the ground state on a fine grid
        {"name": "gs_fine", "kind": "gs", "NG": 256, "NK": 32, "NB": 4, "NBocc": 4, "acell": 10.0, "ions": 2, "nscf": 2, "ncg": 2},
        # an ensemble of uneven runs (k-points, bands, lattice constants, pulses)
        {"name": "batch_uneven", "kind": "batch", "NG": 128, "runs": 24, "nkmax": 64, "nomax": 4, "nt": 3},
        # the differentiation workload's shape: a window of small steps and its gradient
        {"name": "adjoint_small", "kind": "adjoint", "NG": 128, "NK": 16, "NB": 2, "NBocc": 2, "acell": 10.0, "ions": 1, "nt": 24, "objective": "energy"},
        # the gradient of a run that fills the GPU
        {"name": "adjoint_fine", "kind": "adjoint", "NG": 256, "NK": 32, "NB": 4, "NBocc": 4, "acell": 10.0, "ions": 2, "nt": 3, "objective": "current"},
        # a rank of a split run: its rows of every apply, the axpys on torch tensors
        {"name": "slice_rank", "kind": "slice", "NG": 256, "NK": 32, "NB": 3, "NBocc": 3, "acell": 10.0, "ions": 2, "nt": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(["rt", "rt", "rt", "hpsi", "hpsi", "gs", "batch", "adjoint", "adjoint", "slice"])
        NG = rng.choice([16, 32, 64, 128, 256, 512])
        nocc = rng.randint(1, 8)
        extra = rng.choice([0, 0, 0, 1, 2]) if kind in ("rt", "hpsi", "gs", "slice") else 0
        c = {"kind": kind, "NG": NG, "NK": _log_int(rng, 2, 128), "NB": nocc + extra, "NBocc": nocc,
             "acell": round(rng.uniform(8.0, 14.0), 2), "ions": rng.choice([1, 2, 3])}
        if kind in ("rt", "slice"):
            c["nt"] = _log_int(rng, 1, 30)
        elif kind == "hpsi":
            c["nbw"] = rng.choice([0, 0, 1, 2, 5, 8, 16])
        elif kind == "gs":
            # every Krylov power amplifies rounding by the largest kinetic energy: fine grids take short blocks
            c["nscf"], c["ncg"] = rng.randint(1, 2 if NG > 64 else 3), rng.randint(2, 4) if NG <= 32 else 2
            if c["NB"] * c["ncg"] > NG // 2:
                continue
        elif kind == "adjoint":
            c["nt"], c["objective"] = _log_int(rng, 2, 30), rng.choice(["energy", "current"])
        else:
            c = {"kind": kind, "NG": rng.choice([32, 64, 128, 256]), "runs": _log_int(rng, 2, 48),
                 "nkmax": rng.choice([8, 16, 32, 64]), "nomax": rng.randint(1, 4), "nt": rng.randint(1, 4)}
        if "NB" in c and c["NB"] > NG // 4:
            continue
        if kind == "adjoint" and c["NBocc"] ** 2 * c["NK"] ** 2 * NG * c["nt"] > 2e8:
            continue
        if work(c)["flops"] <= most / 2:
            return c


def _runs(case):
    """The members of an ensemble: uneven, but the same for every seed."""
    r = np.random.default_rng([case["runs"], case["nkmax"], case["nomax"], case["NG"]])
    nks = [k for k in (8, 16, 32, 64) if k <= case["nkmax"]]
    return [dict(NG=case["NG"], NK=int(r.choice(nks)), NBocc=int(n), NB=int(n), acell=float(round(a, 3)), ions=1)
            for n, a in zip(r.integers(1, case["nomax"] + 1, case["runs"]), r.uniform(8.0, 14.0, case["runs"]))]


def _config(c):
    return RunConfig(acell=c["acell"], NG=c["NG"], NK=c["NK"], NB=c["NB"], NBocc=c["NBocc"], **IONS[c["ions"]])


def _orbitals(c, rng, nb):
    """Smooth Bloch orbitals [NK][nb][NG], orthonormal per k-point under the cell's weight."""
    NG = c["NG"]
    G = np.fft.fftfreq(NG, 1.0 / NG) * (2 * math.pi / c["acell"])
    z = rng.standard_normal((c["NK"], NG, nb)) + 1j * rng.standard_normal((c["NK"], NG, nb))
    z *= np.exp(-0.15 * G * G)[None, :, None]
    u = np.fft.ifft(z, axis=1)
    q, _ = np.linalg.qr(u)
    return np.ascontiguousarray(q.transpose(0, 2, 1)) * math.sqrt(NG / c["acell"])


def _field(c, rng, nt):
    """Pulse samples A, their averages with the previous sample, and the time step."""
    amp, w = math.exp(rng.uniform(math.log(0.02), math.log(0.2))), rng.uniform(0.03, 0.1)
    g = math.pi * (c["NG"] + 2) / c["acell"] + 0.2
    dt = 1.8 / (0.5 * g * g + 6.0)
    t = dt * np.arange(1, nt + 1)
    A = amp * np.sin(w * (t + 20.0)) + 1e-3 * rng.standard_normal(nt)
    return A, 0.5 * (A + np.concatenate([[0.0], A[:-1]])), dt


def _inputs(case, seed):
    """The numbers that a pass starts from, as host arrays."""
    rng = np.random.default_rng([seed, case["NG"]])
    if case["kind"] == "batch":
        runs = _runs(case)
        us = [_orbitals(c, rng, c["NB"]) for c in runs]
        f = [_field(c, rng, case["nt"]) for c in runs]
        return {"u": us, "A": np.stack([x[0] for x in f]), "Aave": np.stack([x[1] for x in f]), "dt": np.array([x[2] for x in f])}
    u = _orbitals(case, rng, case["NB"])
    if case["kind"] == "hpsi":
        return {"u": u, "w": _orbitals(case, rng, case["nbw"]) if case["nbw"] else None, "A": float(rng.uniform(-0.1, 0.1))}
    if case["kind"] == "gs":
        return {"u": u}
    A, Aave, dt = _field(case, rng, case["nt"])
    return {"u": u, "A": A, "Aave": Aave, "dt": dt}


def prepare(case, seed):
    s = dict(_inputs(case, seed), case=case)
    if case["kind"] == "batch":
        s["batch"] = Batch([_config(c) for c in _runs(case)])
    elif case["kind"] == "slice":
        from mattohf_gb300.sharded import DeviceBackend, ShardedRun
        cfg = _config(case)
        s["run"] = ShardedRun(cfg, DeviceBackend(cfg))
    else:
        s["ctx"] = Context(_config(case))
    return s


def run(s):
    case, u = s["case"], s["u"]
    kind = case["kind"]
    if kind == "batch":
        b = s["batch"]
        for r, ur in enumerate(u):
            b[r].set_orbitals(ur)
        E, J, N = b.rk4_run(s["A"], s["Aave"], s["dt"])
        return {"E": E, "J": J, "N": N, "u": [b[r].get_orbitals() for r in range(len(b))]}
    if kind == "slice":
        r = s["run"]
        r.set_orbitals(u)
        E, J, N = r.rk4_run(s["A"], s["Aave"], s["dt"])
        return {"E": E, "J": J, "N": N, "u": r.get_orbitals()}
    ctx = s["ctx"]
    if kind == "hpsi":
        return ctx.ubkwbk_hwbk(u, u if s["w"] is None else s["w"], s["A"])
    ctx.set_orbitals(u)
    if kind == "rt":
        o = ctx.observables(0.0)
        E, J, N = ctx.rk4_run(s["A"], s["Aave"], s["dt"])
        return {"start": [o["Etot"], o["Je"], o["Nele"]], "E": E, "J": J, "N": N, "u": ctx.get_orbitals()}
    if kind == "gs":
        r = ctx.GS_calculation(case["nscf"], case["ncg"])
        return {"Etot": r["Etot"], "Je": r["Je"], "dnsdiff": r["dnsdiff"], "eps": r["epsbk"],
                "dns": ctx.ubk_dns(ctx.get_orbitals())}
    L, dA, dv = ctx.adjoint(s["A"], s["dt"], case["objective"])
    return {"L": L, "dA": dA, "dv": dv, "u": ctx.get_orbitals()}


def _apply_flops(NG, NK, NBocc, nbw, same):
    """Flops of one exchange apply, each unordered pair once where both sides are the same orbitals."""
    fft, M = 5 * NG * math.log2(NG), NK * NBocc
    pairs = M * (M + 1) / 2 if same else 0
    other = M * NK * (nbw - NBocc if same else nbw)
    return (pairs + other) * (2 * fft + 24 * NG) + NK * nbw * (2 * fft + 20 * NG)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        each = [work(dict(c, kind="rt", nt=case["nt"])) for c in _runs(case)]
        return {"bytes": sum(e["bytes"] for e in each), "flops": sum(e["flops"] for e in each)}
    NG, NK, NB, no = case["NG"], case["NK"], case["NB"], case["NBocc"]
    state, own = 16 * NG * NK * NB, _apply_flops(NG, NK, no, NB, True)
    table = 8 * NG * (2 * NK - 1)
    if kind == "hpsi":
        nbw = case["nbw"]
        return {"bytes": state + table + 16 * NG * NK * ((nbw or NB) + nbw), "flops": _apply_flops(NG, NK, no, nbw, False) if nbw else own}
    if kind == "gs":
        # per iteration: the powers of the block, h on its basis, and two applies on the orbitals
        n = 2 * case["ncg"] - 1
        return {"bytes": 2 * state + table, "flops": case["nscf"] * (n * _apply_flops(NG, NK, no, NB, False) + 2 * own)}
    if kind == "adjoint":
        # forward, then twice the transforms for each stage's adjoint
        return {"bytes": 2 * state + table, "flops": (4 * case["nt"] + 1) * own + 8 * case["nt"] * own}
    if kind == "slice":  # a rank's rows against all orbitals, and the observables of each step
        return {"bytes": 2 * state + table, "flops": 5 * case["nt"] * _apply_flops(NG, NK, no, NB, False)}
    return {"bytes": 2 * state + table, "flops": (4 * case["nt"] + 2) * own}


class _Exact:
    """The equations in 64 bits with torch's own transforms."""

    def __init__(self, c):
        self.c, self.dev = c, "cuda" if torch.cuda.is_available() else "cpu"
        NG, NK, a = c["NG"], c["NK"], c["acell"]
        self.NG, self.NK, self.no, self.a = NG, NK, c["NBocc"], a
        self.dv = a / NG
        T = lambda x: torch.as_tensor(x, device=self.dev)  # noqa: E731
        m = np.concatenate([np.arange(NG // 2), np.arange(-(NG // 2), 0)])  # the self-aliased frequency counts as negative
        b = 2 * math.pi / a
        self.G, self.k = T(m * b), T((-0.5 + (2.0 * np.arange(1, NK + 1) - 1.0) / (2 * NK)) * b)
        # 2 dx sum of trapezoids of cos(q x)/sqrt(x^2+1) up to x = NK a: q is a multiple of 2 pi/(NK a), so the sum is a transform
        n, dx = 20 * NG * NK, a / float(NG) / 20.0
        trips = n - 2
        while float(trips) * dx < NK * a:
            trips += 1
        f = 1.0 / np.sqrt((np.arange(trips + 1) * dx) ** 2 + 1.0)
        f[0], f[-1] = 0.5 * f[0], 0.5 * f[-1]
        g = np.zeros(n)
        np.add.at(g, np.arange(trips + 1) % n, f)
        table = 2 * dx * np.fft.fft(g).real
        vG = table[(m * NK) % n]
        vG[0] = 0.0
        self.vG = T(vG)
        d = np.arange(NK)
        self.vq = T(-table[(m[None, None, :] * NK + d[:, None, None] - d[None, :, None]) % n] / (NG * NK))  # [kr][kc][G]
        ion, x = IONS[c["ions"]], np.arange(NG) / NG * a
        v = np.zeros(NG)
        for R, K in zip(ion["Rion"], ion["Kion"]):
            cells = np.arange(-4 * NK, 4 * NK + 1)
            v -= (ion["Zeff"][K - 1] / np.sqrt((x[:, None] - a * R - a * cells) ** 2 + ion["alpha"][K - 1] ** 2)).sum(axis=1)
        self.vion = T(v - v.max())

    def kinetic(self, w, A):
        t = 0.5 * (self.G[None, :] + self.k[:, None] + A) ** 2
        return torch.fft.ifft(t[:, None, :] * torch.fft.fft(w))

    def exchange(self, u, w):
        o = u[:, :self.no]
        step = max(1, (1 << 23) // (self.NK * self.no * w.shape[1] * self.NG))
        rows = []
        for k in range(0, self.NK, step):
            p = w[k:k + step, None, :, None, :] * o.conj()[None, :, None, :, :]
            V = torch.fft.ifft(self.vq[k:k + step, :, None, None, :] * torch.fft.fft(p), norm="forward")
            rows.append((V * o[None, :, None, :, :]).sum(dim=(1, 3)))
        return torch.cat(rows)

    def density(self, u):
        return (2.0 / self.NK) * (u[:, :self.no].real ** 2 + u[:, :self.no].imag ** 2).sum(dim=(0, 1))

    def hartree(self, rho):
        return torch.fft.ifft(self.vG * torch.fft.fft(rho.to(torch.complex128))).real

    def h(self, u, w, A, vion=None):
        v = self.hartree(self.density(u)) + (self.vion if vion is None else vion)
        return self.kinetic(w, A) + v * w + self.exchange(u, w)

    def energy(self, u, A, vion=None):
        rho, o = self.density(u), u[:, :self.no]
        e = (2.0 / self.NK) * (o.conj() * (self.kinetic(o, A) + 0.5 * self.exchange(u, o))).real.sum() * self.dv
        return e + ((0.5 * self.hartree(rho) + (self.vion if vion is None else vion)) * rho).sum() * self.dv

    def current(self, u, A):
        m = (self.G[None, :] + self.k[:, None] + A)[:, None, :]
        return -(2.0 / self.NK) * (m * torch.fft.fft(u[:, :self.no]).abs() ** 2).sum() / self.NG * self.dv / self.a

    def step(self, u, Aave, A, dt, vion=None):
        f = lambda x, a: -1j * self.h(x, x, a, vion)  # noqa: E731
        k1 = f(u, 2 * Aave - A)
        k2 = f(u + 0.5 * dt * k1, Aave)
        k3 = f(u + 0.5 * dt * k2, Aave)
        return u + (k1 + 2 * k2 + 2 * k3 + f(u + dt * k3, A)) * (dt / 6)

    def rt(self, u, A, Aave, dt):
        E, J, N = [], [], []
        for a, b in zip(A, Aave):
            u = self.step(u, float(b), float(a), float(dt))
            E.append(self.energy(u, float(a)).item())
            J.append(self.current(u, float(a)).item())
            N.append(self.density(u).sum().item() * self.dv)
        return np.array(E), np.array(J), np.array(N), u.cpu().numpy()

    def gs(self, u, nscf, ncg):
        NB, w = u.shape[1], math.sqrt(self.dv)
        orth = lambda x: torch.linalg.qr(x.transpose(1, 2))[0].transpose(1, 2) / w  # noqa: E731
        E, J, D, rho = [self.energy(u, 0.0).item()], [], [], self.density(u)
        for _ in range(nscf):
            u = orth(u)
            blocks = [u]
            for _ in range(ncg - 1):
                blocks.append(self.h(u, blocks[-1], 0.0))
            x = orth(torch.cat(blocks, dim=1))
            for ref, base in ((u, x), (None, None)):
                if base is None:
                    ref = base = u = orth(u)
                M = (base.conj() @ self.h(ref, base, 0.0).transpose(1, 2)) * self.dv
                C = torch.linalg.eigh(0.5 * (M + M.mH))[1][:, :, :NB]
                u = C.transpose(1, 2) @ base
            E.append(self.energy(u, 0.0).item())
            J.append(self.current(u, 0.0).item())
            new = 0.5 * (self.density(u) + rho)
            D.append((new - rho).abs().sum().item() / self.NG)
            rho = new
        hu = self.h(u, u, 0.0)
        eps = (u.conj() * hu).real.sum(dim=2) * self.dv
        return {"Etot": np.array(E), "Je": np.array(J), "dnsdiff": np.array(D), "eps": eps.cpu().numpy(),
                "dns": self.density(u).cpu().numpy()}

    def adjoint(self, u0, A, dt, objective):
        At = torch.tensor(A, device=self.dev, requires_grad=True)
        v = self.vion.clone().requires_grad_(True)
        u = u0
        for n in range(len(A)):
            u = self.step(u, 0.5 * (At[n] + (At[n - 1] if n else 0.0)), At[n], dt, v)
        L = self.energy(u, At[-1], v) - self.energy(u0, 0.0, v) if objective == "energy" else self.current(u, At[-1])
        L.backward()
        gv = torch.zeros_like(v) if v.grad is None else v.grad
        return {"L": L.item(), "dA": At.grad.cpu().numpy(), "dv": gv.cpu().numpy(), "u": u.detach().cpu().numpy()}


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        got = []
        for r, c in enumerate(_runs(case)):
            X = _Exact(c)
            got.append(X.rt(torch.as_tensor(s["u"][r], device=X.dev), s["A"][r], s["Aave"][r], s["dt"][r]))
        return {"E": np.stack([g[0] for g in got]), "J": np.stack([g[1] for g in got]), "N": np.stack([g[2] for g in got]),
                "u": [g[3] for g in got]}
    X = _Exact(case)
    u = torch.as_tensor(s["u"], device=X.dev)
    if kind == "hpsi":
        w = u if s["w"] is None else torch.as_tensor(s["w"], device=X.dev)
        return X.h(u, w, s["A"]).cpu().numpy()
    if kind == "gs":
        return X.gs(u, case["nscf"], case["ncg"])
    if kind == "adjoint":
        return X.adjoint(u, s["A"], s["dt"], case["objective"])
    start = [f.item() for f in (X.energy(u, 0.0), X.current(u, 0.0), X.density(u).sum() * X.dv)]
    E, J, N, u = X.rt(u, s["A"], s["Aave"], s["dt"])
    if kind == "rt":
        return {"start": start, "E": E, "J": J, "N": N, "u": u}
    return {"E": E, "J": J, "N": N, "u": u}
