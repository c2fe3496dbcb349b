"""The fixed-point exchange and column transforms against extended precision (needs a GB300)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
L, CL = np.longdouble, np.clongdouble


def _cfg(NG, NK, nb, nocc=None):
    from mattohf_gb300 import RunConfig
    return RunConfig(acell=10.0, NG=NG, NK=NK, NB=nb, NBocc=nocc or nb, Zeff=[1.5, 0.5], alpha=[1.0, 1.0],
                     Rion=[0.25, 0.75], Kion=[1, 2])


def _functions(NG, NK, nb, seed):
    """Complex functions with a decaying spectrum, orthonormal per k-point."""
    rng = np.random.default_rng(seed)
    G = np.fft.fftfreq(NG, 1.0 / NG) * (2 * np.pi / 10.0)
    z = rng.standard_normal((NK, NG, nb)) + 1j * rng.standard_normal((NK, NG, nb))
    q, _ = np.linalg.qr(np.fft.ifft(z * np.exp(-0.15 * G * G)[None, :, None], axis=1))
    return np.ascontiguousarray(q.transpose(0, 2, 1)) * np.sqrt(NG / 10.0)


def _exchange(u, w, vq):
    """ubkwbk_vFwbk (F:237-261) in extended precision from the given table."""
    NK, _, N = u.shape
    U, W = u.astype(CL), w.astype(CL)
    out = np.zeros_like(W)
    for kr in range(NK):
        for kc in range(NK):
            k = vq[kr - kc + NK - 1].astype(L) * (L(-1) / (L(N) * L(NK)))
            V = np.fft.ifft(k * np.fft.fft(W[kr][:, None, :] * np.conj(U[kc])[None]), norm="forward")
            out[kr] += (V * U[kc][None]).sum(axis=1)
    return out


def _rel(a, b):
    return float(np.sqrt((np.abs(a - b) ** 2).sum() / (np.abs(b) ** 2).sum()))


def _tol(N, M):
    """Two FP64 roundings of the result, and per pair half a place of 2^60 at each of
    N points, random over N points and M pairs against a sum of the size of one
    pair's (at most 2^4 below full scale): sqrt(N M) 2^-57, twice."""
    return 2.0 ** -52 + 2.0 * np.sqrt(N * M) * 2.0 ** -57


@pytest.mark.parametrize("NG,NK,nb", [(16, 1, 1), (16, 5, 3), (32, 3, 3), (64, 9, 1), (64, 4, 4), (128, 7, 3),
                                      (256, 3, 1), (256, 5, 5), (512, 1, 1), (512, 3, 3)])
def test_exchange_rows_and_symmetric(built_lib, NG, NK, nb):
    """h[u]u pairs (tiles with remainders) and other functions (teams with remainders, every chunking)."""
    from mattohf_gb300 import Context
    u = _functions(NG, NK, nb, 1)
    w = _functions(NG, NK, 2, 2) * (10.0 ** np.linspace(-9, 9, NK * 2)).reshape(NK, 2, 1)
    with Context(_cfg(NG, NK, nb)) as ctx:
        vq = ctx.coulomb()[1]
        ref, refw = _exchange(u, u, vq), _exchange(u, w, vq)
        for tile in (1, 2, 4):
            ctx.set_option(7, tile)
            assert _rel(ctx.ubkwbk_vFwbk(u, u), ref) <= _tol(NG, NK * nb), tile
        for chunks in (0, 1, 2, 3):
            ctx.set_option(2, chunks)
            got = ctx.ubkwbk_vFwbk(u, w)
            for k in range(NK):
                for b in range(2):
                    assert _rel(got[k, b], refw[k, b]) <= _tol(NG, NK * nb), (chunks, k, b)


def test_orbital_scales(built_lib):
    """Any common scale gives the same digits; unequal norms stay accurate normwise;
    zero orbitals give zero, values that are not finite give no number."""
    from mattohf_gb300 import Context
    NG, NK, nb = 64, 5, 3
    u = _functions(NG, NK, nb, 3)
    with Context(_cfg(NG, NK, nb)) as ctx:
        vq = ctx.coulomb()[1]
        F = ctx.ubkwbk_vFwbk(u, u)
        for e in (-400, -60, 60, 400):
            s = 2.0 ** e
            us = u * s
            got = ctx.ubkwbk_vFwbk(us, us)
            if abs(e) < 400:
                assert np.array_equal(got, F * s * s * s)
            else:  # s^3 leaves the exponent range
                assert np.all(got == 0) if e < 0 else not np.all(np.isfinite(got))
        un = u * (10.0 ** np.random.default_rng(4).uniform(-4, 0, (NK, nb, 1)))
        assert _rel(ctx.ubkwbk_vFwbk(un, un), _exchange(un, un, vq)) <= 4 * _tol(NG, NK * nb)
        uz = u.copy()
        uz[2, 1] = 0.0
        got = ctx.ubkwbk_vFwbk(uz, uz)
        assert np.all(got[2, 1] == 0) and _rel(got, _exchange(uz, uz, vq)) <= _tol(NG, NK * nb)
        assert np.all(ctx.ubkwbk_vFwbk(0 * u, 0 * u) == 0)
        for bad in (np.nan, np.inf):
            ub = u.copy()
            ub[1, 0, 7] = bad
            assert not np.any(np.isfinite(ctx.ubkwbk_vFwbk(ub, ub)))


@pytest.mark.parametrize("NG", [16, 32, 64, 128, 256, 512])
def test_kinetic_and_hartree(built_lib, NG):
    """The column transforms: kinetic term and Hartree potential against extended precision.
    Both are limited by white noise of the transforms, at most a place of FP64 of the
    input's norm per coefficient, under the largest kinetic energy."""
    from mattohf_gb300 import Context
    NK, nb, A = 3, 3, 0.07
    u = _functions(NG, NK, nb, 5)
    with Context(_cfg(NG, NK, nb, 2)) as ctx:
        g = ctx.grids()
        t = 0.5 * (g["Gx"].astype(L)[None] + g["kx"].astype(L)[:, None] + L(A)) ** 2
        ref = np.fft.ifft(t[:, None] * np.fft.fft(u.astype(CL)))
        noise = 2.0 ** -52 * float(t.max()) * float(np.linalg.norm(u) / np.linalg.norm(ref))
        assert _rel(ctx.ubk_tubk(u, A), ref) <= 2.0 ** -51 + noise
        for e in (0, -900, 900):  # linear: any scale, and zeros stay zero
            us = u * 2.0 ** e
            us[1, 1] = 0.0
            got = ctx.ubk_tubk(us, A)
            assert np.all(got[1, 1] == 0) and _rel(got[0] * 2.0 ** -e, ref[0]) <= 2.0 ** -51 + noise
        rho = (2.0 / NK) * (np.abs(u[:, :2].astype(CL)) ** 2).sum(axis=(0, 1))
        vH = np.fft.ifft(ctx.coulomb()[0].astype(L) * np.fft.fft(rho)).real
        assert _rel(ctx.ubk_dns(u), rho) <= 2.0 ** -50
        assert _rel(ctx.dns_vH_of(u), vH) <= 2.0 ** -49
