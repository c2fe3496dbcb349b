"""The exchange through the density matrix against extended precision (needs a GB300)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_fixed_point import _cfg, _functions, _rel, CL, L

pytestmark = pytest.mark.gpu


def _rows(u, w, vq, ks, xs):
    """ubkwbk_vFwbk (F:237-261) at the k-points ks and grid points xs, in extended precision,
    W by its definition over k."""
    NK, _, N = u.shape
    U = u.astype(CL)
    v = np.fft.ifft(vq.astype(L) * (L(-1) / (L(N) * L(NK))), norm="forward", axis=-1)
    d = (xs[:, None] - np.arange(N)[None, :]) % N
    D = [U[k][:, xs].T @ np.conj(U[k]) for k in range(NK)]
    W = [sum(D[kc] * v[k - kc + NK - 1][d] for kc in range(NK)) for k in ks]
    return [[x[k].astype(CL) @ Wk.T for k, Wk in zip(ks, W)] for x in w]


# Two FP64 roundings of the result, and W's and w's own: W is at most 2^59.4 in units of
# its last place, some 2^7 below that for a few bands' smooth orbitals, and is off by the
# roundings of two transforms of length L over k (each log2 L stages of under a place):
# 2 log2(2 NK) 2^-52 of its largest element.
def _tol(NK):
    return 2.0 ** -52 * (1.0 + 2.0 * np.log2(4 * NK))


# NK a power of two, one above it and one below; 1 to 9 bands of w (all group sizes and
# remainders); every transform length from 64 (NK = 17) up, the largest grid and W
@pytest.mark.parametrize("NG,NK,nocc,nb,nbw", [(64, 64, 4, 4, 7), (64, 65, 4, 6, 2), (64, 31, 9, 9, 9), (128, 33, 8, 8, 3),
                                               (128, 32, 8, 9, 4), (256, 17, 12, 12, 5), (256, 64, 4, 4, 6),
                                               (64, 255, 2, 2, 1), (512, 16, 16, 16, 8)])
def test_density_matrix_exchange(built_lib, NG, NK, nocc, nb, nbw):
    """w = u (with unoccupied bands), other functions, the pairs on the same input."""
    from mattohf_gb300 import Context
    u = _functions(NG, NK, nb, NG + NK)
    w = _functions(NG, NK, nbw, 2) * (10.0 ** np.linspace(-9, 9, NK * nbw)).reshape(NK, nbw, 1)
    with Context(_cfg(NG, NK, nb, nocc)) as ctx:
        vq = ctx.coulomb()[1]
        ks, xs = sorted({0, 1, NK // 2, NK - 1}), np.unique(np.linspace(0, NG - 1, 13).astype(int))
        refs = _rows(u[:, :nocc], (u, w), vq, ks, xs)
        for x, ref in zip((u, w), refs):
            ctx.set_option(7, 0)
            got = ctx.ubkwbk_vFwbk(u, x)
            for k, r in zip(ks, ref):
                assert max(_rel(got[k][b][xs], r[b]) for b in range(len(r))) <= _tol(NK), k
            ctx.set_option(7, 2)  # pairs
            assert _rel(ctx.ubkwbk_vFwbk(u, x), got) <= 2 * _tol(NK)


def test_density_matrix_scales(built_lib):
    """Any common scale gives the same digits, zero orbitals give zero, values that are
    not finite give no number, in u as well as in w, and nothing of them stays behind."""
    from mattohf_gb300 import Context
    NG, NK, nb = 64, 64, 4
    u = _functions(NG, NK, nb, 3)
    with Context(_cfg(NG, NK, nb)) as ctx:
        F, Fw = ctx.ubkwbk_vFwbk(u, u), ctx.ubkwbk_vFwbk(u, u.copy())
        for e in (-60, 60, 300):
            us = u * 2.0 ** e
            assert np.array_equal(ctx.ubkwbk_vFwbk(us, us), F * 2.0 ** e * 2.0 ** e * 2.0 ** e)
        assert np.all(ctx.ubkwbk_vFwbk(0 * u, u) == 0) and np.all(ctx.ubkwbk_vFwbk(u, 0 * u) == 0)
        for bad in (np.nan, np.inf):
            ub = u.copy()
            ub[5, 1, 7] = bad
            assert not np.any(np.isfinite(ctx.ubkwbk_vFwbk(ub, u)))
            got = ctx.ubkwbk_vFwbk(u, ub)
            assert not np.any(np.isfinite(got[5, 1]))
            got[5, 1] = Fw[5, 1]
            assert np.array_equal(got, Fw)
        assert np.array_equal(ctx.ubkwbk_vFwbk(u, u), F)


# the runs through the density matrix (no tile pairs) first, between and last, alone, and
# all of them; two roundings a stage each way on top of the steps' own: 2^-52 times
# 4 stages times the tolerance of one apply
@pytest.mark.parametrize("shapes", [[(64, 8), (3, 2), (33, 9)], [(3, 2), (33, 9), (5, 1)], [(33, 9), (64, 8)], [(4, 3)]])
def test_batch_members_through_the_density_matrix(built_lib, shapes):
    """A batch of runs either way against the runs by pairs, twice (graph replay), and after a tile is asked for."""
    from mattohf_gb300 import Batch, _capi
    nt, dt = 3, 0.003
    A = 0.02 * np.random.default_rng(8).standard_normal((len(shapes), nt))
    u0 = [_functions(64, NK, nb, NK) for NK, nb in shapes]
    tol = 4 * nt * _tol(64)
    with Batch([_cfg(64, NK, nb) for NK, nb in shapes]) as b:
        def run():
            for r, u in enumerate(u0):
                b[r].set_orbitals(u)
            return b.rk4_run(A, A, dt), [b[r].get_orbitals() for r in range(len(u0))]
        first, again = run(), run()
        b.set_option(_capi.OPT_SYM_TILE, 2)  # pairs
        pairs = run()
    for x, y in zip(first[0], again[0]):
        assert np.array_equal(x, y)
    for x, y in zip(first[0], pairs[0]):
        assert np.max(np.abs(np.asarray(x) - np.asarray(y))) <= tol * max(1.0, np.max(np.abs(np.asarray(y))))
    for a, p in zip(first[1], pairs[1]):
        assert _rel(a, p) <= tol
