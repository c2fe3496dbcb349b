"""The exchange through the density matrix inside h[u] w, the observables and a gradient,
against extended precision (needs a GB300)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_fixed_point import _cfg, _functions, _rel, CL, L
from test_gpu_density_matrix import _rows, _tol

pytestmark = pytest.mark.gpu
OPT_TILE, OPT_SMALL = 7, 8


def _norm(a):
    return float(np.sqrt((np.abs(a) ** 2).sum()))


# Every transform length over k from the shortest (16: NK up to 8) on, NK a power of two, one
# above and one below; 1 to 32 functions (all group sizes and remainders); the largest grid.
# The exchange is what h[u] w has beyond the kinetic term and the potential, which are the
# same FP64 values in calls of their own: 2^-51 of h w more than its own error.
@pytest.mark.parametrize("NG,NK,nocc,nb,nbw", [(64, 8, 8, 8, 32), (256, 7, 30, 30, 24), (128, 8, 24, 25, 33),
                                               (128, 16, 12, 12, 9), (64, 64, 4, 4, 7), (64, 65, 4, 6, 2),
                                               (128, 33, 8, 8, 3), (256, 64, 4, 4, 6), (64, 255, 2, 2, 1),
                                               (512, 16, 16, 16, 8)])
def test_exchange_in_h(built_lib, NG, NK, nocc, nb, nbw):
    from mattohf_gb300 import Context
    u = _functions(NG, NK, nb, NG + NK)
    w = np.ascontiguousarray(_functions(NG, NK, nbw, 2) * (10.0 ** np.linspace(-9, 9, NK * nbw)).reshape(NK, nbw, 1))
    took = []
    with Context(_cfg(NG, NK, nb, nocc)) as ctx:
        ctx.vion = np.zeros(NG)
        vq = ctx.coulomb()[1]
        ks, xs = sorted({0, 1, NK // 2, NK - 1}), np.unique(np.linspace(0, NG - 1, 13).astype(int))
        vH = ctx.dns_vH_of(u).astype(L)
        for x, ref in zip((u, w), _rows(u[:, :nocc], (u, w), vq, ks, xs)):
            ctx.set_option(OPT_TILE, 0)
            h = ctx.ubkwbk_hwbk(u, x, 0.1)
            rest = ctx.ubk_tubk(x, 0.1).astype(CL) + vH * x
            for k, r in zip(ks, ref):
                for b in range(len(r)):
                    err = _norm(h[k, b][xs] - rest[k, b][xs] - r[b])
                    assert err <= _tol(NK) * _norm(r[b]) + 2.0 ** -51 * (_norm(h[k, b][xs]) + _norm(rest[k, b][xs])), (k, b)
            ctx.set_option(OPT_TILE, 2)
            took.append(not np.array_equal(ctx.ubkwbk_hwbk(u, x, 0.1), h))  # the pairs round otherwise
    assert any(took)


@pytest.mark.parametrize("NG,NK,nb", [(64, 64, 4), (256, 64, 4), (128, 33, 8)])
def test_exchange_energy(built_lib, NG, NK, nb):
    """Exc = occ / 2 <u| F u> of both forms; any common scale of the orbitals."""
    from mattohf_gb300 import Context
    u = _functions(NG, NK, nb, 6)
    with Context(_cfg(NG, NK, nb)) as ctx:
        def exc(tile, scale=1.0):
            ctx.set_option(OPT_TILE, tile)
            ctx.set_orbitals(u * scale)
            return ctx.observables(0.1)["Exc"]
        pairs, dm = exc(2), exc(0)
        assert abs(dm - pairs) <= 2 * _tol(NK) * abs(pairs)
        assert exc(0, 2.0 ** 60) == dm * 2.0 ** 240 and exc(0, 2.0 ** -60) == dm * 2.0 ** -240


def test_gradient_whose_forward_uses_the_density_matrix(built_lib):
    """Objective and gradient with the forward through the density matrix against the
    forward by pairs: two steps of four stages each way, each apply off by its tolerance,
    the gradient's own cancellation within a factor of 2^6."""
    from mattohf_gb300 import Context
    NG, NK, nb, dt = 64, 64, 4, 0.004
    A = np.array([0.05, 0.08])
    u = _functions(NG, NK, nb, 9)
    out = []
    with Context(_cfg(NG, NK, nb)) as ctx:
        ctx.set_option(OPT_SMALL, 0)
        for tile in (0, 2):
            ctx.set_option(OPT_TILE, tile)
            ctx.set_orbitals(u)
            out.append((*ctx.adjoint(A, dt), ctx.get_orbitals()))
    (_, g0, v0, u0), (_, g1, v1, u1) = out
    assert not np.array_equal(u0, u1) and _rel(u0, u1) <= 8 * _tol(NK)
    assert _rel(g0, g1) <= 2.0 ** 6 * 16 * _tol(NK) and _rel(v0, v1) <= 2.0 ** 6 * 16 * _tol(NK)


def test_batch_members_take_their_form(built_lib):
    """Large members go through the density matrix, whose roundings are others than the
    pairs'; small ones by pairs, whose sums are exact at any tile."""
    from mattohf_gb300 import Batch
    shapes, nt = [(64, 8), (3, 2), (33, 9)], 2
    u0 = [_functions(64, NK, nb, NK) for NK, nb in shapes]
    out = []
    with Batch([_cfg(64, NK, nb) for NK, nb in shapes]) as b:
        for tile in (0, 2):
            b.set_option(OPT_TILE, tile)
            for r, u in enumerate(u0):
                b[r].set_orbitals(u)
            b.rk4_run(np.zeros((3, nt)), np.zeros((3, nt)), 0.003)
            out.append([b[r].get_orbitals() for r in range(3)])
    assert [np.array_equal(x, y) for x, y in zip(*out)] == [False, True, False]
