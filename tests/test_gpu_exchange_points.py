"""The exchange by itself, grid point by grid point, for functions that decay over many
orders of magnitude, against extended precision (needs a GB300)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_fixed_point import _cfg, _exchange, _tol

pytestmark = pytest.mark.gpu


def _localised(NG, NK, nb, seed, width, norms=0.0, zeros=0):
    """Gaussians of that width (in grid points) about nearby centres, polynomials times
    phases, norms spread over 10^norms; the last points zero."""
    rng = np.random.default_rng(seed)
    x = np.arange(NG)[None, None, :] - NG / 2 - rng.uniform(-0.5, 0.5, (NK, nb, 1)) * width
    u = np.exp(-0.5 * (x / width) ** 2) * (x / width) ** np.arange(nb)[None, :, None]
    u = u * np.exp(2j * np.pi * (rng.uniform(0, 1, (NK, nb, 1)) + 0.1 * rng.standard_normal((NK, nb, NG))))
    u *= 10.0 ** -rng.uniform(0.0, norms, (NK, nb, 1)) if norms else 1.0
    if zeros:
        u[:, :, -zeros:] = 0.0
    return np.ascontiguousarray(u)


def _scaled_rel(got, ref, m):
    """Error norm with every grid point in units of m(x); where m is zero, so is the result."""
    on = m > 0
    assert np.all(got[..., ~on] == 0)
    g, r = got[..., on] / m[on], ref[..., on] / m[on]
    return float(np.sqrt((np.abs(g - r) ** 2).sum() / (np.abs(r) ** 2).sum()))


# Pairs: the terms phi_ab(x) u_b(x) of a point are as accurate as phi_ab, that is as the
# normwise bound has it, in units of the largest |u_b(x)| times b's norm.  The least of the
# values is 1e-5 to 1e-200 of the largest; norms a factor of 1e6 apart; empty points.
@pytest.mark.parametrize("NG,NK,nb,width,norms,zeros", [(32, 5, 2, 3.0, 0, 0), (64, 3, 3, 4.0, 0, 5), (128, 4, 2, 2.2, 6, 0),
                                                        (256, 3, 3, 16.0, 6, 9), (512, 2, 2, 30.0, 0, 0)])
def test_pairs_point_by_point(built_lib, NG, NK, nb, width, norms, zeros):
    from mattohf_gb300 import Context
    u = _localised(NG, NK, nb, 1, width, norms, zeros)
    w = _localised(NG, NK, 2, 2, NG / 3.0) * (10.0 ** np.linspace(-9, 9, NK * 2)).reshape(NK, 2, 1)
    m = (np.abs(u) * np.linalg.norm(u, axis=-1)[..., None]).max(axis=(0, 1))
    with Context(_cfg(NG, NK, nb)) as ctx:
        vq = ctx.coulomb()[1]
        for tile in (1, 2, 4):
            ctx.set_option(7, tile)
            for x in (u, w):
                got, ref = ctx.ubkwbk_vFwbk(u, x), _exchange(u, x, vq)
                for k in range(NK):
                    for b in range(x.shape[1]):
                        assert _scaled_rel(got[k, b], ref[k, b], m) <= 4 * _tol(NG, NK * nb), (tile, k, b)


# where h[u] w goes through the density matrix, the exchange by itself takes the pairs
def test_many_orbitals_point_by_point(built_lib):
    from mattohf_gb300 import Context
    NG, NK, nb = 64, 40, 4
    u = _localised(NG, NK, nb, 3, 5.0, 0, 3)
    w = _localised(NG, NK, 3, 4, NG / 3.0)
    m = (np.abs(u) * np.linalg.norm(u, axis=-1)[..., None]).max(axis=(0, 1))
    with Context(_cfg(NG, NK, nb)) as ctx:
        vq = ctx.coulomb()[1]
        for x in (u, w):
            got, ref = ctx.ubkwbk_vFwbk(u, x), _exchange(u, x, vq)
            for k in range(NK):
                for b in range(x.shape[1]):
                    assert _scaled_rel(got[k, b], ref[k, b], m) <= 4 * _tol(NG, NK * nb), (k, b)


def test_rank_rows_point_by_point(built_lib):
    """A rank's rows: the exchange alone of a range of k-points, the same bits as the whole."""
    import torch
    from mattohf_gb300 import Context, _capi
    NG, NK, nb = 64, 6, 2
    u = _localised(NG, NK, nb, 5, 4.0)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x).view(np.float64)).cuda()
    with Context(_cfg(NG, NK, nb)) as ctx:
        ctx.set_option(4, 0)  # by rows
        whole = ctx.ubkwbk_vFwbk(u, u)
        du, dw = dev(u), dev(u[2:5])
        out = torch.empty_like(dw)
        torch.cuda.synchronize()
        assert ctx.lib.mattohf_hpsi_kslice_device(ctx.h, du.data_ptr(), 2, 3, dw.data_ptr(), nb, 0.0, 1, out.data_ptr()) == _capi.OK
        ctx.synchronize()
        assert np.array_equal(out.cpu().numpy().view(np.complex128), whole[2:5])
