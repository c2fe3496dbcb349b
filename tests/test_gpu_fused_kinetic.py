"""The kinetic factors of the fused fixed-point stages over many steps (needs a GB300)."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from test_gpu_fixed_point import _cfg

pytestmark = pytest.mark.gpu
L, CL = np.longdouble, np.clongdouble
OPT_SMALL = 8


def _rk4(c, T, v0, occ, dt, nt, block=500):
    """nt RK4 steps of plane-wave amplitudes: h = T + v0 n, with the uniform density n = sum
    occ |c|^2.  A step multiplies each by a factor that depends on the moduli alone, which
    change by less than 1e-16 a step: one factor for a block of steps."""
    def h(z):
        return -1j * (T + v0 * (occ * (z.real ** 2 + z.imag ** 2)).sum()) * z
    assert nt % block == 0
    for _ in range(nt // block):
        k0 = h(c)
        k1 = h(c + dt / 2 * k0)
        k2 = h(c + dt / 2 * k1)
        k3 = h(c + dt * k2)
        f = 1 + dt / 6 * (k0 + 2 * k1 + 2 * k2 + k3) / c
        n = block
        while n:
            if n & 1:
                c = c * f
            f, n = f * f, n >> 1
    return c


# One plane wave of a low frequency per band, no exchange, no ions: the result is known.  A
# step rounds a value a few times at random, 2^-53 of it each: 8 sqrt(4 nt) 2^-53 after nt
# steps.  An error of the factors is the same in every step: their last place, were it
# that of the largest factor (2.9e-14 at NG = 256), would give up to 5e-12 over these times.
@pytest.mark.parametrize("NG,NK,nb", [(256, 4, 2), (128, 8, 2), (64, 8, 4)])
def test_low_frequencies_keep_their_energy(built_lib, NG, NK, nb):
    from mattohf_gb300 import Context
    cfg = dataclasses.replace(_cfg(NG, NK, nb), functional="none")
    nt = 150000
    with Context(cfg) as ctx:
        g = ctx.grids()
        dt = 2.5 / float(0.5 * (np.abs(g["Gx"]).max() + np.abs(g["kx"]).max()) ** 2)
        n = np.arange(nb)
        x = np.arange(NG) / NG
        wave = np.exp(2j * np.pi * n[:, None] * x[None])
        u = np.repeat(wave[None], NK, axis=0) / np.sqrt(10.0)
        ctx.vion = np.zeros(NG)
        ctx.set_option(OPT_SMALL, 1)
        ctx.set_orbitals(u)
        A = np.zeros(nt)
        ctx.rk4_run(A, A, dt)
        got = ctx.get_orbitals()
        T = 0.5 * (g["Gx"][n].astype(L)[None] + g["kx"].astype(L)[:, None]) ** 2
        v0 = L(ctx.coulomb()[0][0])
        c = _rk4(np.full((NK, nb), 1 / np.sqrt(L(10)), dtype=CL), T, v0, L(2) / L(NK), L(dt), nt)
        amp = np.einsum("kbx,bx->kb", got.astype(CL), np.conj(wave.astype(CL))) / NG
        assert np.max(np.abs(amp - c) / np.abs(c)) <= 8 * np.sqrt(4.0 * nt) * 2.0 ** -53
