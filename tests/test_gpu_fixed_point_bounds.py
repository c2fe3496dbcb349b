"""Bounds of the fixed-point exchange: sums of many large terms of one sign (needs a GB300).

The inputs are far from orthonormal: equal functions, flat on six neighbouring points with
equal real and imaginary parts, so that every component sits at its bound, and one
function a quarter of a right angle from them, so that the whole modulus of every term
falls on one component.  The amplitudes leave the short scale factors no slack.
"""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_fixed_point import _exchange, _rel, _tol

pytestmark = pytest.mark.gpu


def _cfg(NG, NK, nb, nocc=None, acell=10.0):
    from mattohf_gb300 import RunConfig
    return RunConfig(acell=acell, NG=NG, NK=NK, NB=nb, NBocc=nocc or nb, Zeff=[2.0], alpha=[1.0], Rion=[0.5], Kion=[1])


def _flat(NG, NK, nb, amp):
    u = np.zeros((NK, nb, NG), dtype=np.complex128)
    u[:, :, 3:9] = amp * (1 + 1j)
    return u


# sums of 16 sources in one accumulator: by the default chunks (36 sources), by one chunk
# for all; sums of those terms reach 1.11 to 1.19 times 2^63
@pytest.mark.parametrize("NG,NK,nb,acell,chunks", [(32, 64, 16, 10.0, 0), (32, 64, 16, 4.0, 0), (64, 1, 16, 10.0, 1),
                                                   (128, 1, 24, 10.0, 1), (256, 1, 40, 10.0, 1)])
def test_rows_accumulator(built_lib, NG, NK, nb, acell, chunks):
    from mattohf_gb300 import Context
    u = _flat(NG, NK, nb, 1.75)
    w = 1.1 * np.exp(-0.25j * np.pi) * u[:, :16]
    with Context(_cfg(NG, NK, nb, acell=acell)) as ctx:
        ctx.set_option(2, chunks)
        vq = ctx.coulomb()[1]
        got = ctx.ubkwbk_vFwbk(u, w)
        # the functions of a k-point are alike: one of each in extended precision
        ref = _exchange(np.sqrt(float(nb)) * u[:, :1], w[:, :1], vq)
        for b in range(w.shape[1]):
            assert _rel(got[:, b], ref[:, 0]) <= _tol(NG, NK * nb), b


# the symmetric tiles take eight sources per accumulator
@pytest.mark.parametrize("NG,NK,nb", [(32, 4, 16), (64, 2, 16), (256, 1, 17)])
def test_symmetric_accumulator(built_lib, NG, NK, nb):
    from mattohf_gb300 import Context
    u = _flat(NG, NK, nb, 1.75)
    u[:, -1] *= np.exp(-0.25j * np.pi)
    with Context(_cfg(NG, NK, nb)) as ctx:
        vq = ctx.coulomb()[1]
        ref = _exchange(u, u, vq)
        for tile in (4, 8) if NG < 256 else (2, 4):
            ctx.set_option(7, tile)
            assert _rel(ctx.ubkwbk_vFwbk(u, u), ref) <= _tol(NG, NK * nb), tile


# A CTA of the fused stages with 16 and 24 pairs; the terms of the last, unoccupied band
# have the modulus on one component.  Both paths round every orbital value a few times
# a stage: 2^-48 of the largest leaves room for 32 of them.
@pytest.mark.parametrize("NG,nocc,amp,ampw", [(128, 16, 1.3125, 0.9722718), (128, 24, 1.75, 1.1490485),
                                              (64, 32, 1.3125, 0.7513010), (256, 16, 1.3125, 0.9722718)])
def test_fused_stage_accumulator(built_lib, NG, nocc, amp, ampw):
    from mattohf_gb300 import Context
    u = _flat(NG, 1, nocc + 1, amp)
    u[:, -1] *= ampw * np.exp(-0.25j * np.pi)
    out = []
    with Context(_cfg(NG, 1, nocc + 1, nocc)) as ctx:
        for small in (1, 0):
            ctx.set_option(8, small)
            if small:
                ctx.set_option(9, 1)
            ctx.set_orbitals(u)
            ctx.rk4_run(np.zeros(1), np.zeros(1), 1e-6)
            out.append(ctx.get_orbitals())
    assert np.max(np.abs(out[0] - out[1])) <= 2.0 ** -48 * np.max(np.abs(u))
