"""Functions over the whole exponent range of FP64: each column by itself (needs a GB300)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_fixed_point import _cfg, _functions

pytestmark = pytest.mark.gpu


# h[u] w is linear in w, column by column: a power of two changes no digit while all values
# are normal numbers.  Below 2^-1022 the test's inputs are rounded at 2^-1074 themselves, half
# a place of which the kinetic term enlarges by (pi NG / 10)^2 / 2 at most, and the last
# rounding of a result may then fall the other way: a place of the largest.
SHAPES = [(16, 3, 2, 2), (64, 4, 2, 3), (128, 3, 1, 1), (256, 2, 2, 2), (512, 2, 1, 2),
          (64, 64, 4, 3)]  # the last through the density matrix


@pytest.mark.parametrize("NG,NK,nocc,nbw", SHAPES)
def test_small_functions(built_lib, NG, NK, nocc, nbw):
    from mattohf_gb300 import Context
    u, w = _functions(NG, NK, nocc, 1), _functions(NG, NK, nbw, 2)
    with Context(_cfg(NG, NK, nocc)) as ctx:
        calls = [lambda x: ctx.ubk_tubk(x, 0.1), lambda x: ctx.ubkwbk_vFwbk(u, x), lambda x: ctx.ubkwbk_hwbk(u, x, 0.1)]
        refs = [f(w) for f in calls]
        for e in (-1010, -970, -940, -600):
            for f, ref in zip(calls, refs):
                got = np.ldexp(f(np.ldexp(w.view(float), e).view(complex)).view(float), -e)
                if e > -900:
                    assert np.array_equal(got, ref.view(float)), e
                else:
                    tol = 2.0 ** -52 * np.max(np.abs(ref)) + 2.0 ** (-1075 - e) * (0.5 * (np.pi * NG / 10.0) ** 2 + 1.0)
                    assert np.max(np.abs(got - ref.view(float))) <= tol, e


@pytest.mark.parametrize("NG,NK,nb", [(32, 3, 2), (256, 2, 2)])
def test_small_orbitals(built_lib, NG, NK, nb):
    """Orbitals down to 2^-500: density and Hartree potential as squares of them, the exchange on w."""
    from mattohf_gb300 import Context
    u, w = _functions(NG, NK, nb, 3), _functions(NG, NK, 2, 4)
    with Context(_cfg(NG, NK, nb)) as ctx:
        ctx.vion = np.zeros(NG)
        vH, F = ctx.dns_vH_of(u), ctx.ubkwbk_vFwbk(u, w)
        for e in (-450, -490, -500):
            us = u * 2.0 ** e
            for got, ref in ((ctx.dns_vH_of(us), vH), (ctx.ubkwbk_vFwbk(us, w).view(float), F.view(float))):
                assert np.max(np.abs(np.ldexp(got, -2 * e) - ref)) <= 2.0 ** -60 * np.max(np.abs(ref)), e


@pytest.mark.parametrize("NG,NK,nocc,nbw", SHAPES)
def test_large_functions(built_lib, NG, NK, nocc, nbw):
    """Beyond 2^510 the square of w is no number, but nothing in h[u] w needs it, and the
    exchange alone needs no square of u."""
    from mattohf_gb300 import Context
    u, w = _functions(NG, NK, nocc, 1), _functions(NG, NK, nbw, 2)
    with Context(_cfg(NG, NK, nocc)) as ctx:
        F = ctx.ubkwbk_vFwbk(u, w)
        for f in (lambda x: ctx.ubk_tubk(x, 0.1), lambda x: ctx.ubkwbk_vFwbk(u, x), lambda x: ctx.ubkwbk_hwbk(u, x, 0.1)):
            ref = f(w)
            for e in (505, 515, 900):
                assert np.array_equal(f(w * 2.0 ** e), ref * 2.0 ** e), e
        assert np.array_equal(ctx.ubkwbk_vFwbk(u * 2.0 ** 520, w * 2.0 ** -100), F * 2.0 ** 940)
