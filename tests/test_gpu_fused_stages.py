"""The fused RK4 stages in fixed point against the oracle (needs a GB300)."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from test_gpu_fixed_point import _functions

pytestmark = pytest.mark.gpu


def _cfg(NG, NK, nb, nocc):
    from mattohf_gb300 import RunConfig
    return RunConfig(acell=10.0, NG=NG, NK=NK, NB=nb, NBocc=nocc, Zeff=[1.5, 0.5], alpha=[1.0, 1.0],
                     Rion=[0.25, 0.75], Kion=[1, 2])


def _rel(a, b):
    return float(np.max(np.abs(np.asarray(a) - b)) / max(1e-300, np.max(np.abs(b))))


# Each size at and just above the line to the FP64 stages (M NG = 2048), the most
# columns (NK NB = 64), unoccupied bands, and 1 to 8 CTAs a column: one CTA alone,
# several rounds of its pair teams, teams without a pair.  The energy is dominated by
# terms of the size of the largest kinetic energy's noise, 2^-52 of it a transform,
# eight transforms a step: the tolerance is 2^-52 (8 nt Gmax^2 / 2 + 64) of the
# orbitals (norm 1), and the same of the energies and currents.
@pytest.mark.parametrize("NG,NK,nb,nocc", [(64, 8, 4, 4), (64, 16, 4, 2), (64, 11, 3, 3), (128, 4, 4, 4), (128, 9, 3, 2),
                                           (256, 8, 1, 1), (256, 5, 3, 2), (256, 4, 5, 5)])
def test_fused_fixed_point_stages(built_lib, NG, NK, nb, nocc):
    """RK4 steps with a field, observables and unoccupied bands."""
    from mattohf_gb300 import Context, _capi
    from oracle import mattohf_oracle as O
    from conftest import to_oracle_config
    nt, dt = 2, 0.004 * (64.0 / NG) ** 2
    cfg = dataclasses.replace(_cfg(NG, NK, nb, nocc), dt=dt, NT=nt)
    u = _functions(NG, NK, nb, NG + NK)
    A = 0.05 * np.cos(0.7 * np.arange(nt))
    Aave = A + 0.01
    S = O.make_system(to_oracle_config(cfg))
    ref = O.rt_calculation(S, u, nt=nt, A=A, Aave=Aave)
    tol = 2.0 ** -52 * (8 * nt * 0.5 * (np.pi * NG / 10.0) ** 2 + 64)
    with Context(cfg) as ctx:
        ctx.set_option(_capi.OPT_SMALL_STAGES, 1)
        for ctas in (0, 1, 2, 5, 8):
            ctx.set_option(_capi.OPT_SMALL_CTAS, ctas)
            ctx.set_orbitals(u)
            E, J, N = ctx.rk4_run(A, Aave, dt)
            got = ctx.get_orbitals()
            assert _rel(E, ref.Etot) <= tol and _rel(N, ref.Nele) <= tol, ctas
            assert np.max(np.abs(J - ref.Jtot)) <= tol * max(1.0, np.max(np.abs(ref.Jtot))), ctas
            assert np.linalg.norm(got - ref.ubk) <= tol * np.linalg.norm(ref.ubk), ctas


def test_fused_fixed_point_zeros_and_nan(built_lib):
    """Zero orbitals stay zero; a value that is not finite is reported."""
    from mattohf_gb300 import Context, MattohfError, _capi
    NG, NK, nb = 64, 8, 4
    u = _functions(NG, NK, nb, 1)
    A = np.zeros(2)
    with Context(_cfg(NG, NK, nb, nb)) as ctx:
        ctx.set_option(_capi.OPT_SMALL_STAGES, 1)
        ctx.set_orbitals(0 * u)
        E, J, N = ctx.rk4_run(A, A, 0.01)
        assert np.all(E == 0) and np.all(J == 0) and np.all(N == 0) and np.all(ctx.get_orbitals() == 0)
        u[3, 1, 5] = np.nan
        ctx.set_orbitals(u)
        with pytest.raises(MattohfError):
            ctx.rk4_run(A, A, 0.01)
