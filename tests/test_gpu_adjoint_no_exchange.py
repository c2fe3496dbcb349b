"""The gradient without exchange (any functional but HF), both forms of the stages, against
the oracle's discrete adjoint (needs a GB300)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("NG,NK,nb", [(32, 4, 2), (64, 8, 2), (128, 2, 1), (256, 1, 4)])
@pytest.mark.parametrize("objective", ["energy", "current"])
@pytest.mark.parametrize("small", [0, 1, 2])
def test_gradient_without_exchange(built_lib, NG, NK, nb, objective, small):
    from mattohf_gb300 import Context, RunConfig, _capi
    from oracle import mattohf_oracle as O
    from conftest import to_oracle_config
    cfg = RunConfig(acell=8.0, NG=NG, NK=NK, NB=nb, NBocc=nb, Zeff=[2.0], alpha=[1.0], Rion=[0.5], Kion=[1],
                    functional="none")
    S = O.make_system(to_oracle_config(cfg))
    u0 = O.gram_schmidt(S, O.init_wf(S))
    A = 0.05 * np.random.default_rng(4).standard_normal(5)
    dt = 0.004 * min(1.0, (64.0 / NG) ** 2)
    Lr, gr, gvr = O.rt_adjoint(S, u0, A, dt, objective)
    with Context(cfg) as ctx:
        ctx.set_option(_capi.OPT_SMALL_STAGES, small)
        ctx.set_orbitals(u0)
        L, g, gv = ctx.adjoint(A, dt, objective)
    assert abs(L - Lr) <= 1e-10 * max(1.0, abs(Lr))
    assert np.max(np.abs(g - gr)) <= 1e-9 * np.max(np.abs(gr))
    assert np.max(np.abs(gv - gvr)) <= 1e-9 * np.max(np.abs(gvr))
