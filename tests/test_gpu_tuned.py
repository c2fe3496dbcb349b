"""What the autotuner chose for h[u]u and the forward step does not decide other shapes
(needs a GB300)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_fixed_point import _cfg, _functions

pytestmark = pytest.mark.gpu


# fused or separate launches, whichever the tuner finds: where the rule for the reverse
# stages (separate: 256/8/2, 64/8/4; fused: 32/16/2) and the forward's choice agree and differ
@pytest.mark.parametrize("NG,NK,nb", [(256, 8, 2), (64, 8, 4), (32, 16, 2), (128, 8, 4)])
def test_gradient_of_a_tuned_context(built_lib, NG, NK, nb):
    """The reverse stages of a tuned context are those of the size rule: the same bits as
    from a context whose forward is set to the tuner's choice by other means."""
    from mattohf_gb300 import Context, _capi
    u = _functions(NG, NK, nb, 1)
    A = 0.05 * np.sin(1.0 + np.arange(3))
    dt = 0.05 / NG
    with Context(_cfg(NG, NK, nb)) as ctx:
        ctx.set_orbitals(u)
        t = ctx.autotune(steps=20)
        got = ctx.adjoint(A, dt)
        end = ctx.get_orbitals()
    out = []
    for small in (0, 1, 2):
        with Context(_cfg(NG, NK, nb)) as ctx:
            if small != 2:
                ctx.set_option(_capi.OPT_SMALL_STAGES, small)
            if t["small_ctas"]:
                ctx.set_option(_capi.OPT_SMALL_CTAS, t["small_ctas"])
            ctx.set_option(_capi.OPT_SYM_TILE, t["sym_tile"])
            ctx.set_orbitals(u)
            out.append((*ctx.adjoint(A, dt), ctx.get_orbitals()))
    forward = 1 if t["small_stages"] else 0
    assert np.array_equal(end, out[forward][3])
    if not np.array_equal(out[2][3], end):
        pytest.skip("the rule's forward is not the tuner's: nothing to compare the reverse with")
    for a, b in zip(got, out[2]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("NG,NK,nb,nbw", [(64, 8, 8, 32), (128, 8, 12, 24), (256, 16, 2, 2)])
def test_other_functions_of_a_tuned_context(built_lib, NG, NK, nb, nbw):
    """h[u]w on other functions takes the same path before and after tuning."""
    from mattohf_gb300 import Context
    u, w = _functions(NG, NK, nb, 1), _functions(NG, NK, nbw, 2)
    with Context(_cfg(NG, NK, nb)) as ctx:
        before = ctx.ubkwbk_hwbk(u, w, 0.1)
        ctx.set_orbitals(u)
        ctx.autotune(steps=5)
        assert np.array_equal(ctx.ubkwbk_hwbk(u, w, 0.1), before)
