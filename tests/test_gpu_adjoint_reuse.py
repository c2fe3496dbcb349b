"""Repeated adjoint calls on one context, which keep buffers and step graphs (needs a GB300)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("NG,NK,NB", [(32, 4, 2), (64, 18, 4)])  # fused stages; separate launches
def test_sequence_matches_fresh_contexts(built_lib, NG, NK, NB):
    """Window, checkpoint interval, time step, objective, options and other calls may change between
    two gradients: each equals, bit for bit, the one of a context that makes only that call."""
    from mattohf_gb300 import Context, RunConfig
    cfg = RunConfig(acell=9.0, NG=NG, NK=NK, NB=NB, NBocc=NB, Zeff=[2.0], alpha=[1.0], Rion=[0.5], Kion=[1])
    rng = np.random.default_rng(0)
    A = 0.05 * rng.standard_normal(19)
    calls = [(10, 0.002, 0, "energy"), (10, 0.002, 0, "current"), (19, 0.002, 0, "energy"), (5, 0.002, 0, "energy"),
             (19, 0.002, 4, "energy"), (17, 0.001, 4, "current"), (8, 0.001, 8, "energy"), (10, 0.002, 0, "energy")]

    def start(ctx):
        ctx.Init_wf()
        ctx.Gram_Schmidt()

    with Context(cfg) as ctx:
        start(ctx)
        u0 = ctx.get_orbitals()
        for i, (nt, dt, every, obj) in enumerate(calls):
            if i == 3:  # another loop's graph in between
                ctx.set_orbitals(u0)
                ctx.rk4_run(A[:9], A[:9], 0.002)
            if i == 4:
                v = ctx.vion
                ctx.vion = v * 1.1
            if i == 6:
                ctx.set_option(8, 0)
            ctx.set_orbitals(u0)
            got = ctx.adjoint(A[:nt], dt, obj, every) + (ctx.get_orbitals(),)
            with Context(cfg) as one:
                if i >= 4:
                    one.vion = v * 1.1
                if i >= 6:
                    one.set_option(8, 0)
                one.set_orbitals(u0)
                ref = one.adjoint(A[:nt], dt, obj, every) + (one.get_orbitals(),)
            for x, y in zip(got, ref):
                assert np.array_equal(x, y), (i, nt, dt, every, obj)
