"""Calls on a device with next to no free memory (needs a GB300): what has a form that needs
less takes it, what has none reports it, and the context stays usable."""
from __future__ import annotations

import contextlib

import numpy as np
import pytest

from test_gpu_fixed_point import _cfg, _functions, _rel

pytestmark = pytest.mark.gpu
OPT_CHUNKS, OPT_TILE, OPT_GRAPH = 2, 7, 1
LEFT = 24 << 20
SHAPE = (512, 128, 32)  # 33 MB of orbitals in the density matrix's layout


@contextlib.contextmanager
def _no_room():
    """All but LEFT bytes of the device's memory taken (nothing is written to them)."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - LEFT, dtype=torch.uint8, device="cuda")
    try:
        assert torch.cuda.mem_get_info()[0] <= LEFT
        yield
    finally:
        del held
        torch.cuda.empty_cache()


@pytest.fixture(scope="module")
def orbitals(built_lib):
    from mattohf_gb300 import Context
    with Context(_cfg(64, 64, 4)) as ctx:  # every kernel is loaded before the memory goes
        u = _functions(64, 64, 4, 1)
        ctx.ubkwbk_hwbk(u, u, 0.1)
        ctx.ubkwbk_hwbk(u, u[:, :2], 0.1)
    NG, NK, nb = SHAPE
    return _functions(NG, 4, nb, 2).repeat(NK // 4, axis=0)


def test_density_matrix_tables_without_room(orbitals):
    """No room for the density matrix's tables: the pairs, which were there, and the
    density matrix again once there is."""
    from mattohf_gb300 import Context
    u = orbitals
    with Context(_cfg(*SHAPE)) as ctx:
        ctx.set_option(OPT_CHUNKS, 1)  # pairs
        pairs = ctx.ubkwbk_hwbk(u, u, 0.1)
        ctx.set_option(OPT_CHUNKS, 0)
        with _no_room():
            assert np.array_equal(ctx.ubkwbk_hwbk(u, u, 0.1), pairs)
        ctx.set_option(OPT_TILE, 0)
        dm = ctx.ubkwbk_hwbk(u, u, 0.1)
        assert not np.array_equal(dm, pairs) and _rel(dm, pairs) <= 2.0 ** -45


def test_step_without_room(orbitals):
    """The same for a propagation."""
    from mattohf_gb300 import Context
    A = np.full(1, 0.01)
    out = []
    with Context(_cfg(*SHAPE)) as ctx:
        ctx.set_option(OPT_GRAPH, 0)
        for chunks in (1, 0):
            ctx.set_option(OPT_CHUNKS, chunks)
            ctx.set_orbitals(orbitals)
            with _no_room() if chunks == 0 else contextlib.nullcontext():
                obs = ctx.rk4_run(A, A, 1e-4)
            out.append((ctx.get_orbitals(), *obs))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_apply_that_runs_out_of_room(orbitals):
    """An apply whose exchange finds no memory after its density was started: an error; once
    the streams are synchronised the caller's buffers are free, and the context works."""
    import torch
    from mattohf_gb300 import Context, _capi
    NG, NK, nb = SHAPE
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x).view(np.float64)).cuda()
    with Context(_cfg(*SHAPE)) as ctx:
        u, w = dev(orbitals), dev(orbitals[:, :2])
        ctx.ubk_tubk(orbitals[:, :2], 0.1)  # the buffers that every apply takes
        out = torch.empty_like(w)
        torch.empty_like(u).zero_()  # its kernel is loaded too
        call = lambda: ctx.lib.mattohf_hpsi_device(ctx.h, u.data_ptr(), w.data_ptr(), 2, 0.1, out.data_ptr())
        torch.cuda.synchronize()
        with _no_room():
            assert call() == _capi.ERR_ALLOC
            ctx.synchronize()
            u.zero_()
            torch.cuda.synchronize()
        u.copy_(dev(orbitals))
        torch.cuda.synchronize()
        assert call() == _capi.OK
        ctx.synchronize()
        got = out.cpu().numpy().view(np.complex128)
        assert np.array_equal(got, ctx.ubkwbk_hwbk(orbitals, orbitals[:, :2], 0.1))


def test_smaller_calls_after_one_that_found_no_room(orbitals):
    """A call that fails to enlarge the work buffers leaves none of them half made: smaller
    calls, which the old ones served, make them again and give the same bits."""
    from mattohf_gb300 import Context, MattohfError, _capi
    NG, NK, nb = SHAPE
    A = np.full(3, 0.01)
    with Context(_cfg(NG, NK, 2)) as ctx:
        u = np.ascontiguousarray(orbitals[:, :2])

        def small():
            ctx.set_orbitals(u)
            return [ctx.ubkwbk_hwbk(u, u[:, :1], 0.1), *ctx.rk4_run(A, A, 1e-4), ctx.GS_calculation(1, 2)["Etot"]]

        before = small()
        with _no_room():
            for call in (lambda: ctx.ubkwbk_hwbk(u, orbitals, 0.1), lambda: ctx.rk4_run(np.zeros(1 << 21), np.zeros(1 << 21), 1e-4),
                         lambda: ctx.GS_calculation(1, 32)):
                with pytest.raises(MattohfError) as e:
                    call()
                assert e.value.status == _capi.ERR_ALLOC
        for a, b in zip(small(), before):
            assert np.array_equal(a, b)
