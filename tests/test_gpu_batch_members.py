"""Members of an ensemble used as contexts of their own between its runs (needs a GB300)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_fixed_point import _cfg, _functions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grow", ["longer run", "more functions", "gradient", "ground state"])
def test_batch_after_its_members_buffers_grew(built_lib, grow):
    """A member's own call may move buffers that the ensemble's arguments point to: the
    next run of the ensemble uses the new ones, with the same results."""
    from mattohf_gb300 import Batch
    shapes = [(5, 2), (3, 1), (4, 3)]
    nt, dt = 3, 0.003
    A = 0.02 * np.random.default_rng(8).standard_normal((len(shapes), nt))
    u0 = [_functions(64, NK, nb, NK) for NK, nb in shapes]
    with Batch([_cfg(64, NK, nb) for NK, nb in shapes]) as b:
        def run():
            for r, u in enumerate(u0):
                b[r].set_orbitals(u)
            return [*b.rk4_run(A, A, dt), *(b[r].get_orbitals() for r in range(len(u0)))]

        first = run()
        for r, (NK, nb) in enumerate(shapes):
            if grow == "longer run":
                b[r].rk4_run(np.zeros(500 + r), np.zeros(500 + r), 1e-3)
            elif grow == "more functions":
                b[r].ubkwbk_hwbk(u0[r], _functions(64, NK, 20, 2), 0.1)
            elif grow == "gradient":
                b[r].adjoint(np.zeros(40), 1e-3)
            else:
                b[r].GS_calculation(1, 4)
        keep = [b[r].ubkwbk_hwbk(u0[r], u0[r], 0.1) for r in range(len(shapes))]  # other work in what was freed
        for x, y in zip(run(), first):
            assert np.array_equal(x, y)
        del keep
