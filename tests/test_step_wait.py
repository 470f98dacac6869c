"""The lock-step plan on chains so long that a solve takes longer than the
second after which a wait gives up."""
import numpy as np
import pytest

import lap_gb300 as gb


@pytest.mark.parametrize("elem,step_ns", [(8, 125), (4, 68)])  # as measured on a path of 100,000
def test_no_tile_waits_a_second(elem, step_ns):
    """The tiles that run at once wait for one another: their steps together,
    on a chain as long as they are, take less than half of that second."""
    for n in (3_000_000, 9_000_000):
        ia = np.clip(3 * np.arange(n + 1) - 1, 0, 3 * n - 2).astype(np.int32)
        cols = np.arange(n)[:, None] + np.array([-1, 0, 1])
        ja = cols[(cols >= 0) & (cols < n)].astype(np.int32)
        info = np.zeros(12, np.int32)
        assert gb.lib().gb_debug_step_plan(n, ia.ctypes.data, ja.ctypes.data, 1, elem, 0, info.ctypes.data, *[None] * 6) == 0
        assert min(int(info[0]), 152) * int(info[6]) * step_ns < 0.5e9
