"""The streaming stage kernel's bounded waits. (tests/test_timeout_gpu.py's case is a small grid, whose steps run in the
whole-step kernel: there the switch withholds a block's barrier arrivals.)

With a tile shape asked for, a small grid runs the streaming kernel, and the switch of nsf_debug_wait_limit makes its
producer issue none of its epilogue loads: the column warps' waits for them run out after a few thousand polls, raise the
block's abort flag, which ends the staging warps' waits, and the producer waits, bounded, for the copies it did issue.
Nothing faults or hangs; nsf_sync reports NSF_ERR_TIMEOUT, and a fresh solver runs as before. A grid with a body takes
the staging loop that looks up filter nodes, one without the plain one; both tile shapes."""
import numpy as np
import pytest

import nsfsi
from test_step_kernel_gpu import config

TIMEOUT = 5  # NSF_ERR_TIMEOUT


@pytest.mark.gpu
@pytest.mark.parametrize("tile", ["32x8", "16x16"])
@pytest.mark.parametrize("flow,steps", [("sphere", 1), ("sphere", 3), ("tgv", 1)])
def test_withheld_epilogue_loads_time_out_and_are_reported(flow, steps, tile, monkeypatch):
    cfg = config(flow, (33, 31, 29), 9)
    with nsfsi.Solver(cfg) as w:  # the whole-step kernel's result, which the streaming kernel's equals
        w.march(4)
        w.sync()
        ref = w.download()
    monkeypatch.setenv("NSF_STAGE_TILE", tile)
    with nsfsi.Solver(cfg) as s:
        assert s.launches_per_step() > 1
        s.debug_wait_limit(polls=4096, withhold_epilogue=True)
        s.march(steps)
        for _ in range(2):  # the flag is sticky
            with pytest.raises(nsfsi.NsfError) as e:
                s.sync()
            assert e.value.code == TIMEOUT, e.value
    with nsfsi.Solver(cfg) as s:
        s.march(4)
        s.sync()
        assert np.array_equal(s.download(), ref, equal_nan=True)
