"""A handle whose whole-step run gave up at a barrier, then used for an adjoint run, which starts it over from level 0.

The withheld arrivals leave the barrier's counter at no multiple of the block count. The adjoint's reset puts the control
block back to its initial state, the time-out flag with it, so it must put the counter back too: else blocks compute
different targets and barriers pass early, unreported. J, the dt sequence and the gradients are those of a handle that
never timed out, bit for bit (the adjoint is deterministic)."""
import numpy as np
import pytest

import nsfsi
from test_step_kernel_gpu import config

TIMEOUT = 5  # NSF_ERR_TIMEOUT


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [1, 3])
def test_adjoint_run_after_a_timed_out_march(steps):
    cfg = config("sphere", (33, 31, 29), 12)
    got = []
    for spoil in (False, True):
        with nsfsi.Solver(cfg) as s:
            assert s.launches_per_step() == 1
            if spoil:
                s.debug_wait_limit(polls=4096, withhold_epilogue=True)
                s.march(steps)
                with pytest.raises(nsfsi.NsfError) as e:
                    s.sync()
                assert e.value.code == TIMEOUT, e.value
            s.adj_configure(4, 5)
            J = s.adj_forward()
            got.append((J, s.adj_dt()) + s.adj_backward())
    (J0, dt0, gi0, gu0), (J1, dt1, gi1, gu1) = got
    assert np.isfinite(J0) and J0 != 0
    assert J1 == J0
    assert np.array_equal(dt1, dt0) and np.array_equal(gi1, gi0) and np.array_equal(gu1, gu0)
