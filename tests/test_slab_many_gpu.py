"""A slab group of more slabs in one process than the GPU holds blocks of the boundary kernel (148 SMs x 4): each slab
then runs its own launches. The fields and the dt sequence are the single-grid solve's, bit for bit, as with few slabs;
the change norms agree to the grouping of their sums (a few roundings: 1e-12)."""
import numpy as np
import pytest

import nsfsi
from test_step_kernel_gpu import config


@pytest.mark.gpu
def test_more_slabs_than_resident_boundary_blocks():
    nslabs, steps = 600, 6
    cfg = config("tgv", (2 * nslabs + 3, 7, 6), steps, filt=3)  # two planes a slab, one slab with three; a filter step
    with nsfsi.Solver(cfg) as s:
        s.march(steps)
        s.sync()
        ref, now, h = s.download(), s.time(), s.history()
    with nsfsi.SlabGroup(cfg, nslabs) as g:
        assert g.info()[0] == nslabs
        g.march(steps)
        g.sync()
        assert np.array_equal(g.download(), ref, equal_nan=True)
        for p in (0, 1, nslabs // 2, nslabs - 1):
            assert g.slab(p).time() == now
            hs = g.slab(p).history()
            assert np.array_equal(hs[:, :2], h[:, :2])
            assert np.all(np.abs(hs[:, 2:] - h[:, 2:]) <= 1e-12 * np.abs(h[:, 2:]).max())
