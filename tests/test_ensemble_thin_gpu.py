"""Ensemble members with fewer than four interior planes along i, which one work item covers: alone, where no chunk of
four planes exists, and beside a member of ordinary length. Each equals its own plain solve, bit for bit (change norms to
the grouping of their sums, 1e-12)."""
import numpy as np
import pytest

import nsfsi
from test_step_kernel_gpu import assert_same, config


@pytest.mark.gpu
@pytest.mark.parametrize("shapes", [[(3, 12, 9)], [(5, 12, 9)], [(3, 6, 5), (4, 9, 34), (5, 35, 7)],
                                    [(4, 12, 9), (30, 20, 22)]], ids=["one_plane", "three_planes", "thin", "mixed"])
def test_members_of_few_planes_equal_their_plain_solves(shapes):
    cfgs = [config("tgv", n, 9) for n in shapes]
    with nsfsi.Ensemble(cfgs) as e:
        e.march(9)
        e.sync()
        for q, c in enumerate(cfgs):
            with nsfsi.Solver(c) as s:
                s.march(9)
                s.sync()
                assert_same(s, e.member(q))
