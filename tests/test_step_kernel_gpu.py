"""The whole-step kernel of small grids (nsf_step.cu) against the launch sequence of the general path.

A plain small solver runs its steps inside one launch; a one-member ensemble of the same case runs the streaming
stage kernel and the fused boundary kernel. Both use the same per-node arithmetic, so every field, t, dt and the
dt history are equal bit for bit; the change norms are sums in another grouping (a handful of roundings of sums of
squares: 1e-12)."""
import numpy as np
import pytest

import nsfsi


def config(flow, n, steps, end_time=None, filt=4):
    if flow == "shipped":
        c = nsfsi.config_defaults()
        c.stop_criterion = 0
        c.lz = 0.05 * (n[2] - 2)
    else:
        c = nsfsi.config_load(nsfsi.case_path("tgv256" if flow == "tgv" else "sphere48"))
    c.NI, c.NJ, c.NK = n
    c.stop_time_level = steps
    c.n_filter_intervals, c.n_filter_change_times = 1, 0
    c.filter_intervals[0] = filt
    if flow in ("sphere", "walls"):
        h = 1.0 / min(n[1] - 3, n[2] - 2)
        c.lx, c.ly, c.lz = h * (n[0] - 1), h * (n[1] - (3 if flow == "walls" else 2)), h * (n[2] - 2)
        c.spheres[0] = nsfsi.Sphere(0.4 * c.lx, 0.5 * c.ly, 0.5 * c.lz, 3.2 * h)
        if flow == "walls":
            c.bc[1][0] = c.bc[1][1] = nsfsi.BC["symmetry"]
    if end_time is not None:
        c.stop_criterion, c.t_end = 1, end_time
    c.machine_precision_buffer = float(np.finfo(np.float64).eps) * (c.lx + c.ly + c.lz)
    return c


def assert_same(plain, member):
    assert plain.time() == member.time()
    got, ref = plain.download(), member.download()
    for f in range(12):
        assert np.array_equal(got[f], ref[f], equal_nan=True), nsfsi.FIELDS[f]
    a, b = plain.history(), member.history()
    assert np.array_equal(a[:, :2], b[:, :2])
    assert np.all(np.abs(a[:, 2:] - b[:, 2:]) <= 1e-12 * np.abs(b[:, 2:]))


# (grid: one tile exactly, one node more, the smallest grids the streaming kernel runs, thin grids up to and past
# the thin tile, a chunk remainder, a grid near the path's limit)
CASES = [("tgv", (18, 10, 18)), ("tgv", (19, 11, 19)), ("tgv", (6, 8, 5)), ("tgv", (33, 29, 45)), ("tgv", (81, 80, 82)),
         ("shipped", (41, 23, 3)), ("shipped", (41, 23, 6)), ("shipped", (41, 23, 7)), ("sphere", (33, 31, 29)),
         ("sphere", (48, 48, 48)), ("walls", (40, 29, 35))]


@pytest.mark.gpu
@pytest.mark.parametrize("flow,n", CASES, ids=["%s_%dx%dx%d" % ((f,) + n) for f, n in CASES])
def test_equals_the_launch_sequence(flow, n):
    cfg = config(flow, n, 9)
    with nsfsi.Solver(cfg) as s, nsfsi.Ensemble([cfg]) as e:
        assert s.launches_per_step() == 1
        s.march(4)
        s.march(5)
        e.march(9)
        s.sync()
        e.sync()
        assert_same(s, e.member(0))


@pytest.mark.gpu
@pytest.mark.parametrize("tile", ["32x8", "16x16"])
@pytest.mark.parametrize("flow,n", [("sphere", (40, 47, 45)), ("walls", (37, 39, 50)), ("shipped", (61, 33, 3))],
                         ids=["sphere", "walls", "shipped"])
def test_streaming_kernel_with_bodies(flow, n, tile, monkeypatch):
    """The streaming kernel's staging of body planes, per tile shape: bodies that lie across tile edges."""
    cfg = config(flow, n, 9, filt=3)
    with nsfsi.Solver(cfg) as s:
        monkeypatch.setenv("NSF_STAGE_TILE", tile)
        with nsfsi.Solver(cfg) as g:
            assert s.launches_per_step() == 1 < g.launches_per_step()
            s.march(9)
            g.march(9)
            assert_same(s, g)


@pytest.mark.gpu
def test_many_steps_and_the_end_time_stop():
    """More steps than one launch takes, and steps past t_end, which are no-ops."""
    cfg = config("sphere", (30, 29, 31), 200, end_time=0.5)
    with nsfsi.Solver(cfg) as s, nsfsi.Ensemble([cfg]) as e:
        s.march(140)
        e.march(140)
        t, level, _ = s.time()
        assert t == 0.5 and 64 < level < 140
        assert_same(s, e.member(0))


@pytest.mark.gpu
def test_two_solvers_side_by_side():
    """Whole-step launches of two handles queued without waiting: each equals its own run alone."""
    cfgs = [config("sphere", (34, 30, 33), 40), config("walls", (37, 31, 30), 40)]
    alone = []
    for c in cfgs:
        with nsfsi.Solver(c) as s:
            s.march(40)
            alone.append(s.download())
    with nsfsi.Solver(cfgs[0]) as a, nsfsi.Solver(cfgs[1]) as b:
        for _ in range(8):
            a.march(5)
            b.march(5)
        for s, ref in ((a, alone[0]), (b, alone[1])):
            s.sync()
            assert np.array_equal(s.download(), ref, equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("flow,first,second", [("tgv", (81, 80, 82), (19, 11, 19)), ("shipped", (161, 83, 3), (21, 12, 3)),
                                               ("sphere", (64, 60, 62), (30, 20, 20))], ids=["tgv", "thin", "sphere"])
def test_a_later_smaller_handle_leaves_an_earlier_one_alone(flow, first, second):
    """The kernel's shared-memory limit is a property of the function: a handle whose plan takes less, created after
    one whose plan takes more, must not lower it (and the other way round)."""
    big, small = config(flow, first, 3), config(flow, second, 3)
    with nsfsi.Solver(big) as s:
        s.march(3)
        ref = s.download()
    with nsfsi.Solver(big) as a, nsfsi.Solver(small) as b:
        a.march(3)
        b.march(3)
        a.sync()
        b.sync()
        assert a.launches_per_step() == b.launches_per_step() == 1
        assert np.array_equal(a.download(), ref, equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("tile", [None, "32x8"], ids=["whole_step", "streaming"])
def test_reynolds_numbers_without_viscosity(tile, monkeypatch):
    """The viscosity squares the Reynolds number: values whose square overflows run as ones that only make the viscous
    terms vanish against the last bit of the others."""
    if tile:
        monkeypatch.setenv("NSF_STAGE_TILE", tile)
    fields = []
    for re in (1e60, 1e200, 1e300):
        cfg = config("tgv", (24, 21, 23), 5)
        cfg.re = re
        with nsfsi.Solver(cfg) as s:
            s.march(5)
            s.sync()
            fields.append(s.download(range(5)))
    assert np.all(np.isfinite(fields[0]))
    assert np.array_equal(fields[0], fields[1]) and np.array_equal(fields[0], fields[2])
