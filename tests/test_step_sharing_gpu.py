"""Several small handles whose steps are in flight at once: they take a half or a quarter of the SMs each, or the launch
sequence above 120,000 nodes, and alone all of them. Whichever way the steps of a handle go, and in whatever mixture,
fields, t, dt and the dt history are those of the handle run alone, bit for bit; the change norms are sums in another
grouping (a handful of roundings of sums of squares: 1e-12)."""
import threading

import numpy as np
import pytest

import nsfsi
from test_step_kernel_gpu import assert_same, config

# (a cube with a body, walls, the thin tile, the cube tile on a thin grid with more tiles a block than it keeps in
# shared memory at a quarter of the SMs, and a grid above the limit)
CASES = [("sphere", (34, 30, 33)), ("walls", (37, 31, 30)), ("shipped", (61, 33, 3)), ("tgv", (3, 5200, 7)),
         ("tgv", (54, 50, 49))]


@pytest.mark.gpu
@pytest.mark.parametrize("handles", [2, 3, 5])
@pytest.mark.parametrize("flow,n", CASES, ids=["%s_%dx%dx%d" % ((f,) + n) for f, n in CASES])
def test_handles_at_once_equal_a_handle_alone(flow, n, handles):
    cfg = config(flow, n, 100)
    with nsfsi.Solver(cfg) as ref:
        ref.march(38)
        ref.sync()
        hs = [nsfsi.Solver(cfg) for _ in range(handles)]
        try:
            hs[0].march(3)  # alone, and waited for
            hs[0].sync()
            for s in hs[1:]:
                s.march(3)
            for _ in range(5):  # in turn, nobody waits
                for s in hs:
                    s.march(5)
            for s in hs:
                s.sync()
            for s in hs:  # one call each: the first now expects the others
                s.march(10)
            for s in hs:
                s.sync()
                assert_same(s, ref)
        finally:
            for s in hs:
                s.close()


@pytest.mark.gpu
def test_handles_in_threads_and_an_adjoint_run_beside_them():
    cfg = config("sphere", (33, 31, 29), 30)
    with nsfsi.Solver(cfg) as s:
        s.march(30)
        s.sync()
        ref = s.download()
    with nsfsi.Solver(cfg) as s:
        s.adj_configure(4, 5)
        J = s.adj_forward()
        gi, gu = s.adj_backward()
    got = {}

    def march(q):
        with nsfsi.Solver(cfg) as s:
            for _ in range(30):
                s.march(1)
                s.time()
            got[q] = s.download()

    def adjoint():
        with nsfsi.Solver(cfg) as s:
            s.adj_configure(4, 5)
            got["J"] = s.adj_forward()
            got["g"] = s.adj_backward()

    threads = [threading.Thread(target=march, args=(q,)) for q in range(3)] + [threading.Thread(target=adjoint)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for q in range(3):
        assert np.array_equal(got[q], ref, equal_nan=True)
    assert got["J"] == J and np.array_equal(got["g"][0], gi) and np.array_equal(got["g"][1], gu)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["handle", "ensemble", "slabs"])
def test_small_handles_beside_large_steps(kind):
    """Small handles whose steps are queued beside those of a large grid, an ensemble or a slab group, and alone before
    and after."""
    small = [config("sphere", (34, 30, 33), 100), config("shipped", (61, 33, 3), 100)]
    big = config("tgv", (84, 82, 85), 100)
    ref, big_ref = [], None
    for c in small:
        with nsfsi.Solver(c) as s:
            s.march(24)
            s.sync()
            ref.append((s.download(), s.time()))
    with nsfsi.Solver(big) as s:
        assert s.launches_per_step() > 1
        s.march(12)
        s.sync()
        big_ref = s.download()
    large = {"handle": lambda: nsfsi.Solver(big), "ensemble": lambda: nsfsi.Ensemble([big]),
             "slabs": lambda: nsfsi.SlabGroup(big, 2)}[kind]()
    hs = [nsfsi.Solver(c) for c in small]
    try:
        for s in hs:
            s.march(4)
            s.sync()
        for _ in range(3):
            for s in hs:
                s.march(3)
            large.march(4)
            for s in hs:
                s.march(3)
        large.sync()
        for s in hs:
            s.sync()
        for s in hs:  # expects the large steps again, then finds none
            s.march(1)
            s.sync()
            s.march(1)
            s.sync()
        got = large.member(0).download() if kind == "ensemble" else large.download()
        assert np.array_equal(got, big_ref)
        for s, (fields, now) in zip(hs, ref):
            assert s.time() == now
            assert np.array_equal(s.download(), fields, equal_nan=True)
    finally:
        for s in hs:
            s.close()
        large.close()
