"""Change norms of slab groups and ensembles: the same bits from run to run, and as close to a sum in extended precision as
a single grid's.

A norm is the square root of dx dy dz times a sum of squares. The terms' errors average out; what remains are the
roundings of the last additions of the trees (each within u = 2^-53, the square root halves them), of the product, of
dx dy dz and of the root: an rms of about u, 1.1e-16. Sums built by hundreds of additions one after another reach twice
that. 1.5 u is asked."""
import numpy as np
import pytest

import nsfsi
from test_step_kernel_gpu import config

GRIDS = [(40, 37, 50), (64, 60, 58), (33, 29, 45)]
STEPS = 8


def cases():
    out = []
    for n in GRIDS:
        c = config("tgv", n, 100, filt=1000)
        c.conv_history = 2
        out.append(c)
    return out


def errors(c, before, after, row):
    n = (int(c.NI), int(c.NJ), int(c.NK))
    d = (after - before).reshape(5, *n)[:, 1:-1, 1:-1, 1:-1].reshape(5, -1).astype(np.longdouble)
    h = [np.longdouble(L) / (m - 2) for L, m in zip((c.lx, c.ly, c.lz), n)]
    ref = np.sqrt(h[0] * h[1] * h[2] * (d * d).sum(1))
    return ((row - ref) / ref).astype(float)


def run_slabs(slabs):
    err, rows = [], []
    for c in cases():
        with nsfsi.SlabGroup(c, slabs) as g:
            for k in range(STEPS):
                before = g.download(range(5))
                g.march(1)
                g.sync()
                row = g.slab(0).history()[k, 2:]
                err.append(errors(c, before, g.download(range(5)), row))
                rows.append(row)
    return np.array(err), np.array(rows)


def run_ensemble():
    err, rows = [], []
    with nsfsi.Ensemble(cases()) as e:
        for k in range(STEPS):
            before = [e.member(q).download(range(5)) for q in range(len(GRIDS))]
            e.march(1)
            e.sync()
            for q, c in enumerate(cases()):
                row = e.member(q).history()[k, 2:]
                err.append(errors(c, before[q], e.member(q).download(range(5)), row))
                rows.append(row)
    return np.array(err), np.array(rows)


@pytest.mark.gpu
@pytest.mark.parametrize("run", [lambda: run_slabs(2), lambda: run_slabs(3), run_ensemble],
                         ids=["two_slabs", "three_slabs", "ensemble"])
def test_change_norms_are_accurate_and_repeatable(run):
    err, rows = run()
    rms = float(np.sqrt(np.mean(err ** 2)))
    print("rms %.3g, largest %.3g" % (rms, float(np.abs(err).max())))
    assert rms <= 1.5 * 2.0 ** -53
    assert np.array_equal(run()[1], rows)
