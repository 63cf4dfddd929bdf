"""Every form of the candidate rebuild on the same tissues.

The search takes a thread per particle or a group of 32, 16, 8 or 4 lanes,
by the number of particles to rebuild; all of them must leave the same rows in
the same order, so the steps that follow are the same bits. Sizes lie on
either side of the lines between the forms (32 lanes up to 9,472 particles of
a 148 SM device, 16 up to 18,944, 8 up to 37,888), with even and odd grids.

Bins hold about six particles at unit spacing; a tissue at half the spacing
and radii puts some fifty into each, the sort's case of more than one pass of
its lanes. Its connections are compared with all pairs taken one by one.
"""
import numpy as np
import pytest

from epi_b200 import capi
from epi_b200 import tissue as T

pytestmark = pytest.mark.gpu

FP64, MIXED = capi.EPI_PREC_FP64, capi.EPI_PREC_MIXED


def run(tissues, switch, precision, steps, **cfg):
    with capi.Context(precision=precision, skin=0.05, search_switch=switch, **cfg) as ctx:
        ctx.upload(tissues)
        first = ctx.connections()
        ctx.step(steps, "per_tissue")  # the kernel sequence
        return first, ctx.connections(), ctx.positions(), ctx.rebuild_count()


@pytest.mark.parametrize("side,layers", [(16, 2), (43, 4), (44, 4), (61, 4), (62, 4), (67, 7),
                                         (69, 7), (71, 9)])
def test_search_forms_leave_the_same_rows(built, side, layers):
    ts = [T.layered_tissue(side, layers, side)]
    precision = FP64 if side % 2 else MIXED
    groups, threads = run(ts, 1 << 30, precision, 12), run(ts, 1, precision, 12)
    assert threads[3] > 1
    for a, b in zip(groups[:2], threads[:2]):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    for a, b in zip(groups[2], threads[2]):
        assert np.array_equal(a, b)


def halved():
    t = T.layered_tissue(24, 9, 3)
    for k in ("x", "y", "z", "radius"):
        setattr(t, k, getattr(t, k) * 0.5)
    t.lx, t.ly = t.lx * 0.5, t.ly * 0.5
    return t


def all_pairs(t):
    """Connections of every particle, one pair at a time (connect_proc's test)."""
    lt, n = t.params.lj_thresh, t.n
    rows = []
    for i in range(n):
        d = t.x[i] - t.x
        dx = np.where(d > 0.5 * t.lx, d - t.lx, np.where(d <= -0.5 * t.lx, d + t.lx, d))
        d = t.y[i] - t.y
        dy = np.where(d > 0.5 * t.ly, d - t.ly, np.where(d <= -0.5 * t.ly, d + t.ly, d))
        dz = t.z[i] - t.z
        rs = t.radius[i] + t.radius
        near = dx * dx + dy * dy + dz * dz <= lt * lt * rs * rs
        near[i] = False
        if i < t.nmemb:
            near[:t.nmemb] = False
        rows.append(np.flatnonzero(near))
    return rows


@pytest.mark.parametrize("switch", [1, 1 << 30])
def test_crowded_bins(built, switch):
    t = halved()
    ref = all_pairs(t)
    with capi.Context(precision=FP64, search_switch=switch) as ctx:
        ctx.upload([t])
        off, idx = ctx.connections()
    links = t.nadj if hasattr(t, "nadj") else 4
    for i in range(t.n):
        row = idx[off[i]:off[i + 1]]
        if i < t.nmemb:
            row = row[links:]  # the lattice's come first
        assert np.array_equal(np.sort(row), ref[i]), i
