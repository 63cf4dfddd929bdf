"""The cell-map stamp over its windows: grids finer, coarser and uneven per
axis, so a particle's window is cut at the floor and the ceiling, wraps round
one side or both, and its columns leave a remainder for the lanes that share
it. The maps and the stimulus must be the oracle's, bit for bit, on the same
positions.
"""
import numpy as np
import pytest

from epi_b200 import capi
from epi_b200 import tissue as T
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def spread():
    """The all-states field tissue with cells moved to the box's sides, its
    floor and its ceiling."""
    t = T.field_tissue()
    cells = np.arange(t.nmemb, t.n)
    t.x[cells[0::7]] = 0.01
    t.x[cells[1::7]] = t.lx - 0.01
    t.y[cells[2::7]] = 0.0
    t.y[cells[3::7]] = t.ly - 1e-9
    t.z[cells[4::7]] = 0.3
    t.z[cells[5::7]] = t.lz - 3.0
    return t


@pytest.mark.parametrize("grid", [(32, 32, 64), (21, 34, 41), (45, 30, 29), (67, 70, 90)])
def test_maps_over_uneven_grids(built, grid):
    t = spread()
    ora = O.OracleTissue(t)
    fld = O.OracleField(ora, *grid)
    with capi.Context(precision=capi.EPI_PREC_FP64, max_conn=96, max_cand=192) as ctx:
        ctx.upload([T.field_tissue()])
        ctx.field_init(*grid)
        for _ in range(3):
            ctx.set_positions(*ora.positions())
            rc, zz = fld.step()
            assert rc == 0
            ctx.field_step(1)
        m1, m2, ex, gzz = ctx.field(0)
        o1, o2, oex = fld.get()
        assert gzz == zz
        assert np.array_equal(m1, o1) and np.array_equal(m2, o2) and np.array_equal(ex, oex)
        assert (o1 >= 0).any() and len(np.unique(o2)) > 1
