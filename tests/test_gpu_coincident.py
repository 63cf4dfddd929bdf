"""Two cells at the same place: the pair coefficient is infinite, which is the
reference's abort (cell_interaction.cpp:51-55) and EPI_ERR_COEF_RANGE here,
naming both cells, in the resident kernel as in the kernel sequence. Laws: two
ALIVE cells, two dermis cells (whose softened law divides by the distance), a
FIX pair, a dividing pair (whose spring does)."""
import numpy as np
import pytest

from epi_b200 import capi
from epi_b200 import tissue as T

pytestmark = pytest.mark.gpu

FP64, MIXED = capi.EPI_PREC_FP64, capi.EPI_PREC_MIXED


def place(t, i, j):
    t.x[j], t.y[j], t.z[j] = t.x[i], t.y[i], t.z[i]
    t.radius[j] = t.radius[i]
    return t, {i, j}


def alive():
    t = T.config1()
    return place(t, t.nmemb + 10, t.nmemb + 11)


def general(state, k=0):
    """The first two unpaired cells of a state in the tissue of every state."""
    t = T.mixed_state_tissue()
    c = np.flatnonzero((t.state == state) & (t.pair < 0))[k:k + 2]
    return place(t, int(c[0]), int(c[1]))


def dividing():
    """A pair far above everything else: the spring alone acts between them
    beyond the connection's own law."""
    t = T.mixed_state_tissue()
    i = int(np.flatnonzero((t.state == T.ALIVE) & (t.pair >= 0))[0])
    return place(t, i, int(t.pair[i]))


CASES = {"alive": alive, "alive in all states": lambda: general(T.ALIVE),
         "dermis": lambda: general(T.DER), "stem": lambda: general(T.FIX), "dividing": dividing}


def error_of(t, mode, precision):
    with capi.Context(precision=precision, max_conn=96, max_cand=192) as ctx:
        ctx.upload([t])
        with pytest.raises(capi.EpiError) as e:
            ctx.step(1, mode)
        info = ctx.error_info()
        return e.value.code, {info["particle"], info["other"]}, info["value"]


@pytest.mark.parametrize("mode", ["eager", "per_tissue"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_coincident_cells_fp64(built, name, mode):
    t, pair = CASES[name]()
    code, cells, value = error_of(t, mode, FP64)
    assert code == capi.EPI_ERR_COEF_RANGE
    assert cells == pair
    assert np.isinf(value)


@pytest.mark.parametrize("mode", ["eager", "per_tissue"])
@pytest.mark.parametrize("name", ["alive", "alive in all states", "stem"])
def test_coincident_cells_mixed(built, name, mode):
    t, pair = CASES[name]()
    code, cells, _ = error_of(t, mode, MIXED)
    assert code == capi.EPI_ERR_COEF_RANGE
    assert cells == pair
