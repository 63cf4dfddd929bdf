"""Gradients with candidate rows that only just fit max_cand: rows built at the
positions the forward steps build them at fit, those at the middle of the
recomputed steps do not. In the first case no particle moves skin/2 over the
run; in the second some do, so candidates are rebuilt on the way back."""
import numpy as np
import pytest

from epi_b200 import capi
from epi_b200 import tissue as T

pytestmark = pytest.mark.gpu


def still():  # rows of 25 up to step 8, of 26 from step 9 to 21
    return T.layered_tissue(16, 3, 1, jitter=0.1), 0.3, 25, 24


def moving():  # rows of 23 up to step 14, of 24 from step 15 to 23; rebuilt at step 4
    return T.layered_tissue(12, 4, 2, jitter=0.15), 0.2, 23, 32


@pytest.mark.parametrize("sequence", [False, True])
@pytest.mark.parametrize("case", [still, moving])
def test_rows_that_just_fit_the_forward_steps_do_for_the_gradient(built, case, sequence):
    t, skin, rows, steps = case()
    target = (t.x + 0.01, t.y, t.z + 0.02)
    cfg = dict(precision=capi.EPI_PREC_FP64, skin=skin, max_conn=16,
               **(dict(variant=3) if sequence else {}))

    def gradient(max_cand):
        with capi.Context(max_cand=max_cand, **cfg) as ctx:
            ctx.upload([t])
            loss, grad = ctx.adjoint(steps, target, checkpoint_every=steps)
            end = ctx.positions()
            ctx.step(5)
            return loss, grad, end, ctx.positions()

    with capi.Context(max_cand=rows - 1, **cfg) as ctx:  # the rows are as long as stated
        with pytest.raises(capi.EpiError) as e:
            ctx.upload([t])
        assert e.value.code == capi.EPI_ERR_LIST_OVERFLOW
    tight, wide = gradient(rows), gradient(96)
    assert np.allclose(tight[0], wide[0], rtol=1e-12, atol=0)
    assert np.allclose(tight[1], wide[1], rtol=1e-9, atol=1e-14)
    for a, b in zip(tight[2] + tight[3], wide[2] + wide[3]):
        assert np.max(np.abs(a - b)) <= 1e-12
