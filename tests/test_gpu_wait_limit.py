"""A bounded wait that gives up (epi_set_wait_limit, one poll: some block of a
resident run finds another not yet there and leaves): the call reports
EPI_ERR_TIMEOUT, steps are refused until the next upload, and after it the
context steps as a new one does, whether the run ended between steps or within
a candidate rebuild (whose bin counts it leaves behind)."""
import numpy as np
import pytest

from epi_b200 import capi
from epi_b200 import tissue as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", ["step", "rebuild"])
def test_a_wait_that_gives_up_needs_an_upload(built, where):
    ts = [T.layered_tissue(48, 3, k) for k in range(3)]
    with capi.Context(precision=capi.EPI_PREC_MIXED, skin=0.05) as ctx:
        ctx.upload(ts)
        ctx.step(5)
        if where == "rebuild":
            ctx.set_tuning(0.05, 0)  # flags every tissue
        ctx.set_wait_limit(1)
        with pytest.raises(capi.EpiError) as e:
            ctx.step(20)
        assert e.value.code == capi.EPI_ERR_TIMEOUT
        ctx.set_wait_limit()
        for call in (lambda: ctx.step(1), lambda: ctx.step(1, "per_tissue"), ctx.connect):
            with pytest.raises(capi.EpiError) as e:
                call()
            assert e.value.code == capi.EPI_ERR_STATE
        ctx.upload(ts)
        ctx.step(20)
        got = ctx.positions() + ctx.connections()
    with capi.Context(precision=capi.EPI_PREC_MIXED, skin=0.05) as ref:
        ref.upload(ts)
        ref.step(20)
        for a, b in zip(got, ref.positions() + ref.connections()):
            assert np.array_equal(a, b)
