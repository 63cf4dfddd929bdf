"""Which steps run resident (small batches: one kernel for a run of steps) and
which as the kernel sequence, told by epi_resident_count."""
import numpy as np
import pytest

from epi_b200 import capi
from epi_b200 import tissue as T

pytestmark = pytest.mark.gpu

FP64, MIXED = capi.EPI_PREC_FP64, capi.EPI_PREC_MIXED


def counted(ctx, steps, mode):
    """(kernels run, resident runs, kernels these stood for) of `steps` steps."""
    a = (ctx.kernels_run(),) + ctx.resident_count()
    ctx.step(steps, mode)
    b = (ctx.kernels_run(),) + ctx.resident_count()
    return tuple(v - u for u, v in zip(a, b))


def test_resident_runs_count_as_the_kernels_they_are(built):
    with capi.Context(precision=MIXED) as ctx:
        ctx.upload([T.config1()])
        assert counted(ctx, 10, "eager") == (1, 1, 80)
        assert counted(ctx, 1, "eager") == (1, 1, 8)
        ran, runs, stood_for = counted(ctx, 1100, "graph")  # two launches of at most 1,024 steps
        assert (ran, runs) == (2, 2) and stood_for >= 1100 * 3 + 550
        assert counted(ctx, 10, "per_tissue") == (80, 0, 0)


def test_a_batch_that_fills_the_gpu_steps_in_the_sequence(built):
    ts = [T.layered_tissue(64, 4, k) for k in range(7)]  # 143,360 particles
    with capi.Context(precision=MIXED) as ctx:
        ctx.upload(ts)
        assert counted(ctx, 2, "eager") == (16, 0, 0)
