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


def paired(ts):
    """One dividing pair in the middle of the first tissue's cells."""
    t = ts[0]
    i = (t.nmemb + t.n) // 2
    t.pair[i], t.pair[i + 1] = i + 1, i
    t.spr_nat_len[i:i + 2] = 1.0
    return ts


# batches of up to 131,072 particles on either side of the line where the
# kernel sequence becomes the faster one in a run of 50 steps: (tissues, resident
# in FP64, in mixed precision)
def routes():
    tri = lambda side, layers, k: T.tri_layered_tissue(side, T.tri_rows(side), layers, k)
    return {
        "tri, few": (lambda: [tri(24, 3, k) for k in range(6)], True, True),
        "tri, wide": (lambda: [tri(50, 3, k) for k in range(6)], False, False),
        "one": (lambda: [T.layered_tissue(64, 8, 1)], True, True),
        "one, large": (lambda: [T.layered_tissue(120, 7, 1)], False, False),
        "a pair, small": (lambda: paired([T.layered_tissue(48, 5, 1)]), True, True),
        "a pair, many": (lambda: paired([T.layered_tissue(48, 3, k) for k in range(12)]), False, False),
        "a pair, tri": (lambda: paired([tri(48, 3, k) for k in range(10)]), False, False),
        "all states, 40": (lambda: [T.mixed_state_tissue(k) for k in range(40)], True, True),
        "all states, 100 tri": (lambda: [T.mixed_state_tissue(k, T.TRIANGULAR) for k in range(100)],
                                False, False),
    }


@pytest.mark.parametrize("name", sorted(routes()))
def test_the_faster_route_is_taken(built, name):
    make, *resident = routes()[name]
    ts = make()
    for precision, want in zip((FP64, MIXED), resident):
        with capi.Context(precision=precision, max_conn=96, max_cand=192) as ctx:
            ctx.upload(ts)
            assert counted(ctx, 50, "eager")[1] == (1 if want else 0), precision


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("named", [dict(variant=v) for v in (1, 2, 3, 4)] +
                         [dict(rebuild_gate=g) for g in (1, 2)])
def test_a_named_form_is_the_one_that_runs(built, named, precision):
    """A variant or a rebuild node in the configuration keeps a small batch in
    the kernel sequence, eager and graph; the results are the same bits."""
    ts = [T.mixed_state_tissue(2), T.layered_tissue(16, 2, 1), T.tri_layered_tissue(16, 18, 2, 0)]
    got = []
    for cfg in ({}, named):
        with capi.Context(precision=precision, skin=0.05, max_conn=96, max_cand=192, **cfg) as ctx:
            ctx.upload(ts)
            runs = [counted(ctx, 15, mode)[1] for mode in ("eager", "graph")]
            assert runs == ([0, 0] if cfg else [1, 1])
            got.append(ctx.positions() + ctx.connections())
    for a, b in zip(*got):
        assert np.array_equal(a, b)


def test_autotuner_times_the_resident_kernel_as_one_form(built):
    ts = [T.config1(k) for k in range(2)]
    with capi.Context(precision=MIXED) as ctx:
        ctx.upload(ts)
        runs = ctx.resident_count()[0]
        _, variant, _ = ctx.autotune(16)
        # six skins in the run loop, two launches each; the forms of the
        # sequence (four variants, two nodes) in none of theirs
        tried = ctx.resident_count()[0] - runs
        assert tried == 2 * (6 + (4 if variant == 0 else 0))
        cfg = ctx.config()
        assert cfg["variant"] == variant
        if variant == 0:
            assert cfg["rebuild_gate"] == 0
        assert counted(ctx, 4, "graph")[1] == (1 if variant == 0 else 0)
