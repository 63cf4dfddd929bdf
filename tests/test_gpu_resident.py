"""Resident stepping (small batches: one cooperative kernel for a whole run)
against the kernel sequence, which epi_step_per_tissue always runs.

Both evaluate the same operations in the same order, so positions must agree
bit for bit, with candidate rebuilds along the way (a small skin forces
many). Forms: the smallest grid, sizes around the tiles a block is dealt,
both lattices, every cell state (long rows, several turns of a block's pair
terms, then of its membrane terms as well), up to eight tissues dealt tile by
tile over all blocks and more over groups of blocks, old cells, runs longer than one launch, one step per call.
"""
import numpy as np
import pytest

from epi_b200 import capi
from epi_b200 import tissue as T

pytestmark = pytest.mark.gpu

FP64, MIXED = capi.EPI_PREC_FP64, capi.EPI_PREC_MIXED
ALL = dict(max_conn=96, max_cand=192)


def aged(t):
    t.agek[t.nmemb:] = np.linspace(0.0, 6.0, t.n - t.nmemb)
    return t


def cases():
    small = T.layered_tissue
    return {
        "smallest": ([small(10, 1, 1)], 40, {}),
        "odd": ([small(17, 3, 2)], 40, {}),
        "tile+1": ([small(11, 2, 3), small(13, 1, 4)], 40, {}),
        "aged": ([aged(small(19, 2, 5))], 40, {}),
        "tri": ([T.tri_layered_tissue(16, 18, 2, 0)], 40, {}),
        "wide": ([small(64, 4, 6)], 30, {}),
        "eight": ([small(12 + k, 2, k) for k in range(8)], 30, {}),
        "eleven": ([small(12 + k, 2, k) for k in range(11)], 30, {}),
        "sixty": ([small(10 + k % 5, 1 + k % 3, k) for k in range(60)], 20, {}),
        "lattices": ([small(16, 2, 1), T.tri_layered_tissue(17, 20, 3, 2)], 30, {}),
        "all states": ([T.mixed_state_tissue(3)], 30, ALL),
        "all states tri": ([T.mixed_state_tissue(4, T.TRIANGULAR), small(16, 2, 7)], 30, ALL),
        "all states x 12": ([T.mixed_state_tissue(k) for k in range(12)], 20, ALL),
        "all states x 70": ([T.mixed_state_tissue(k, k % 2) for k in range(70)], 6, ALL),
        "all states x 40": ([T.mixed_state_tissue(k) for k in range(40)], 6, ALL),
        "long": ([small(12, 2, 8)], 1100, {}),
    }


def run(tissues, steps, mode, precision, cfg):
    with capi.Context(precision=precision, skin=0.05, **cfg) as ctx:
        ctx.upload(tissues)
        if mode == "each":
            for _ in range(steps):
                ctx.step(1)
        else:
            ctx.step(steps, mode)
        return ctx.positions(), ctx.rebuild_count(), ctx.connections(), ctx.dermis()


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("name", sorted(cases()))
def test_resident_steps_equal_the_kernel_sequence(built, name, precision):
    tissues, steps, cfg = cases()[name]
    ref = run(tissues, steps, "per_tissue", precision, cfg)
    for mode in ("eager", "graph") + (("each",) if steps <= 40 else ()):
        got = run(tissues, steps, mode, precision, cfg)
        for a, b in zip(ref[0], got[0]):
            assert np.array_equal(a, b), mode
        assert ref[1] == got[1], mode
        assert np.array_equal(ref[2][0], got[2][0]) and np.array_equal(ref[2][1], got[2][1])
        assert np.array_equal(ref[3], got[3])


def test_resident_errors_are_those_of_the_sequence(built):
    t = T.config1()
    k = t.nmemb
    t.x[k + 1], t.y[k + 1], t.z[k + 1] = t.x[k] + 0.3, t.y[k], t.z[k]
    for mode in ("eager", "graph", "per_tissue"):
        with capi.Context(precision=MIXED) as ctx:
            ctx.upload([t])
            with pytest.raises(capi.EpiError) as e:
                ctx.step(3, mode)
            assert e.value.code in (capi.EPI_ERR_COEF_RANGE, capi.EPI_ERR_BIN_RANGE), mode
            ctx.upload([T.config1()])  # usable afterwards
            ctx.step(5, mode)
