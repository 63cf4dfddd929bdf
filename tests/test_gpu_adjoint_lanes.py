"""The adjoint's split over lanes and its candidate reach, against the oracle's
forward-mode gradient: sizes on either side of each lane count's range, a
checkpoint interval over which particles outrun candidates built at its
middle (a small skin), both lattices in one batch on every lane count.

Bar: 1e-6 relative per component against the oracle (as the other adjoint
tests), 1e-10 between single and batched runs.
"""
import numpy as np
import pytest

from epi_b200 import capi
from epi_b200 import tissue as T
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def gradient(tissues, steps, shift=0.02, **cfg):
    with capi.Context(precision=capi.EPI_PREC_FP64, **cfg) as ctx:
        ctx.upload(tissues)
        tgt = [np.concatenate([getattr(t, k) for t in tissues]) for k in "xyz"]
        tgt[0] = tgt[0] + shift
        return ctx.adjoint(steps, tgt, checkpoint_every=20)


def reference(t, steps, shift=0.02):
    return O.tangent_gradient(t, steps, target=(t.x + shift, t.y, t.z))


@pytest.mark.parametrize("side,layers", [(23, 5), (41, 9), (43, 9)])  # 3174, 16810, 18490
def test_lane_counts_match_the_oracle(built, side, layers):
    t = T.layered_tissue(side, layers, side)
    loss, grad = gradient([t], 30)
    rloss, rgrad, _ = reference(t, 30)
    assert loss[0] == pytest.approx(rloss, rel=1e-9)
    assert np.allclose(grad[0], rgrad, rtol=1e-6, atol=1e-9 * np.abs(rgrad).max())


@pytest.mark.parametrize("skin", [0.004, 0.02, 0.5])
def test_positions_that_outrun_the_candidates(built, skin):
    t = T.config1(5)
    loss, grad = gradient([t], 50, skin=skin)
    rloss, rgrad, _ = reference(t, 50)
    assert loss[0] == pytest.approx(rloss, rel=1e-9)
    assert np.allclose(grad[0], rgrad, rtol=1e-6, atol=1e-9 * np.abs(rgrad).max())


def test_large_mixed_lattice_batch_equals_single_runs(built):
    """Two lanes per particle (beyond 262,144 particles), the triangular
    lattice's exchange beside square tissues, the kernel sequence."""
    big = T.layered_tissue(128, 15, 3)
    tri = T.tri_layered_tissue(16, 18, 2, 0)
    small = T.config1(6)
    loss, grad = gradient([big, tri, small], 8)
    for k, t in enumerate((tri, small), start=1):
        l1, g1 = gradient([t], 8)
        assert loss[k] == pytest.approx(l1[0], rel=1e-12)
        assert np.allclose(grad[k], g1[0], rtol=1e-10, atol=1e-13 * np.abs(g1).max())
        rl, rg, _ = reference(t, 8)
        assert np.allclose(grad[k], rg, rtol=1e-6, atol=1e-9 * np.abs(rg).max())
