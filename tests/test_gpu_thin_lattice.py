"""Membranes three particles wide, so long that a resident run (which keeps
column and row of a membrane particle in 16 bits each) meets rows from 32,768
on: against the kernel sequence, bit for bit, and the oracle. The three columns
stand on a triangle, so that neighbours are nearer than half the box from each
other; one DER cell far below makes the batch general, and the rows lie close, as
those of a batch of every state do: the form that takes this many membrane
particles per block."""
import numpy as np
import pytest

from epi_b200 import capi
from epi_b200 import tissue as T
from oracle import oracle as O
from tests.helpers import rel_pos_err

pytestmark = pytest.mark.gpu

STEPS = 4


def thin(rows, lattice):
    s, nm = 0.05, 3 * rows
    jj, kk = np.meshgrid(np.arange(3), np.arange(rows), indexing="xy")
    jj, kk = jj.ravel(), kk.ravel()
    jit = (2.0 * T.splitmix64_uniform(rows, 3 * nm).reshape(nm, 3) - 1.0) * s / 36
    x = np.append(3.0 + np.array([0.0, s, s / 2])[jj] + jit[:, 0], 4.0)
    y = np.append((kk + 0.5) * s + jit[:, 1], 4.0)
    z = np.append(8.0 + np.array([0.0, 0.0, s * 0.75 ** 0.5])[jj] + jit[:, 2], 1.5)
    n = nm + 1
    # constants for the small spacing: displacements per step as at 1.8
    p = T.Params(der_der_const=0.2 * s / 1.8, kbend=0.5 * (s / 1.8) ** 2,
                 eps_m=0.01 * (s / 1.8) ** 2)
    t = T.Tissue(nmx=3, nmy=rows, lx=10.0, ly=rows * s, lz=20.0, x=x, y=y, z=z,
                 radius=np.append(np.full(nm, 1.3 / 1.8 * s), 1.4),
                 state=np.append(np.full(nm, T.MEMB), T.DER).astype(np.uint8),
                 agek=np.zeros(n), spr_nat_len=np.zeros(n), pair=np.full(n, -1, np.int32),
                 rest_div_times=np.zeros(n, np.int32), nmemb=nm, nder=1, lattice=lattice,
                 params=p)
    t.validate()
    return t


@pytest.mark.parametrize("precision", [capi.EPI_PREC_FP64, capi.EPI_PREC_MIXED])
@pytest.mark.parametrize("rows,lattice", [(32780, T.SQUARE), (32800, T.SQUARE),
                                          (32800, T.TRIANGULAR), (43600, T.SQUARE)])
def test_rows_beyond_15_bits(built, rows, lattice, precision):
    t = thin(rows, lattice)
    # 43,600 rows' FP64 terms are beyond a block's shared memory: the sequence
    fits = rows < 43600 or precision == capi.EPI_PREC_MIXED
    got = []
    for mode in ("eager", "per_tissue"):
        with capi.Context(precision=precision, max_cand=256) as ctx:
            ctx.upload([t])
            ctx.step(STEPS, mode)
            assert ctx.resident_count()[0] == (1 if fits and mode == "eager" else 0)
            got.append(ctx.positions())
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    if precision == capi.EPI_PREC_FP64:
        ora = O.OracleTissue(t)
        assert ora.step(STEPS) == 0
        assert rel_pos_err(got[0], ora.positions(), t.lx, t.ly) <= 1e-10  # the parity tests' FP64 bound
