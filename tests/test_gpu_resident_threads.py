"""Contexts of different sizes stepping at once from several host threads (each
context in one thread): their resident kernels share the kernel's attributes on
the device, so each must launch, and give what it gives alone."""
import threading

import numpy as np
import pytest

from epi_b200 import capi
from epi_b200 import tissue as T

pytestmark = pytest.mark.gpu

FP64, MIXED = capi.EPI_PREC_FP64, capi.EPI_PREC_MIXED


def small():
    return [T.layered_tissue(16, 2, 1)], 400, {}


def wide():
    return [T.layered_tissue(96, 6, 2)], 120, {}


def turns():  # as much shared memory per block as a plan takes
    return [T.mixed_state_tissue(k) for k in range(40)], 40, dict(max_conn=96, max_cand=192)


def step_all(make, precision):
    tissues, calls, cfg = make()
    with capi.Context(precision=precision, skin=0.05, **cfg) as ctx:
        ctx.upload(tissues)
        for _ in range(calls):
            ctx.step(1)
        return ctx.positions()


@pytest.mark.parametrize("precision", [FP64, MIXED])
def test_contexts_in_threads_step_as_alone(built, precision):
    forms = (small, wide, turns)
    alone = [step_all(f, precision) for f in forms]
    got, failed = [None] * len(forms), []

    def work(k):
        try:
            got[k] = step_all(forms[k], precision)
        except Exception as e:  # reported below, in the test's own thread
            failed.append((forms[k].__name__, e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(forms))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for a, b in zip(alone, got):
        for u, v in zip(a, b):
            assert np.array_equal(u, v)
