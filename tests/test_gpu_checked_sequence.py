"""The bounds-checked build on the kernel sequence: the kernels that batches
beyond the resident kernel's limit run, with a thread per particle. On small
tissues of every kind a named step-kernel form or epi_step_per_tissue takes
that path; one batch is large enough by itself. The build must report nothing
and give the release build's results."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from epi_b200 import build as B
from epi_b200 import capi
from epi_b200 import tissue as T
from tests.test_gpu_checked_build import CASES

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
# (mode, configuration): every step-kernel form, both rebuild nodes
FORMS = {"per_tissue": ("per_tissue", {}), "shared 8": ("eager", dict(variant=1)),
         "shared 15": ("graph", dict(variant=2)), "registers 3": ("eager", dict(variant=3)),
         "node": ("graph", dict(variant=4, rebuild_gate=1)), "launched": ("graph", dict(rebuild_gate=2))}


def large():
    return [T.layered_tissue(64, 4, k) for k in range(6)] + [T.tri_layered_tissue(64, 66, 4, 9)]


def runs():
    for name, make in CASES.items():
        for prec in (capi.EPI_PREC_FP64, capi.EPI_PREC_MIXED):
            for form, (mode, cfg) in FORMS.items():
                yield f"{prec}/{name}/{form}", make, prec, mode, cfg, 12
    for prec in (capi.EPI_PREC_FP64, capi.EPI_PREC_MIXED):
        for mode in ("eager", "graph"):
            yield f"{prec}/large/{mode}", large, prec, mode, {}, 6


RUNNER = r"""
import sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from epi_b200 import capi
from tests.test_gpu_checked_sequence import runs
out = {}
for key, make, prec, mode, cfg, steps in runs():
    with capi.Context(precision=prec, max_conn=96, max_cand=192, skin=0.05, **cfg) as ctx:
        ctx.upload(make())
        ctx.step(steps, mode)
        assert ctx.resident_count()[0] == 0, key
        out[key + "/x"] = np.stack(ctx.positions())
        out[key + "/offsets"], out[key + "/idx"] = ctx.connections()
np.savez(sys.argv[2], **out)
"""


def run(lib, path):
    env = dict(os.environ, EPI_MECH_LIB=str(lib))
    r = subprocess.run([sys.executable, "-c", RUNNER, str(ROOT), str(path)], env=env,
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-3000:]
    return np.load(path)


def test_checked_build_on_the_kernel_sequence(built, tmp_path):
    got = run(B.build_library(check=True), tmp_path / "checked.npz")
    ref = run(B.LIB, tmp_path / "release.npz")
    assert sorted(got.files) == sorted(ref.files)
    for k in ref.files:
        if k.endswith("/x"):
            # as for the resident runs: rounding of the two builds
            tol = 1e-12 if k.startswith(f"{capi.EPI_PREC_FP64}/") else 1e-8
            assert np.max(np.abs(got[k] - ref[k])) <= tol, k
        else:
            assert np.array_equal(got[k], ref[k]), k
