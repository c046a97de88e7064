"""A served job's bytes do not depend on whether the library has been
initialised: a server's budget may be laid out with them before there is one."""
import os
import subprocess
import sys

import pytest

from tests.conftest import ROOT

SIZES = [(32, 32, 32), (96, 96, 96), (17, 40, 23), (20, 128, 40), (24, 250, 20), (24, 270, 20), (420, 20, 20), (128, 96)]
PRINT = """
from mantaflow_gb300.batch import PlumeServer, PLUME, DAM_BREAK
def show():
    print([PlumeServer.job_bytes(s, k) for s in %r for k in (PLUME, DAM_BREAK)])
show()
""" % (SIZES,)


def _run(code):
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "PYTHONPATH": ROOT})
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout.strip().split("\n")


def test_bytes_before_initialisation():
    """room for the cluster sweeps' diagonal and bits in level order: six bytes
    for each of ceil(ny / 16) x ceil(nz / 16) x 256 lines of whole chunks of levels"""
    got = eval(_run(PRINT)[0])
    for (shape, plume) in zip(SIZES, got[::2]):
        if len(shape) < 3 or shape[1] > 256 or shape[0] > 400:
            continue
        nx, ny, nz = shape
        n = nx * ny * nz
        levels = (nx + 14 + 7) // 8 * 8
        floats = -(-ny // 16) * -(-nz // 16) * 256 * levels
        scene = n * (4 + 24 + 8 + 16 + 24 + 2)  # flags, two velocities and densities, advection's scratch, CG vectors, codes
        need = scene + 6 * floats + (8 * floats if 2 * floats > 4 * n else 0)
        assert plume >= need, shape


@pytest.mark.gpu
def test_bytes_before_and_after_initialisation():
    before, after = _run(PRINT + "from mantaflow_gb300._lib import ensure_init\nensure_init()\nshow()\n")
    assert before == after
