"""A batch with a scene too wide for a cluster: its sweeps by tiles and the other
scenes' cluster sweeps run beside each other."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

pytest.importorskip("mantaflow_gb300")
from mantaflow_gb300 import batch as mb  # noqa: E402

WIDE = (420, 40, 40)
OTHERS = [(64, 64, 64), (80, 80, 80), (48, 48, 48)]


def _run(sizes, steps, seeds):
    b = mb.BatchedPlumes(sizes, [(0, -4e-3, 0)] * len(sizes), seeds)
    for _ in range(3):
        b.step()
    b.sync()
    t = time.perf_counter()
    for _ in range(steps):
        b.step()
    b.sync()
    t = time.perf_counter() - t
    out = [(b.download(q, mb.PRESSURE), b.download(q, mb.VELOCITY), b.iterations(q)) for q in range(len(sizes))]
    b.close()
    return t, out


def test_scenes_alone_and_beside_the_wide_one():
    _, mixed = _run([WIDE] + OTHERS, 3, range(4))
    for q, size in enumerate([WIDE] + OTHERS):
        _, alone = _run([size], 3, [q])
        assert alone[0][2] == mixed[q][2]
        assert np.array_equal(alone[0][0], mixed[q][0]) and np.array_equal(alone[0][1], mixed[q][1]), size


def test_the_others_run_beside_it():
    """their chain is a fifth of the wide scene's; at least some of it is hidden
    (one after the other, the step took 1.20 times as long as the wide scene's)"""
    alone = min(_run([WIDE], 6, [0])[0] for _ in range(3))
    mixed = min(_run([WIDE] + OTHERS, 6, range(4))[0] for _ in range(3))
    assert mixed < 1.16 * alone
