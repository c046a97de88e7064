"""What a batch reports of its sweeps' tile height."""
import pytest

pytestmark = pytest.mark.gpu

pytest.importorskip("mantaflow_gb300")
from mantaflow_gb300 import batch as mb  # noqa: E402


def _batch(sizes):
    return mb.BatchedPlumes(sizes, [(0, -4e-3, 0)] * len(sizes), range(len(sizes)))


def test_batch_without_sweeps_over_tiles():
    """2D scenes in clusters: a height is reported after the first solve, and
    nothing has been timed"""
    b = _batch([(64, 64), (96, 80)])
    assert b.tuning()[0] == 0
    b.step()
    assert b.tuning() == (8, [0.0] * 4)


@pytest.mark.parametrize("sizes", [[(48, 48, 48)], [(40, 44, 36), (200, 180), (96, 96), (32, 32, 32)],
                                   [(40, 40, 40), (510, 500), (480, 512)]])
def test_the_fastest_timed_height_is_kept(sizes):
    """after sixteen runs that gave no timing, if it takes so many, at the
    latest: two runs a step at least"""
    b = _batch(sizes)
    for _ in range(40):
        if b.tuning()[0]:
            break
        b.step()
    rows, ms = b.tuning()
    timed = {r: t for r, t in zip((8, 16, 32, 64), ms) if t > 0}
    assert rows == (min(timed, key=timed.get) if timed else 8)
