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
