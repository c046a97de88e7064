"""A copy into the MIC(0) cluster sweeps' shared memory that does not come
(miccluster.cu): the wait for it is bounded, and giving up is reported.  The
grids are one bundle of lines, whose warps wait for nothing else."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

m = pytest.importorskip("mantaflow_gb300")


def _solve(s, shape):
    rng = np.random.default_rng(2)
    flags, vel, p = s.create(m.FlagGrid), s.create(m.MACGrid), s.create(m.RealGrid)
    flags.initDomain(boundaryWidth=0)
    flags.fillGrid()
    m.setOpenBound(flags, 0, "Y", m.FlagOutflow | m.FlagEmpty)
    m.copyArrayToGridReal(rng.standard_normal(shape[::-1] + (3,)).astype(np.float32), vel)
    m.solvePressure(flags=flags, vel=vel, pressure=p, preconditioner=m.PcMIC)
    return p.numpy().copy()


@pytest.mark.parametrize("shape", [(20, 8, 8), (60, 7, 6)])
def test_copies_that_do_not_come_are_reported(shape):
    s = m.Solver(name="copies", gridSize=m.vec3(*shape), dim=3)
    s.setWaitLimit(1_000_000, stallNextSolve=2)
    with pytest.raises(m.MantaError) as e:
        _solve(s, shape)
    assert "exceeded its spin limit" in str(e.value)
    s.setWaitLimit(0)
    want = _solve(m.Solver(name="other", gridSize=m.vec3(*shape), dim=3), shape)
    assert np.array_equal(_solve(s, shape), want) and np.abs(want).max() > 0
