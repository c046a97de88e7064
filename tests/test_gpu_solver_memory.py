"""Device memory of the pressure solver's state (runtime.cu): what a solver
reports is what it holds, and the buffers of the MIC(0) sweeps come with the
first MIC(0) solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

m = pytest.importorskip("mantaflow_gb300")
torch = pytest.importorskip("torch")

N = 224
SLACK = 48 << 20  # two dozen allocations in steps of 2 MB


def _scene(n):
    s = m.Solver(name="mem", gridSize=m.vec3(n, n, n), dim=3)
    flags, vel, p, rhs = s.create(m.FlagGrid), s.create(m.MACGrid), s.create(m.RealGrid), s.create(m.RealGrid)
    flags.initDomain(boundaryWidth=0)
    flags.fillGrid()
    m.setOpenBound(flags, 0, "Y", m.FlagOutflow | m.FlagEmpty)
    vel.setConst(m.vec3(0.1, 0.2, 0.3))
    return s, flags, vel, p, rhs


def _free(grid):
    grid.getMaxAbs()  # waits for the solver's stream
    return torch.cuda.mem_get_info()[0]


def test_reported_bytes_are_the_held_ones():
    s, flags, vel, p, rhs = _scene(16)
    for pc in (m.PcMIC, m.PcMGStatic):  # the kernels are loaded
        m.solvePressure(flags=flags, vel=vel, pressure=p, preconditioner=pc)
    s, flags, vel, p, rhs = _scene(N)
    free, held = _free(p), s.memoryBytes()
    m.computePressureRhs(rhs=rhs, vel=vel, pressure=p, flags=flags)
    cells = N ** 3
    # codes (2 bytes) and three float grids; none of MIC(0)'s
    assert free - _free(p) <= cells * 14 + SLACK
    assert abs((free - _free(p)) - (s.memoryBytes() - held)) <= SLACK
    m.solvePressureSystem(rhs=rhs, vel=vel, pressure=p, flags=flags, preconditioner=m.PcMIC, cgMaxIterFac=2.5 / N)
    # r, z, P and the stencil bits in level order: 14 bytes a cell and more
    assert free - _free(p) >= cells * 28
    assert abs((free - _free(p)) - (s.memoryBytes() - held)) <= SLACK
