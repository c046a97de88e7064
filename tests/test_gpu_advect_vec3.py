"""First-order advection of a Vec3 grid beside that of a Real one.  A cell moves
36 bytes against 20, 1.8 times as many, and the arithmetic of the trace and the
index is shared, so a pass may take twice a Real's time.  (With the index of the
MacCormack passes, which takes more registers, it took 2.2 times as long.)"""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

m = pytest.importorskip("mantaflow_gb300")


def test_vec3_pass_beside_a_real_one():
    n = 200
    rng = np.random.default_rng(1)
    s = m.Solver(name="vec3", gridSize=m.vec3(n, n, n), dim=3)
    s.timestep = 1.0
    flags, vel = s.create(m.FlagGrid), s.create(m.MACGrid)
    flags.initDomain(boundaryWidth=0)
    flags.fillGrid()
    m.copyArrayToGridReal(0.3 * rng.standard_normal((n, n, n, 3)).astype(np.float32), vel)
    real, vec = s.create(m.RealGrid), s.create(m.VecGrid)
    m.copyArrayToGridReal(rng.random((n, n, n), dtype=np.float32), real)
    m.copyArrayToGridReal(rng.random((n, n, n, 3), dtype=np.float32), vec)

    def seconds(grid):
        best = 1e9
        for _ in range(5):
            real.getMaxAbs()  # waits for the stream
            t = time.perf_counter()
            for _ in range(200):
                m.advectSemiLagrange(flags=flags, vel=vel, grid=grid, order=1)
            real.getMaxAbs()
            best = min(best, time.perf_counter() - t)
        return best

    seconds(real)
    assert seconds(vec) < 2.0 * seconds(real)
