"""The cluster launch that runs the coarse end of a V-cycle (multigrid.cu):
whether a level runs in it or as launches of its own, a solve's pressure must
have the same bits.  The shapes put the edges of its loops to the test: levels
with more vertices of a colour than the cluster has threads, levels of a few
vertices, coarsest levels with one and two vertices per thread, flat and long
grids, 2D, with and without the stencil dictionary."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

m = pytest.importorskip("mantaflow_gb300")


def _solve(shape, seed):
    nx, ny, nz = shape
    rng = np.random.default_rng(seed)
    s = m.Solver(name="tail", gridSize=m.vec3(nx, ny, nz), dim=3 if nz > 1 else 2)
    flags, vel, p = s.create(m.FlagGrid), s.create(m.MACGrid), s.create(m.RealGrid)
    flags.initDomain()
    flags.fillGrid()
    f = flags.numpy().copy()
    f[(rng.random(f.shape) < 0.1) & (f == m.FlagFluid)] = m.FlagObstacle
    m.copyArrayToGridReal(f, flags)
    m.copyArrayToGridReal(rng.standard_normal(f.shape + (3,)).astype(np.float32), vel)
    m.solvePressure(flags=flags, vel=vel, pressure=p, preconditioner=m.PcMGStatic, cgAccuracy=1e-4)
    return p.numpy().copy()


@pytest.mark.parametrize("dictionary", [True, False])
@pytest.mark.parametrize("shape", [(96, 90, 88), (12, 11, 10), (37, 29, 41), (9, 150, 8), (300, 7, 9), (61, 203, 1), (700, 20, 1)])
def test_levels_in_and_out_of_the_cluster(shape, dictionary, monkeypatch):
    if not dictionary:
        monkeypatch.setenv("MANTAGPU_MG_NO_DICT", "1")
    out = []
    for slots in ("0", "2000", "10000000"):
        monkeypatch.setenv("MANTAGPU_MG_TAIL_SLOTS", slots)
        out.append(_solve(shape, sum(shape)))
    assert np.isfinite(out[0]).all() and np.abs(out[0]).max() > 0
    assert np.array_equal(out[0], out[1])
    assert np.array_equal(out[0], out[2])
