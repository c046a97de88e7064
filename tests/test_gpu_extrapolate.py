"""extrapolateMACSimple and extrapolateLsSimple (forces.cu) against the oracle,
bit for bit, where the passes' marks could go wrong: no layers, one, more than
the marks' period of three, more than the grid has; thin and tiny grids, whose
cells are mostly sides; 2D; fluid up to the walls and none at all."""
import numpy as np
import pytest

from oracle import oracle as og

pytestmark = pytest.mark.gpu

m = pytest.importorskip("mantaflow_gb300")

SHAPES = [(3, 3, 3), (4, 3, 5), (33, 9, 8), (31, 34, 1), (3, 50, 1)]
DISTANCES = [0, 1, 2, 3, 4, 5, 8, 200]


def _grid(s, cls, a):
    g = s.create(cls)
    m.copyArrayToGridReal(a, g)
    return g


def _solver(shape):
    nx, ny, nz = shape
    return m.Solver(name="extrapolate", gridSize=m.vec3(nx, ny, nz), dim=3 if nz > 1 else 2)


@pytest.mark.parametrize("distance", DISTANCES)
@pytest.mark.parametrize("shape", SHAPES)
def test_mac(shape, distance):
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + distance)
    for fluid, into in ((0.03, False), (0.03, True), (0.5, False), (0.0, False)):
        f = rng.choice(np.array([m.FlagFluid, m.FlagObstacle, m.FlagEmpty], np.int32), size=(nz, ny, nx),
                       p=[fluid, 0.1, 0.9 - fluid]).astype(np.int32)
        v = rng.standard_normal((nz, ny, nx, 3)).astype(np.float32)
        if nz == 1:
            v[..., 2] = 0
        s = _solver(shape)
        flags, vel = _grid(s, m.FlagGrid, f), _grid(s, m.MACGrid, v)
        m.extrapolateMACSimple(flags=flags, vel=vel, distance=distance, intoObs=into)
        want = v.copy()
        og.extrapolate_mac_simple(f, want, distance, into)
        assert np.array_equal(vel.numpy(), want)


@pytest.mark.parametrize("distance", DISTANCES)
@pytest.mark.parametrize("shape", SHAPES)
def test_levelset(shape, distance):
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + distance)
    for share, inside in ((0.05, False), (0.95, True), (0.5, False), (0.0, False)):
        phi = np.where(rng.random((nz, ny, nx)) < share, -1, 1) * rng.uniform(0.1, 1, size=(nz, ny, nx))
        phi = phi.astype(np.float32)
        g = _grid(_solver(shape), m.LevelsetGrid, phi)
        m.extrapolateLsSimple(phi=g, distance=distance, inside=inside)
        want = phi.copy()
        og.extrapolate_ls_simple(want, distance, inside)
        assert np.array_equal(g.numpy(), want)
