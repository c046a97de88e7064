"""Advection's clamps against the oracle, bit for bit (signs of zeros aside):
traces that end on the first and last sample, between cells, and far outside on
either side, in grids of a few cells and in 2D, with each mode of the MacCormack
clamp, flags that the clamp passes over and values that tie."""
import numpy as np
import pytest

from oracle import oracle as og

pytestmark = pytest.mark.gpu

m = pytest.importorskip("mantaflow_gb300")


def _grid(s, cls, a):
    g = s.create(cls)
    m.copyArrayToGridReal(a, g)
    return g


@pytest.mark.parametrize("clamp", [1, 2])
@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("shape", [(4, 4, 4), (33, 6, 7), (5, 40, 1)])
def test_traces_onto_the_ends(shape, order, clamp):
    nx, ny, nz = shape
    rng = np.random.default_rng(sum(shape) + order)
    # steps of quarters of a cell (traces then end on samples), some of them long
    v = rng.integers(-6, 7, size=(nz, ny, nx, 3)).astype(np.float32) / 4
    v[rng.random(v.shape[:3]) < 0.1] *= 1000
    if nz == 1:
        v[..., 2] = 0
    f = rng.choice(np.array([m.FlagFluid, m.FlagObstacle, m.FlagEmpty], np.int32), size=(nz, ny, nx), p=[0.8, 0.1, 0.1])
    f = f.astype(np.int32)
    real = rng.integers(-3, 4, size=(nz, ny, nx)).astype(np.float32)
    mac = rng.integers(-3, 4, size=(nz, ny, nx, 3)).astype(np.float32)
    if nz == 1:
        mac[..., 2] = 0
    s = m.Solver(name="edges", gridSize=m.vec3(nx, ny, nz), dim=3 if nz > 1 else 2)
    flags, vel = _grid(s, m.FlagGrid, f), _grid(s, m.MACGrid, v)
    for cls, kind, a in ((m.RealGrid, og.KIND_REAL, real), (m.MACGrid, og.KIND_MAC, mac)):
        g = _grid(s, cls, a)
        m.advectSemiLagrange(flags=flags, vel=vel, grid=g, order=order, clampMode=clamp)
        want = a.copy()
        og.advect_semi_lagrange(f, v, want, kind, order=order, clampMode=clamp)
        assert np.array_equal(g.numpy(), want)
