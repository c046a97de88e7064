"""The two forms of the interpolation index, on either side of the sizes where
one takes over from the other: the same values, the oracle's, at positions
inside, on and beyond the grid's borders."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

m = pytest.importorskip("mantaflow_gb300")
from oracle import oracle as og  # noqa: E402


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("shape", [(64, 64, 63), (64, 64, 64), (65, 64, 64), (511, 512, 1), (513, 512, 1)])
@pytest.mark.parametrize("kind", ["real", "mac", "vec3"])
def test_first_pass(shape, kind, order):
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + ny)
    f = np.full((nz, ny, nx), og.FLUID, np.int32)
    og.init_domain(f, 0)
    og.fill_grid(f)
    v = (2.0 * rng.standard_normal(f.shape + (3,))).astype(np.float32)
    v[:, :3] *= 8  # traces far beyond the border
    if nz == 1:
        v[..., 2] = 0
    s = m.Solver(name="index", gridSize=m.vec3(*shape), dim=3 if nz > 1 else 2)
    s.timestep = 1.0
    flags, vel = s.create(m.FlagGrid), s.create(m.MACGrid)
    m.copyArrayToGridReal(f, flags)
    m.copyArrayToGridReal(v, vel)
    if kind == "mac":
        grid, want, k = vel, v.copy(), og.KIND_MAC
    elif kind == "real":
        want, k = rng.random(f.shape, dtype=np.float32), og.KIND_REAL
        grid = s.create(m.RealGrid)
        m.copyArrayToGridReal(want, grid)
    else:
        want, k = rng.random(f.shape + (3,), dtype=np.float32), og.KIND_VEC3
        grid = s.create(m.VecGrid)
        m.copyArrayToGridReal(want, grid)
    m.advectSemiLagrange(flags=flags, vel=vel, grid=grid, order=order, clampMode=2)
    og.advect_semi_lagrange(f, want if kind == "mac" else v.copy(), want, k, order=order, clampMode=2)
    assert np.array_equal(grid.numpy(), want)


@pytest.mark.parametrize("count", [65535, 65536])
def test_grid_to_particles(count):
    n = 20
    rng = np.random.default_rng(count)
    s = m.Solver(name="index", gridSize=m.vec3(n, n, n), dim=3)
    flags, vel, old = s.create(m.FlagGrid), s.create(m.MACGrid), s.create(m.MACGrid)
    flags.initDomain(boundaryWidth=0)
    flags.fillGrid()
    v, o = (rng.standard_normal((n, n, n, 3)).astype(np.float32) for _ in range(2))
    m.copyArrayToGridReal(v, vel)
    m.copyArrayToGridReal(o, old)
    pos = rng.uniform(-1.0, n + 1.0, size=(count, 3)).astype(np.float32)
    pos[::5] = np.round(pos[::5])
    flag = np.zeros(count, np.int32)
    pp = s.create(m.BasicParticleSystem)
    pp.setPositions(pos, flag)
    pv = rng.standard_normal((count, 3)).astype(np.float32)
    pvel = pp.create(m.PdataVec3)
    m.copyArrayToPdataVec3(pv, pvel)
    f = flags.numpy()
    m.mapMACToParts(flags=flags, vel=vel, parts=pp, partVel=pvel)
    want = pv.copy()
    og.map_mac_to_parts(f, v, pos, flag, want)
    assert np.array_equal(pvel.numpy(), want)
    m.flipVelocityUpdate(flags=flags, vel=vel, velOld=old, parts=pp, partVel=pvel, flipRatio=0.95)
    og.flip_velocity_update(f, v, o, pos, flag, want, 0.95)
    assert np.array_equal(pvel.numpy(), want)
