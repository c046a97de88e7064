"""mapPartsToMAC's tile lists (particles.cu) against the oracle, bit for bit:
every face adds the same products in particle order.  The cases are the edges
of the tiles and lists: grids below, at and past a tile's edge, of either tile
size, particles on and outside the border and on tile corners, lists on either
side of the length that shared memory sorts, random and ascending order, and
2D, which keeps the sorted buckets."""
import numpy as np
import pytest

from oracle import oracle as og

pytestmark = pytest.mark.gpu

m = pytest.importorskip("mantaflow_gb300")


def _check(shape, pos, flag, pv):
    nx, ny, nz = shape
    s = m.Solver(name="splat", gridSize=m.vec3(nx, ny, nz), dim=3 if nz > 1 else 2)
    flags = s.create(m.FlagGrid)
    flags.initDomain(boundaryWidth=0)
    flags.fillGrid()
    pp = s.create(m.BasicParticleSystem)
    pp.setPositions(pos, flag)
    pvel = pp.create(m.PdataVec3)
    m.copyArrayToPdataVec3(pv, pvel)
    vel, velOld, weight = s.create(m.MACGrid), s.create(m.MACGrid), s.create(m.VecGrid)
    m.mapPartsToMAC(flags=flags, vel=vel, velOld=velOld, parts=pp, partVel=pvel, weight=weight)
    f = flags.numpy()
    v0, v1, w = (np.zeros(f.shape + (3,), np.float32) for _ in range(3))
    og.map_parts_to_mac(f, v0, v1, pos, flag, pv, weight=w)
    assert np.array_equal(weight.numpy(), w)
    assert np.array_equal(vel.numpy(), v0)
    assert np.array_equal(velOld.numpy(), v1)


@pytest.mark.parametrize("shape", [(3, 3, 3), (4, 3, 5), (5, 7, 1), (6, 4, 1), (8, 9, 10), (33, 6, 7), (34, 5, 9)])
def test_rows_and_borders(shape):
    rng = np.random.default_rng(sum(shape))
    count = 40 * shape[0] * shape[1] * shape[2]
    pos = rng.uniform(-1.5, np.array(shape) + 1.5, size=(count, 3)).astype(np.float32)
    pos[::7] = np.round(pos[::7])                      # on cell borders
    pos[::11] = np.round(pos[::11]) + np.float32(0.5)  # on cell centres
    pos[::13] = 4 * np.round(pos[::13] / 4)            # on tile corners
    if shape[2] == 1:
        pos[:, 2] = rng.uniform(0, 1, count)
    flag = np.where(rng.random(count) < 0.1, m.ParticleDelete, 0).astype(np.int32)
    _check(shape, pos, flag, rng.standard_normal((count, 3)).astype(np.float32))


@pytest.mark.parametrize("count", [1, 31, 33, 4608, 4609, 24576, 24577])
def test_one_crowded_tile(count):
    rng = np.random.default_rng(count)
    pos = (np.float32(4.6) + np.float32(2.3) * rng.random((count, 3))).astype(np.float32)  # one tile of 4^3
    _check((12, 10, 9), pos, np.zeros(count, np.int32), rng.standard_normal(pos.shape).astype(np.float32))


@pytest.mark.parametrize("order", ["ascending", "random"])
def test_large_tiles(order):
    """a million cells: the larger tiles"""
    shape = (129, 88, 89)
    rng = np.random.default_rng(3)
    pos = rng.uniform(-1, np.array(shape) + 1.0, size=(3000000, 3)).astype(np.float32)
    if order == "ascending":
        pos = pos[np.lexsort((pos[:, 0] // 1, pos[:, 1] // 1, pos[:, 2] // 1))]
    flag = np.where(rng.random(len(pos)) < 0.05, m.ParticleDelete, 0).astype(np.int32)
    _check(shape, pos, flag, rng.standard_normal(pos.shape).astype(np.float32))
