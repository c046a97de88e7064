"""The transfers' scratch (particles.cu): mapPartsToMAC's tile lists and the
sorts of the other transfers share it, so the first mapPartsToMAC takes no
memory by the particle, and calls of either kind in turn leave each other's
results alone."""
import numpy as np
import pytest

from oracle import oracle as og

pytestmark = pytest.mark.gpu

m = pytest.importorskip("mantaflow_gb300")
torch = pytest.importorskip("torch")


def _scene(n, count):
    rng = np.random.default_rng(count)
    s = m.Solver(name="scratch", gridSize=m.vec3(n, n, n), dim=3)
    flags = s.create(m.FlagGrid)
    flags.initDomain(boundaryWidth=0)
    flags.fillGrid()
    pos = rng.uniform(1, n - 1, size=(count, 3)).astype(np.float32)
    pp = s.create(m.BasicParticleSystem)
    pp.setPositions(pos, np.zeros(count, np.int32))
    pv = rng.standard_normal((count, 3)).astype(np.float32)
    pvel = pp.create(m.PdataVec3)
    m.copyArrayToPdataVec3(pv, pvel)
    vel, velOld = s.create(m.MACGrid), s.create(m.MACGrid)
    return s, dict(flags=flags, vel=vel, velOld=velOld, parts=pp, partVel=pvel), pos, pv


def test_first_transfer_takes_no_memory_by_the_particle():
    _, g, _, _ = _scene(16, 1000)
    m.mapPartsToMAC(**g)  # the kernels are loaded
    g["vel"].numpy()
    _, g, _, _ = _scene(64, 8000000)
    g["vel"].numpy()
    before = torch.cuda.mem_get_info()[0]
    m.mapPartsToMAC(**g)
    g["vel"].numpy()
    # the tiles' tables: 132 bytes for each of 16^3, in an allocation of 2 MB
    assert before - torch.cuda.mem_get_info()[0] <= 4 << 20


def test_transfers_in_turn():
    s, g, pos, pv = _scene(40, 120000)
    tgt = s.create(m.VecGrid)
    f = g["flags"].numpy()
    flag = np.zeros(len(pos), np.int32)
    v0, v1, t0 = (np.zeros(f.shape + (3,), np.float32) for _ in range(3))
    og.map_parts_to_mac(f, v0, v1, pos, flag, pv)
    og.map_parts_to_grid(f, t0, pos, flag, pv)
    for _ in range(3):
        m.mapPartsToMAC(**g)
        m.mapPartsToGridVec3(flags=g["flags"], target=tgt, parts=g["parts"], source=g["partVel"])
        assert np.array_equal(tgt.numpy(), t0)
        assert np.array_equal(g["vel"].numpy(), v0)
        assert np.array_equal(g["velOld"].numpy(), v1)
