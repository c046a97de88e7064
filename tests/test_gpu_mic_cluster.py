"""MIC(0) sweeps in thread-block clusters (miccluster.cu).

A sweep performs the reference's float operations in an order that its
dependencies fix, and the dot products carry 48 bits where the oracle sums in
double, so eight iterations give the oracle's iterates bit for bit (a rounding
to float differs only where a sum lies within 2^-46 of a tie).  The shapes are
the edges of the schedule: one warp, ragged lines and blocks, several clusters
along z, the widest cluster, and grids that the tile sweeps run instead.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

m = pytest.importorskip("mantaflow_gb300")
from oracle import oracle as og  # noqa: E402

SHAPES = [(3, 3, 3), (16, 16, 16), (17, 18, 19), (22, 9, 5), (23, 33, 37), (70, 65, 33), (64, 64, 64), (20, 128, 40),
          (24, 250, 20), (300, 20, 20), (400, 20, 17), (24, 270, 20)]
ITERATIONS = 8


def _scene(nx, ny, nz, liquid):
    rng = np.random.default_rng(nx * 10000 + ny * 100 + nz)
    f = np.full((nz, ny, nx), og.FLUID, np.int32)
    og.init_domain(f, 0)
    og.fill_grid(f)
    phi = None
    if liquid:
        z, y, x = np.meshgrid(*(np.arange(n, dtype=np.float32) for n in f.shape), indexing="ij")
        phi = (y - 0.6 * ny + 0.1 * ny * np.sin(0.4 * x) * np.cos(0.3 * z)).astype(np.float32)
        og.update_from_levelset(f, phi)
    else:
        og.set_open_bound(f, 0, "Y")
        f[nz // 3:nz // 2, ny // 5:ny // 2, nx // 3:nx // 2] = og.OBSTACLE
    return f, (rng.random((nz, ny, nx, 3), dtype=np.float32) - 0.5).astype(np.float32), phi


def _gpu(shape, f, v, phi, s=None, **kw):
    s = s or m.Solver(name="mc", gridSize=m.vec3(*shape), dim=3)
    s.timestep = 1.0
    flags, vel, p = s.create(m.FlagGrid), s.create(m.MACGrid), s.create(m.RealGrid)
    m.copyArrayToGridReal(f, flags)
    m.copyArrayToGridReal(v, vel)
    ph = None
    if phi is not None:
        ph = s.create(m.LevelsetGrid)
        m.copyArrayToGridReal(phi, ph)
    m.solvePressure(flags=flags, vel=vel, pressure=p, phi=ph, preconditioner=m.PcMIC, **kw)
    return p.numpy(), m.lastSolveStats()[0]


@pytest.mark.parametrize("liquid", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_iterates_equal_the_oracle(shape, liquid):
    f, v, phi = _scene(*shape, liquid)
    kw = dict(cgAccuracy=2e-7, cgMaxIterFac=(ITERATIONS + 0.5) / max(shape))
    p, it = _gpu(shape, f, v, phi, **kw)
    po = np.zeros(f.shape, np.float32)
    it_ref, _, _ = og.solve_pressure(f, v.copy(), po, phi=phi, preconditioner=1, **kw)
    assert it == it_ref
    assert np.array_equal(p, po, equal_nan=True), "max diff %g" % np.max(np.abs(p - po))


@pytest.mark.parametrize("shape", [(40, 40, 40), (20, 128, 40)])
def test_wait_that_runs_out(shape):
    """a sweep whose words never come gives up, and the next solve is right"""
    f, v, _ = _scene(*shape, False)
    s = m.Solver(name="mc", gridSize=m.vec3(*shape), dim=3)
    s.setWaitLimit(2_000_000, stallNextSolve=True)
    with pytest.raises(m.MantaError) as e:
        _gpu(shape, f, v, None, s)
    assert "exceeded its spin limit" in str(e.value)
    s.setWaitLimit(0)
    p, it = _gpu(shape, f, v, None, s)
    ref, it_ref = _gpu(shape, f, v, None)
    assert it == it_ref and np.array_equal(p, ref)
