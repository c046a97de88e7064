"""2D pressure solves in one thread-block cluster (cgcluster.cu).

Per cell the float operations are the reference's, and the two dot products
of an iteration carry 48 bits where the oracle sums in double: their roundings
to float agree unless a sum lies within 2^-46 of a tie, a chance below 1e-5
over the twelve iterations run here.  So the iterates equal the oracle's bit
for bit.  The shapes are the edges of the split: one to sixteen CTAs, strips
of one row, a last strip that is short or missing, one to thirty-two cells
per thread, and a scene too large for a cluster.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

m = pytest.importorskip("mantaflow_gb300")
from oracle import oracle as og  # noqa: E402

SHAPES = [(3, 3), (7, 5), (64, 32), (64, 33), (33, 70), (96, 128), (1100, 16), (16, 1100), (181, 197), (300, 300),
          (511, 512), (640, 600)]
ITERATIONS = 12


@pytest.mark.parametrize("liquid", [False, True])
@pytest.mark.parametrize("nx,ny", SHAPES)
def test_iterates_equal_the_oracle(nx, ny, liquid):
    rng = np.random.default_rng(nx * 1000 + ny)
    f = np.full((1, ny, nx), og.FLUID, np.int32)
    og.init_domain(f, 0)
    og.fill_grid(f)
    phi = None
    if liquid:
        y = np.arange(ny, dtype=np.float32)[None, :, None] + np.float32(0.5)
        x = np.arange(nx, dtype=np.float32)[None, None, :]
        phi = np.ascontiguousarray((y - 0.55 * ny - 0.05 * ny * np.sin(x * 0.3)).astype(np.float32) + np.zeros(f.shape, np.float32))
        og.update_from_levelset(f, phi)
    else:
        og.set_open_bound(f, 0, "Y")
        f[0, ny // 5:ny // 2, nx // 3:nx // 2] = og.OBSTACLE
    v = (rng.random((1, ny, nx, 3), dtype=np.float32) - 0.5).astype(np.float32)
    v[..., 2] = 0
    # maxIter = (int)(fac * max) * 4: twelve iterations, none converged
    kw = dict(cgAccuracy=2e-7, cgMaxIterFac=(ITERATIONS / 4 + 0.5) / max(nx, ny), preconditioner=1)
    s = m.Solver(name="cc", gridSize=m.vec3(nx, ny, 1), dim=2)
    s.timestep = 1.0
    flags, vel, p = s.create(m.FlagGrid), s.create(m.MACGrid), s.create(m.RealGrid)
    m.copyArrayToGridReal(f, flags)
    m.copyArrayToGridReal(v, vel)
    ph = None
    if liquid:
        ph = s.create(m.LevelsetGrid)
        m.copyArrayToGridReal(phi, ph)
    m.solvePressure(flags=flags, vel=vel, pressure=p, phi=ph, **kw)
    it, _ = m.lastSolveStats()
    po = np.zeros(f.shape, np.float32)
    it_ref, _, _ = og.solve_pressure(f, v.copy(), po, phi=phi, **kw)
    assert it == it_ref
    assert np.array_equal(p.numpy(), po), "max diff %g" % np.max(np.abs(p.numpy() - po))
