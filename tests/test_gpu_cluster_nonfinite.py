"""NaN, infinities and values beyond a float's square in the cluster solvers:
the outcome is the oracle's, a reported divergence or the same iterations, and
the next solve on the solver is right.  (Residuals that are no numbers are passed
over: where only the cells outside the fluid are left, both find 0 and stop.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

m = pytest.importorskip("mantaflow_gb300")
from oracle import oracle as og  # noqa: E402


def _oracle(f, v):
    p = np.zeros(f.shape, np.float32)
    try:
        return og.solve_pressure(f, v.copy(), p, preconditioner=1)[0], p
    except RuntimeError as e:
        return str(e), None


@pytest.mark.parametrize("value", [np.nan, np.inf, 1e25, 1e37])
@pytest.mark.parametrize("shape", [(33, 40, 1), (200, 180, 1), (20, 18, 22), (40, 60, 40)])
@pytest.mark.parametrize("everywhere", [False, True])
def test_outcome_is_the_oracles(shape, value, everywhere):
    nx, ny, nz = shape
    rng = np.random.default_rng(nx)
    f = np.full((nz, ny, nx), og.FLUID, np.int32)
    og.init_domain(f, 0)
    og.fill_grid(f)
    og.set_open_bound(f, 0, "Y")
    good = (rng.random(f.shape + (3,), dtype=np.float32) - 0.5).astype(np.float32)
    if nz == 1:
        good[..., 2] = 0
    bad = good.copy()
    if everywhere:
        bad[..., :2] *= np.float32(value)
    else:
        bad[nz // 2, ny // 2, nx // 2, 0] = value
    s = m.Solver(name="nonfinite", gridSize=m.vec3(*shape), dim=3 if nz > 1 else 2)
    s.timestep = 1.0
    flags, vel, p = s.create(m.FlagGrid), s.create(m.MACGrid), s.create(m.RealGrid)
    m.copyArrayToGridReal(f, flags)
    for v in (bad, good):
        m.copyArrayToGridReal(v, vel)
        p.setConst(0.0)
        want, po = _oracle(f, v)
        try:
            m.solvePressure(flags=flags, vel=vel, pressure=p, preconditioner=m.PcMIC)
            got = m.lastSolveStats()[0]
        except m.MantaError as e:
            got = str(e)
        assert got == want
    assert np.max(np.abs(p.numpy() - po)) <= 1e-4
