"""The dot products of the cluster solvers carry at least a double's bits.

Three isolated fluid cells give a sum 1 + 2^-24 + 2^-50: half way between two
floats but for the last term, which a sum in 48 bits loses.  In double (the
reference's GridDotProduct, and the other solvers here) it rounds to 1 + 2^-23,
and the first iteration's values follow from that exactly.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

m = pytest.importorskip("mantaflow_gb300")


def _solve(shape, cells):
    """cells: (x, y, z), open neighbours, right-hand side -> pressure there"""
    nx, ny, nz = shape
    s = m.Solver(name="sum", gridSize=m.vec3(nx, ny, nz), dim=3 if nz > 1 else 2)
    f = np.full((nz, ny, nx), m.FlagObstacle, np.int32)
    b = np.zeros(f.shape, np.float32)
    step = [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)]
    for (x, y, z), open_, value in cells:
        f[z, y, x] = m.FlagFluid
        b[z, y, x] = value
        for dx, dy, dz in step[:open_]:
            f[z + dz, y + dy, x + dx] = m.FlagEmpty
    flags, vel, p, rhs = s.create(m.FlagGrid), s.create(m.MACGrid), s.create(m.RealGrid), s.create(m.RealGrid)
    m.copyArrayToGridReal(f, flags)
    m.copyArrayToGridReal(b, rhs)
    m.solvePressureSystem(rhs=rhs, vel=vel, pressure=p, flags=flags, cgAccuracy=1e-3)
    assert m.lastSolveStats()[0] == 1
    out = p.numpy()
    return [float(out[z, y, x]) for (x, y, z), _, _ in cells]


@pytest.mark.parametrize("y,z", [(3, 5), (17, 20)])
def test_mic_sweep(y, z):
    """one row, so one thread's share of (z, r); P is 1 and 1/2, (A s, s) the
    same sum, and with both rounded alike alpha is 1"""
    got = _solve((40, 24, 28), [((5, y, z), 1, 1.0), ((15, y, z), 4, 2.0 ** -11), ((25, y, z), 4, 2.0 ** -24)])
    assert got == [1.0, 2.0 ** -13, 2.0 ** -26]


@pytest.mark.parametrize("shape,cells", [((32, 20), ((3, 5), (9, 5), (15, 5))),      # one warp
                                         ((32, 60), ((3, 5), (9, 25), (15, 45))),    # several warps
                                         ((96, 400), ((3, 5), (9, 200), (15, 390)))])  # several CTAs
def test_2d_solve(shape, cells):
    """(r, r) = 1 + 2^-24 + 2^-50 and (A s, s) = 3 + 2^-22 + ..., no tie"""
    value = (1.0, 2.0 ** -12, 2.0 ** -25)
    got = _solve(shape + (1,), [(c + (0,), 3 if q == 0 else 4, value[q]) for q, c in enumerate(cells)])
    alpha = (np.float32(1) + np.float32(2.0 ** -23)) / (np.float32(3) + np.float32(2.0 ** -22))
    assert got == [float(alpha * np.float32(v)) for v in value]
