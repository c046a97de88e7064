"""An allocation of the pressure solver's state that fails: the call reports it
and the next call on the same solver starts anew and is right.  In a batch: when
the call returns, no solve of another stream is still at work on the scenes.

The failure is made on the host: the library's objects are linked once more,
with cudaMalloc wrapped by a function that answers cudaErrorMemoryAllocation
for one call of the test's choice.  Runs in a child process, which loads that
library instead of the usual one.
"""
import glob
import os
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

SHIM = r"""
#include <stddef.h>
int __real_cudaMalloc(void** p, size_t bytes);
static long left = -1;
void fail_after(long calls) { left = calls; }
int __wrap_cudaMalloc(void** p, size_t bytes) {
  if (left == 0) {
    left = -1;
    return 2; /* cudaErrorMemoryAllocation */
  }
  if (left > 0) left--;
  return __real_cudaMalloc(p, bytes);
}
"""

CHILD = r"""
import ctypes, sys
import numpy as np
from mantaflow_gb300 import _lib
L = _lib.load(sys.argv[1])
L.fail_after.argtypes = [ctypes.c_long]
import mantaflow_gb300 as m
from oracle import oracle as og

shape = tuple(int(v) for v in sys.argv[2].split("x"))
f = np.full(shape[::-1], og.FLUID, np.int32)
og.init_domain(f, 0)
og.fill_grid(f)
og.set_open_bound(f, 0, "Y")
v = (np.random.default_rng(1).random(f.shape + (3,), dtype=np.float32) - 0.5).astype(np.float32)
if shape[2] == 1:
    v[..., 2] = 0


def solver():
    s = m.Solver(name="alloc", gridSize=m.vec3(*shape), dim=3 if shape[2] > 1 else 2)
    s.timestep = 1.0
    flags, vel, p = s.create(m.FlagGrid), s.create(m.MACGrid), s.create(m.RealGrid)
    m.copyArrayToGridReal(f, flags)
    return s, flags, vel, p


def solve(g):
    s, flags, vel, p = g
    m.copyArrayToGridReal(v, vel)
    p.setConst(0.0)
    m.solvePressure(flags=flags, vel=vel, pressure=p, preconditioner=m.PcMIC)
    return p.numpy().copy()


want = solve(solver())
failed = 0
for k in range(100):
    g = solver()
    L.fail_after(k)
    try:
        solve(g)
    except m.MantaError as e:
        assert "memory" in str(e), str(e)
    else:
        break
    finally:
        L.fail_after(-1)
    failed += 1
    assert np.array_equal(solve(g), want), "after allocation %d failed" % k
print("failed", failed)
"""


BATCH = r"""
import ctypes, sys, time
import numpy as np
from mantaflow_gb300 import _lib
L = _lib.load(sys.argv[1])
L.fail_after.argtypes = [ctypes.c_long]
from mantaflow_gb300 import batch as mb
from mantaflow_gb300._lib import MantaError

# 2D scenes of hundreds of iterations on the side streams, a 3D one beside them
sizes = [(511, 512, 1), (500, 480, 1), (300, 420, 1), (24, 24, 24)]


def batch():
    return mb.BatchedPlumes(sizes, [(0, -4e-3, 0)] * len(sizes), range(len(sizes)), cgAccuracy=1e-5)


failed = 0
for k in range(40):
    b = batch()
    L.fail_after(k)
    try:
        b.step()
    except MantaError as e:
        assert "memory" in str(e), str(e)
    else:
        break
    finally:
        L.fail_after(-1)
    failed += 1
    first = [b.download(q, mb.PRESSURE) for q in range(len(sizes))]
    time.sleep(0.2)
    for q in range(len(sizes)):
        assert np.array_equal(first[q], b.download(q, mb.PRESSURE)), "allocation %d: scene %d was still being solved" % (k, q)
    b.close()
print("failed", failed)
"""


SPLAT = r"""
import ctypes, sys
import numpy as np
from mantaflow_gb300 import _lib
L = _lib.load(sys.argv[1])
L.fail_after.argtypes = [ctypes.c_long]
import mantaflow_gb300 as m
from oracle import oracle as og

rng = np.random.default_rng(4)
s = m.Solver(name="splat", gridSize=m.vec3(21, 18, 26), dim=3)
flags, vel, velOld = s.create(m.FlagGrid), s.create(m.MACGrid), s.create(m.MACGrid)
flags.initDomain(boundaryWidth=0)
flags.fillGrid()
pos = rng.uniform(0, 18, size=(30000, 3)).astype(np.float32)
pp = s.create(m.BasicParticleSystem)
pp.setPositions(pos, np.zeros(len(pos), np.int32))
pv = rng.standard_normal(pos.shape).astype(np.float32)
pvel = pp.create(m.PdataVec3)
m.copyArrayToPdataVec3(pv, pvel)
pp._flush()
f = flags.numpy()
v0, v1 = np.zeros(f.shape + (3,), np.float32), np.zeros(f.shape + (3,), np.float32)
og.map_parts_to_mac(f, v0, v1, pos, np.zeros(len(pos), np.int32), pv)
launches = []
for fail in (True, False, False):
    if fail:
        L.fail_after(0)
    n0 = ctypes.c_longlong()
    n1 = ctypes.c_longlong()
    L.mg_launch_count(ctypes.byref(n0))
    m.mapPartsToMAC(flags=flags, vel=vel, velOld=velOld, parts=pp, partVel=pvel)
    L.mg_launch_count(ctypes.byref(n1))
    launches.append(n1.value - n0.value)
    L.fail_after(-1)
    assert np.array_equal(vel.numpy(), v0) and np.array_equal(velOld.numpy(), v1)
print("launches", *launches)
"""


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    d = tmp_path_factory.mktemp("alloc")
    (d / "shim.c").write_text(SHIM)
    objs = sorted(glob.glob(os.path.join(ROOT, "mantaflow_gb300", "_build", "*.o")))
    assert objs
    subprocess.run(["gcc", "-fPIC", "-O1", "-c", str(d / "shim.c"), "-o", str(d / "shim.o")], check=True)
    from mantaflow_gb300 import build
    subprocess.run([build.nvcc()] + build.ARCH + ["-shared", "-o", str(d / "lib.so")] + objs + [str(d / "shim.o")] +
                   ["-Xlinker", "--wrap=cudaMalloc", "-lcudart_static", "-lrt", "-lpthread", "-ldl"], check=True)
    return str(d / "lib.so")


@pytest.mark.parametrize("shape,mic,least", [("20x18x22", "cluster", 18), ("20x18x22", "flow", 13), ("24x30x1", "cluster", 8)])
def test_next_call_starts_anew(library, shape, mic, least):
    r = subprocess.run([sys.executable, "-c", CHILD, library, shape], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "MANTA_GB300_MIC": mic, "PYTHONPATH": ROOT})
    assert r.returncode == 0, r.stderr[-2000:]
    assert int(r.stdout.split()[-1]) >= least  # the state's allocations, each failed once


def test_batch_leaves_nothing_running(library):
    r = subprocess.run([sys.executable, "-c", BATCH, library], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "PYTHONPATH": ROOT})
    assert r.returncode == 0, r.stderr[-2000:]
    assert int(r.stdout.split()[-1]) >= 7  # scenes, scalars, cluster and MIC scenes, tiles, sweep list, jobs: each failed once


def test_splat_without_tables(library):
    """mapPartsToMAC in 3D whose tables cannot be had: that call sorts by cell,
    with the same result, and the next one has the tile lists"""
    r = subprocess.run([sys.executable, "-c", SPLAT, library], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "PYTHONPATH": ROOT})
    assert r.returncode == 0, r.stderr[-2000:]
    sorts, lists, again = (int(v) for v in r.stdout.split()[1:])
    assert lists == again == 6 and sorts > 20
