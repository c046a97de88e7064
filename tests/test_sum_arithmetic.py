"""The multi-float sums of mg_reduce.cuh on the CPU, against exact arithmetic.

The functions are taken out of the header and compiled for the host.  A tree of
three-float sums (TSum) over a block's values, as the cluster solvers and the
multigrid's coarsest solver add them up, has to err no more than the normalised
pairs (ff_add) that those solvers used before, and no more than a sum in double;
rounded() of a sum of squares is the float nearest to the exact sum.
"""
import os
import random
import re
import struct
import subprocess
from fractions import Fraction

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mantaflow_gb300", "csrc")

HOST = r"""
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstring>
#define __device__
#define __forceinline__ inline
static int __float_as_int(float f) { int i; memcpy(&i, &f, 4); return i; }
static float __int_as_float(int i) { float f; memcpy(&f, &i, 4); return f; }
%s
int main() {
  int n;
  while (scanf("%%d", &n) == 1) {
    static ff a[1024], b[1024];
    static TSum t[1024];
    for (int i = 0; i < 1024; i++) {
      a[i] = ff{0.f, 0.f};
      if (i < n && scanf("%%f %%f", &a[i].h, &a[i].l) != 2) return 1;
      t[i] = TSum{a[i].h, a[i].l, 0.f};
    }
    for (int o = 512; o > 0; o >>= 1)
      for (int i = 0; i < o; i++) {
        a[i] = ff_add(a[i], a[i + o]);
        t[i].add(t[i + o]);
      }
    printf("%%a %%a %%a %%a %%a %%a\n", a[0].h, a[0].l, t[0].h, t[0].l, t[0].m, t[0].rounded());
  }
}
"""


def _f32(x):
    return struct.unpack("f", struct.pack("f", x))[0]


def _nearest(x):
    """the float nearest to a Fraction (x > 0, far from the format's ends), ties to even"""
    f = _f32(float(x))
    bits = struct.unpack("I", struct.pack("f", f))[0]
    near = [struct.unpack("f", struct.pack("I", bits + d))[0] for d in (-1, 0, 1)]
    return min(near, key=lambda v: (abs(Fraction(v) - x), struct.unpack("I", struct.pack("f", v))[0] & 1))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    text = open(os.path.join(CSRC, "mg_reduce.cuh")).read()
    parts = [text[text.index("struct ff {"):text.index("__device__ __forceinline__ ff warp_sum_ff")],
             re.search(r"struct TSum \{.*?\n\};", text, re.S).group(0)]
    d = tmp_path_factory.mktemp("sums")
    (d / "sums.cpp").write_text(HOST % "\n".join(parts))
    subprocess.run(["g++", "-O1", "-ffp-contract=off", str(d / "sums.cpp"), "-o", str(d / "sums")], check=True)
    return str(d / "sums")


@pytest.mark.parametrize("squares", [True, False])
def test_trees_of_sums(program, squares):
    rng = random.Random(5)
    cases = []
    for n in (2, 64, 125, 288, 1000):
        for _ in range(40):
            v = []
            for _ in range(n):
                x = rng.gauss(0, 1) * 2.0 ** rng.uniform(-6, 6)
                x = x * x if squares else x * rng.gauss(0, 1)
                h = _f32(x)
                v.append((h, _f32(x - h)))
            cases.append(v)
    text = "".join("%d\n%s\n" % (len(v), "\n".join("%r %r" % p for p in v)) for v in cases)
    out = subprocess.run([program], input=text, capture_output=True, text=True, check=True).stdout.split("\n")
    pair = triple = double = 0.0
    for v, line in zip(cases, out):
        ah, al, th, tl, tm, r = (float.fromhex(w) for w in line.split())
        exact = sum((Fraction(h) + Fraction(l) for h, l in v), Fraction(0))
        size = sum((abs(Fraction(h)) for h, _ in v), Fraction(0))
        d = 0.0
        for h, l in v:
            d += h + l
        pair += float((Fraction(ah) + Fraction(al) - exact) / size) ** 2
        triple += float((Fraction(th) + Fraction(tl) + Fraction(tm) - exact) / size) ** 2
        double += float((Fraction(d) - exact) / size) ** 2
        if squares:
            assert r == _nearest(exact)
    assert triple <= pair and triple <= double


def test_coarse_solver_uses_them():
    """solveCG's sums and its division by the diagonal (multigrid.cu)"""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "multigrid.cu")).read())
    dots = text[text.index("void coarse_dots("):text.index("void coarse_cg(")]
    cg = text[text.index("void coarse_cg("):text.index("void tail_restrict(")]
    assert "TSum" in dots and "a.l + b.l" not in dots
    assert len(re.findall(r"z\[k\] = ff_div_f\(r\[k\], dg\[k\]\)", cg)) == 2
