"""The sweep height that a batch keeps (best_height in batch.cu), compiled for the
host: the fastest of those that were timed."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mantaflow_gb300", "csrc")


def test_fastest_of_the_timed_heights(tmp_path):
    text = open(os.path.join(CSRC, "batch.cu")).read()
    body = re.search(r"int best_height\(const float\* ms\) \{.*?\n\}", text, re.S).group(0)
    (tmp_path / "t.cpp").write_text("#include <cstdio>\n" + body + """
int main() {
  float m[4];
  while (scanf("%f %f %f %f", m, m + 1, m + 2, m + 3) == 4) printf("%d\\n", best_height(m));
}
""")
    subprocess.run(["g++", str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    cases = {(0, 0, 0, 0): 0, (2, 0, 0, 0): 0, (3, 2, 0, 0): 1, (3, 2, 1, 0): 2, (3, 2, 4, 1): 3, (1, 2, 3, 4): 0, (0, 5, 4, 0): 2}
    out = subprocess.run([str(tmp_path / "t")], input="\n".join("%g %g %g %g" % c for c in cases), capture_output=True, text=True,
                         check=True).stdout.split()
    assert [int(v) for v in out] == list(cases.values())


def test_timings_are_of_the_sweeps_alone():
    """no run is taken that 2D solves on the side streams ran beside"""
    text = open(os.path.join(CSRC, "batch.cu")).read()
    solve = text[text.index("int engine_cg("):text.index("int engine_step(")]
    assert "cudaEventQuery(e.join[q])" in solve and "if (timing && alone && " in solve
