"""The exact rotation of a body (csrc/rigid.cuh on the host) returns whatever the state: NaN
and infinite angular velocities or time steps, and bodies of no extent in one or more
directions (atoms on a line, at a point), which have no finite rotation."""
import os
import subprocess

from conftest import ROOT

SRC = r'''
#include <cstdio>
#include "rigid.cuh"
using namespace emdee;
int main() {
  const double nan = NAN, inf = INFINITY;
  const double coords[3][9] = {{0, 0, 0, 1, 0.2, 0, 0, 1, 0.5}, {0, 0, 0, 1, 1, 1, 2, 2, 2}, {1, 1, 1, 1, 1, 1, 1, 1, 1}};
  const double speeds[8][3] = {{1, 2, 3}, {nan, 1, 1}, {1, nan, nan}, {inf, 1, 1}, {1, -inf, 1}, {1e200, 1e200, 1e-200},
                               {1e-200, 0, 3}, {0, 0, 0}};
  const double steps[6] = {0.01, 30.0, nan, inf, 1e300, 0.0};
  int n = 0;
  for (auto& x : coords)
    for (auto& w : speeds)
      for (double dt : steps) {
        BodyState b = {};
        double M[3] = {1.0, 2.0, 3.0}, d[9], delta[9];
        b.NP = 3;
        b.mass = 6.0;
        b.invMass = 1.0 / 6.0;
        rb_update(b, M, x, d, delta);
        for (int k = 0; k < 3; k++) b.omega[k] = w[k];
        rb_rotate_exact(b, dt, d, delta);
        BodyState c = b;
        rb_rotate_elliptic(c, dt, d, delta);
        n++;
      }
  std::printf("%d\n", n);
}
'''


def test_returns(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "emdee_gb300", "csrc"),
                    "-x", "c++", str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, check=True, timeout=60)
    assert r.stdout.split() == ["144"]
