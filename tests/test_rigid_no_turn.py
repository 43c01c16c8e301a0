"""Free rotation of a rigid body over no time at all, or over a time too short to turn it
(csrc/rigid.cuh on the host): quaternion, its momentum and the angular velocity stay finite
and as they were, for asymmetric and symmetric tops.  Bound: 1e-12, the accuracy of the
closed form that the series stands in for."""
import os
import subprocess

from conftest import ROOT

SRC = r'''
#include <cstdio>
#include <random>
#include "rigid.cuh"
using namespace emdee;
int main() {
  std::mt19937_64 rng(1);
  std::normal_distribution<double> g;
  double worst = 0.0;
  int bad = 0;
  for (int n = 0; n < 200; n++) {
    BodyState b = {};
    double M[4] = {16.0, 1.0, 1.0, 1.0}, x[12], d[12], delta[12];
    b.NP = n % 2 ? 4 : 3;
    for (double& v : x) v = g(rng);
    if (n % 2)   // three equal atoms around an axis: a symmetric top
      for (int k = 0; k < 4; k++) {
        x[3 * k] = k ? std::cos(2.0943951023931953 * k) : 0.0;
        x[3 * k + 1] = k ? std::sin(2.0943951023931953 * k) : 0.0;
        x[3 * k + 2] = k ? 0.3 : 0.0;
      }
    for (int k = 0; k < b.NP; k++) b.mass += M[k];
    b.invMass = 1.0 / b.mass;
    rb_update(b, M, x, d, delta);
    double v[3], p[12];
    for (int k = 0; k < 3; k++) {
      b.omega[k] = g(rng);
      v[k] = 2.0 * b.MoI[k] * b.omega[k];
    }
    rb_B(b.q, v, b.pi);
    for (double dt : {0.0, -0.0, 1e-320, 1e-300, -1e-200}) {
      BodyState c = b;
      rb_rotate_exact(c, dt, d, p);
      double e = 0.0;
      for (int k = 0; k < 4; k++) {
        e = fmax(e, std::fabs(c.q[k] - b.q[k]));
        e = fmax(e, std::fabs(c.pi[k] - b.pi[k]));
        if (!std::isfinite(c.q[k]) || !std::isfinite(c.pi[k])) bad++;
      }
      for (int k = 0; k < 3; k++) {
        e = fmax(e, std::fabs(c.omega[k] - b.omega[k]));
        if (!std::isfinite(c.omega[k])) bad++;
      }
      for (int k = 0; k < 3 * b.NP; k++) e = fmax(e, std::fabs(p[k] - delta[k]));
      worst = fmax(worst, e);
    }
  }
  std::printf("%d %g\n", bad, worst);
}
'''


def test_state_stays(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "emdee_gb300", "csrc"),
                    "-x", "c++", str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    bad, worst = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, check=True).stdout.split()
    assert int(bad) == 0 and float(worst) <= 1e-12, (bad, worst)
