"""FP64 forces where the halo of a one-cell tile holds more atoms than fit with their box
fractions in shared memory (4732), in a box of five cells per edge and of six, for one type
and for three with charges, against the CPU oracle; what does not fit at all is refused.
Bound: FP64 rounding of sums of some 1000 terms each, 1e-11 of the RMS force and energies."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
from emdee_gb300.emdee import FP64
from test_gpu_tiles import gpu, oracle, system  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,rc", [(5500, 6.5), (6900, 7.0), (9000, 6.7)])
@pytest.mark.parametrize("models", [dict(pair="sf"), dict(ntypes=3, pair="cut", coul="damped", exclude=True)])
def test_forces(gpu, oracle, N, rc, models):  # noqa: F811
    kw = dict(N=N, rho=0.85, rc=rc, skin=0.5, **models)
    ref, dev = system(oracle, **kw), system(gpu, precision=FP64, **kw)
    F, G = gpu.download(dev, "forces", (N, 3)), oracle.download(ref, "forces", (N, 3))
    assert np.sqrt(((F - G) ** 2).sum()) <= 1e-11 * np.sqrt((G ** 2).sum())
    scale = abs(ref.Energy.Dispersion) + abs(ref.Energy.Coulomb) + abs(ref.Virial.Total)
    assert abs(dev.Energy.Potential - ref.Energy.Potential) <= 1e-11 * scale
    assert abs(dev.Virial.Total - ref.Virial.Total) <= 1e-11 * scale
    assert np.array_equal(gpu.neighbor_pairs(dev), oracle.neighbor_pairs(ref))


def test_refused():
    code = "\n".join(["import sys; sys.path[:0] = [%r, %r]" % (ROOT, os.path.join(ROOT, "tests")),
                      "import emdee_gb300", "from emdee_gb300.emdee import FP64", "from test_gpu_tiles import system",
                      "system(emdee_gb300.load(), N=7500, rho=0.85, rc=7.2, skin=0.5, precision=FP64)"])
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 1 and "too many atoms around a cell" in r.stderr, r.stderr


@pytest.mark.parametrize("N,fits", [(12766, True), (12768, False)])
def test_largest_halo(N, fits):
    """The list build takes 12,766 atoms of one type in a halo (all atoms of a box of five cells
    per edge), no more: 200 KB of positions, offsets and a sentinel"""
    code = "\n".join(["import sys; sys.path[:0] = [%r, %r]" % (ROOT, os.path.join(ROOT, "tests")),
                      "import emdee_gb300", "from emdee_gb300.emdee import MIXED", "from test_gpu_tiles import system",
                      "md = system(emdee_gb300.load(), N=%d, rho=0.85, rc=9.0, skin=0.5, pair='sf', precision=MIXED)" % N,
                      "print(md.Energy.Potential)"])
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    if fits:
        assert r.returncode == 0 and np.isfinite(float(r.stdout)), r.stderr
    else:
        assert r.returncode == 1 and "too many atoms around a cell" in r.stderr, r.stderr
