"""Free rotation of rigid bodies over one displacement, from angles where the series
needs one step to angles that take several and to those left to the closed form
(|w| dt up to ~3 rad at the largest dt), forwards and backwards, against the CPU oracle.

Bound: the oracle's closed form is accurate to a few 1e-13 (elliptic integrals and
their differences), the series to 1e-15; 1e-11 leaves a factor for 750 molecules."""
import ctypes as C

import numpy as np
import pytest

from emdee_gb300.emdee import EmDee, FP64, MIXED
from mdrun import load_golden, setup_water

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import emdee_gb300
    from emdee_gb300.build import build
    build()
    return emdee_gb300.load()


@pytest.fixture(scope="module")
def oracle(oracle_path):
    return EmDee(oracle_path)


def rotated(lib, water, dt, precision):
    run, N = water["run"], len(water["coordinates"])
    md = setup_water(lib, water, "shifted_force(coul_damped)", precision=precision, rigid=True, coords_first=True)
    lib.EmDee_random_momenta(C.byref(md), run["kB"] * run["temp"], True, run["seed"])
    lib.EmDee_displace(C.byref(md), 1.0, 0.0, dt)
    return (lib.download(md, "quaternions", (N // 3, 4)), lib.download(md, "quatmom", (N // 3, 4)),
            lib.download(md, "angmom", (N // 3, 3)), lib.download(md, "coordinates", (N, 3)))


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("dt", [0.25, -1.0, 2.0, 4.0, 7.0, 15.0, -33.0, 60.0])
def test_rotation(gpu, oracle, dt, precision):
    water = load_golden("nist_spce_sample.json")
    ref = rotated(oracle, water, dt, None)
    dev = rotated(gpu, water, dt, precision)
    for a, b in zip(dev, ref):
        assert np.abs(a - b).max() <= 1e-11 * np.abs(b).max()
