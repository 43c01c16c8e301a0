"""A displacement and a Verlet step of rigid water over dt = 0, followed by an ordinary
step, against the CPU oracle.  Bounds: 1e-11 of each quantity, as for a free rotation
(test_gpu_rigid_rotation); the ordinary step adds the force errors of mixed precision
(1e-5 of the RMS force, up to ten times that for one body) in proportion to what it changes."""
import ctypes as C

import numpy as np
import pytest

from emdee_gb300.emdee import FP64, MIXED
from mdrun import load_golden, setup_water
from test_gpu_rigid_rotation import gpu, oracle  # noqa: F401

pytestmark = pytest.mark.gpu


def state(lib, md, N):
    return [lib.download(md, k, s) for k, s in [("quaternions", (N // 3, 4)), ("quatmom", (N // 3, 4)),
                                               ("angmom", (N // 3, 3)), ("coordinates", (N, 3))]]


def course(lib, precision):
    water = load_golden("nist_spce_sample.json")
    run, N = water["run"], len(water["coordinates"])
    md = setup_water(lib, water, "shifted_force(coul_damped)", precision=precision, rigid=True, coords_first=True)
    lib.EmDee_random_momenta(C.byref(md), run["kB"] * run["temp"], True, run["seed"])
    out = [state(lib, md, N)]
    lib.EmDee_displace(C.byref(md), 1.0, 0.0, 0.0)
    out.append(state(lib, md, N))
    lib.EmDee_verlet_step(C.byref(md), 0.0)
    lib.EmDee_verlet_step(C.byref(md), 0.5)
    out.append(state(lib, md, N))
    return out


@pytest.mark.parametrize("precision", [FP64, MIXED])
def test_no_turn(gpu, oracle, precision):  # noqa: F811
    ref, dev = course(oracle, None), course(gpu, precision)
    for a, b in [(dev[1], dev[0]), (dev[1], ref[1])]:
        for x, y in zip(a, b):
            assert np.abs(x - y).max() <= 1e-11 * np.abs(y).max()
    for x, y, y0 in zip(dev[2], ref[2], ref[1]):
        assert np.abs(x - y).max() <= 1e-11 * np.abs(y).max() + 1e-4 * np.abs(y - y0).max()
