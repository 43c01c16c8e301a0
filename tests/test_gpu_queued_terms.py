"""Bonds, angles, k-space sums, the rigid-body virial and the closing half of
EmDee_verlet_step are queued behind the pair kernel and skipped with it when the
skin check, which is still on the device, finds a rebuild due
(emdee_gb300/csrc/motion.cu, api.cpp).  Mixed-precision water runs across at least
two rebuilds: after every step forces, energies and the virial must equal those of
an FP64 system at the same coordinates (which decides on the host and queues nothing
ahead) within the mixed-precision bounds of the water tests, 3e-5 on forces and 4e-5
of the largest energy term on the sums; and free atoms must follow the
boost/displace/boost loop bit for bit, since the arithmetic is the same."""
import ctypes as C

import numpy as np
import pytest

from emdee_gb300.emdee import FP64, MIXED
from mdrun import load_golden, setup_water, velocity_verlet

from test_oracle_ewald import ewald_water

pytestmark = pytest.mark.gpu

TOL_F, TOL_E = 3e-5, 4e-5


@pytest.fixture(scope="module")
def gpu():
    import emdee_gb300
    from emdee_gb300.build import build
    build()
    return emdee_gb300.load()


def make(lib, w, case, precision):
    if case == "damped":
        return setup_water(lib, w, "coul_damped_smoothed", precision=precision, flexible=True)
    return ewald_water(lib, w, 1e-4, precision=precision, flexible=case == "ewald", rigid=case == "rigid")


def terms(md):
    e = md.Energy
    return np.array([e.Dispersion, e.Coulomb, e.Bond, e.Angle, e.Potential, md.Virial.Total])


@pytest.mark.parametrize("case", ["damped", "ewald", "rigid"])
def test_terms_across_rebuilds(gpu, case):
    w = load_golden("nist_spce_sample.json")
    N, run = len(w["coordinates"]), w["run"]
    md, ref = make(gpu, w, case, MIXED), make(gpu, w, case, FP64)
    gpu.EmDee_random_momenta(C.byref(md), 4 * run["kB"] * run["temp"], True, run["seed"])
    first, steps = md.Builds, 0
    while md.Builds < first + 2 and steps < 80:
        gpu.EmDee_verlet_step(C.byref(md), 1.0)
        steps += 1
        gpu.upload(ref, "coordinates", gpu.download(md, "coordinates", (N, 3)))
        gpu.EmDee_compute_forces(C.byref(ref))
        F, Fr = gpu.download(md, "forces", (N, 3)), gpu.download(ref, "forces", (N, 3))
        assert np.sqrt(((F - Fr) ** 2).mean() / (Fr ** 2).mean()) < TOL_F
        E, Er = terms(md), terms(ref)
        assert np.abs(E - Er).max() < TOL_E * np.abs(Er).max(), (E, Er)
    print(case, "steps", steps, "builds", md.Builds - first)
    assert md.Builds == first + 2
    if case != "rigid":
        b = make(gpu, w, case, MIXED)
        gpu.EmDee_random_momenta(C.byref(b), 4 * run["kB"] * run["temp"], True, run["seed"])
        velocity_verlet(gpu, b, 1.0, steps)
        for item in ("coordinates", "momenta"):
            assert np.array_equal(gpu.download(md, item, (N, 3)), gpu.download(b, item, (N, 3)))
