"""A step of free atoms returns as soon as the skin check's decision and the pair kernel's
sums have arrived in pinned memory; with kernel timing switched on it waits for the
stream instead.  Both must report the same energies, virials and rebuilds at every
step, bit for bit, across several rebuilds, with and without energies."""
import ctypes as C

import numpy as np
import pytest

from emdee_gb300.emdee import MIXED

from mdrun import fcc_lattice

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import emdee_gb300
    from emdee_gb300.build import build
    build()
    return emdee_gb300.load()


@pytest.mark.parametrize("N", [200, 4000, 60000])
def test_same_as_waiting(gpu, N):
    L = (N / 0.8) ** (1.0 / 3.0)
    out = []
    for timed in (0, 1):
        md = gpu.system(1, 1, 2.5, 0.3, N)
        gpu.EmDee_set_precision(md, MIXED)
        gpu.EmDee_set_pair_model(md, 1, 1, gpu.EmDee_shifted_force(gpu.EmDee_pair_lj_cut(1.0, 1.0)), 0.0)
        gpu.upload(md, "box", np.array([L]))
        gpu.upload(md, "coordinates", fcc_lattice(N, L, 0.05, 5))
        gpu.EmDee_random_momenta(C.byref(md), 1.5, True, 86245)
        gpu.EmDee_profile(md, timed)
        rows = []
        for k in range(60):
            md.Options.Compute = k % 4 == 3
            gpu.EmDee_boost(C.byref(md), 1.0, 0.0, 0.0025)
            gpu.EmDee_displace(C.byref(md), 1.0, 0.0, 0.005)
            gpu.EmDee_boost(C.byref(md), 1.0, 0.0, 0.0025)
            rows.append([md.Energy.Potential, md.Virial.Total, md.Kinetic.Total, md.Builds])
        out.append((np.array(rows), gpu.download(md, "forces", (N, 3))))
    assert out[0][0][-1, 3] >= out[0][0][0, 3] + 3
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
