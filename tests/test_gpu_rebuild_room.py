"""Rebuilds are queued together with the force kernels on their lists; if a list or a tile
outgrows the room that the build before left it, those kernels do nothing and the build
is repeated with more.  Atoms of a dilute lattice are drawn together into one dense drop
between two force computations, so that lists, tiles and halos all grow several times:
pair sets must equal the FP64 oracle's bit for bit, forces, energy and virial agree within
the mixed mode's bounds (1e-5 of the RMS force and of the sums' scale)."""
import ctypes as C

import numpy as np
import pytest

from emdee_gb300.emdee import EmDee, MIXED

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


@pytest.mark.parametrize("compute", [True, False])
@pytest.mark.parametrize("n", [6, 10, 16])
def test_drop(gpu, oracle, n, compute):
    N, L = n ** 3, 3.0 * n
    rng = np.random.default_rng(n)
    lattice = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3).astype(float)
    jitter = rng.uniform(-0.05, 0.05, lattice.shape)
    md = []
    for lib, prec in ((oracle, None), (gpu, MIXED)):
        s = lib.system(1, 1, 2.5, 0.4, N)
        if prec is not None:
            lib.EmDee_set_precision(s, prec)
        lib.EmDee_set_pair_model(s, 1, 1, lib.EmDee_shifted_force(lib.EmDee_pair_lj_cut(1.0, 1.0)), 0.0)
        lib.upload(s, "box", np.array([L]))
        lib.upload(s, "coordinates", 3.0 * (lattice + 0.2))
        md.append(s)
    for spacing in (2.0, 1.05, 3.0, 1.05):   # dense, dense again after a dilute list in between
        X = spacing * lattice + jitter + 0.6
        for lib, s in zip((oracle, gpu), md):
            lib.upload(s, "coordinates", X)
            s.Options.Compute = True if lib is oracle else compute
            lib.EmDee_compute_forces(C.byref(s))
        ref, dev = md
        assert dev.Builds == ref.Builds
        assert np.array_equal(gpu.neighbor_pairs(dev), oracle.neighbor_pairs(ref))
        F, G = gpu.download(dev, "forces", (N, 3)), oracle.download(ref, "forces", (N, 3))
        assert np.sqrt(((F - G) ** 2).sum()) <= 1e-5 * np.sqrt((G ** 2).sum())
        scale = abs(ref.Energy.Potential) + abs(ref.Virial.Total)
        assert abs(dev.Virial.Total - ref.Virial.Total) <= 1e-5 * scale
        if compute:
            assert abs(dev.Energy.Potential - ref.Energy.Potential) <= 1e-5 * scale
