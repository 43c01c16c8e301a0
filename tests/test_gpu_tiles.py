"""Work splits of the list build and of the mixed-precision force kernels: tile edges
from one cell, one to 32 threads per atom, thread-per-atom, split and warp-per-atom
builds (cells of 2 to 20 atoms), boxes of five cells per edge, one to three types with
and without charges.  Pair sets equal the oracle's bit for bit; forces, energies and
virials agree within the mixed mode's bounds.

Bounds: FP32 pair terms carry a few 1e-7 (relative) each and positions are rounded to
2.4e-7 cell edges, which the steepest part of r^-13 multiplies by about 20: 1e-5 of the
RMS force, 3e-5 with charges (net forces are small differences of Coulomb terms); sums
of terms 1e-5, the virial on the scale of the sum of its terms' magnitudes (energy)."""
import numpy as np
import pytest

from emdee_gb300.emdee import EmDee, MIXED
from mdrun import fcc_lattice

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


MODIFIER = {"cut": lambda lib, m: m, "shifted": lambda lib, m: lib.EmDee_shifted(m),
            "sf": lambda lib, m: lib.EmDee_shifted_force(m), "smooth": lambda lib, m: lib.EmDee_square_smoothed(m, 0.5)}
COULOMB = {"none": lambda lib: lib.EmDee_coul_none(), "damped": lambda lib: lib.EmDee_coul_damped(0.8),
           "damped_sf": lambda lib: lib.EmDee_shifted_force(lib.EmDee_coul_damped(0.6)),
           "damped_smoothed": lambda lib: lib.EmDee_coul_damped_smoothed(0.9, 0.4),
           "cut": lambda lib: lib.EmDee_coul_cut()}


def system(lib, N, rho, rc, skin, ntypes=1, pair="cut", coul="none", exclude=False, precision=None):
    L = (N / rho) ** (1.0 / 3.0)
    rng = np.random.default_rng(N)
    types = np.arange(N) % ntypes + 1
    md = lib.system(1, 1, rc, skin, N, types, [1.0 + 0.5 * t for t in range(ntypes)])
    if precision is not None:
        lib.EmDee_set_precision(md, precision)
    for t in range(1, ntypes + 1):   # the third type has no pair model of its own
        m = lib.EmDee_pair_none() if t == 3 else MODIFIER[pair](lib, lib.EmDee_pair_lj_cut(0.5 + 0.5 * t, 1.0 - 0.05 * t))
        lib.EmDee_set_pair_model(md, t, t, m, 0.0 if t == 2 and ntypes == 2 else 0.9)
    if ntypes > 1:
        lib.EmDee_set_pair_model(md, 1, 2, MODIFIER[pair](lib, lib.EmDee_pair_lj_cut(0.8, 0.9)), 0.7)
    lib.EmDee_set_coul_model(md, COULOMB[coul](lib))
    if exclude:
        for i in range(1, N, 7):
            for j in (i + 1, i + 2, i + 3, i + 5, i + 6):
                lib.EmDee_ignore_pair(md, i, min(j, N))
    if coul != "none":
        lib.upload(md, "charges", rng.uniform(-1, 1, N) * (np.arange(N) % 5 != 0))
    lib.upload(md, "box", np.array([L]))
    lib.upload(md, "coordinates", fcc_lattice(N, L, 0.05, N))
    return md


def compare(gpu, oracle, tol, **kw):
    N = kw["N"]
    ref, dev = system(oracle, **kw), system(gpu, precision=MIXED, **kw)
    assert np.array_equal(gpu.neighbor_pairs(dev), oracle.neighbor_pairs(ref))
    F, G = gpu.download(dev, "forces", (N, 3)), oracle.download(ref, "forces", (N, 3))
    assert np.sqrt(((F - G) ** 2).sum()) <= tol * np.sqrt((G ** 2).sum())
    scale = abs(ref.Energy.Dispersion) + abs(ref.Energy.Coulomb) + abs(ref.Virial.Total)
    assert abs(dev.Energy.Potential - ref.Energy.Potential) <= 1e-5 * scale
    assert abs(dev.Energy.Coulomb - ref.Energy.Coulomb) <= 1e-5 * scale
    assert abs(dev.Virial.Total - ref.Virial.Total) <= 1e-5 * scale


@pytest.mark.parametrize("tile", [1, 2, 3, 5])
@pytest.mark.parametrize("N,rho,rc", [(300, 0.8, 2.5), (1099, 0.85, 2.5), (3001, 0.9, 4.4), (2000, 0.9, 5.0)])
def test_tile_edges(gpu, oracle, monkeypatch, tile, N, rho, rc):
    monkeypatch.setenv("EMDEE_TILE", str(tile))
    compare(gpu, oracle, 1e-5, N=N, rho=rho, rc=rc, skin=0.4, pair="sf")


@pytest.mark.parametrize("N", [2, 33, 500, 2049, 20000])
@pytest.mark.parametrize("pair", ["cut", "smooth"])
def test_sizes(gpu, oracle, N, pair):
    compare(gpu, oracle, 1e-5, N=N, rho=0.8, rc=2.5, skin=0.3, pair=pair)


@pytest.mark.parametrize("pair", ["cut", "shifted", "sf", "smooth"])
@pytest.mark.parametrize("coul", ["none", "damped", "damped_sf", "damped_smoothed", "cut"])
@pytest.mark.parametrize("N,ntypes,rc,exclude", [(500, 2, 2.5, False), (1001, 3, 2.5, True), (1500, 3, 4.0, True)])
def test_models(gpu, oracle, pair, coul, N, ntypes, rc, exclude):
    compare(gpu, oracle, 1e-5 if coul == "none" else 3e-5, N=N, rho=0.85, rc=rc, skin=0.3, ntypes=ntypes, pair=pair,
            coul=coul, exclude=exclude)
