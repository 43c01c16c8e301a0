"""k-space sums at the edges of their work split, against the CPU oracle in FP64
mode: few and odd numbers of charges (chunks of 16 atoms, blocks of 4), charged
types of one atom, atoms without charge in a charged type, and few or many wave
vectors (rows without n3 > 0 up to several blocks of m).

Bound: both sides sum at most ~1e5 FP64 terms of the size of the self energy, so they
agree to 1e-11 of it (forces: of the self energy per length unit)."""
import numpy as np
import pytest

from emdee_gb300.emdee import EmDee, FP64

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


def ions(lib, n, acc, L, precision=None):
    rng = np.random.default_rng(n)
    types = np.concatenate([[1, 2, 3], rng.integers(1, 3, n - 3)]) if n > 3 else np.arange(1, n + 1)
    q = rng.uniform(0.2, 1.5, n) * rng.choice([-1, 1], n)
    if n > 8:
        q[5] = 0.0
    md = lib.system(1, 1, 2.2, 0.3, n, types, [1.0] * int(types.max()))
    if precision is not None:
        lib.EmDee_set_precision(md, precision)
    for t in range(1, int(types.max()) + 1):
        lib.EmDee_set_pair_model(md, t, t, lib.EmDee_pair_none(), 0.7 + 0.2 * t)
    lib.EmDee_set_coul_model(md, lib.EmDee_coul_long())
    lib.EmDee_set_kspace_model(md, lib.EmDee_kspace_ewald(acc))
    lib.upload(md, "charges", q)
    lib.upload(md, "box", [L])
    lib.upload(md, "coordinates", rng.uniform(-L, 2 * L, (n, 3)))
    return md, q


@pytest.mark.parametrize("n,acc,L", [(1, 1e-4, 7.0), (2, 1e-1, 6.3), (3, 1e-6, 6.3), (5, 1e-2, 7.0), (17, 1e-4, 7.0),
                                     (33, 1e-8, 8.0), (130, 1e-6, 15.0), (401, 1e-3, 11.0), (1000, 1e-5, 9.0)])
def test_kspace_edges(gpu, oracle, n, acc, L):
    ref, q = ions(oracle, n, acc, L)
    dev, _ = ions(gpu, n, acc, L, precision=FP64)
    scale = float((q * q).sum())
    assert abs(dev.Energy.Coulomb - ref.Energy.Coulomb) <= 1e-11 * scale
    assert abs(dev.Virial.Total - ref.Virial.Total) <= 1e-11 * scale
    F, G = gpu.download(dev, "forces", (n, 3)), oracle.download(ref, "forces", (n, 3))
    assert np.abs(F - G).max() <= 1e-11 * max(scale, np.abs(G).max())
