"""Kernel variants that other tests reach only through the tuner's choice, against the CPU
oracle: the packed Lennard-Jones loop with one thread per atom (tiles of more atoms than a
block could split), and shifted damped Coulomb in the kernel of several types; and steps
whose results are read while the grid drains.  Bounds as in test_gpu_tiles; over 20 steps of
0.004 errors of 1e-5 in the forces leave the energies within 1e-5 of their scale."""
import ctypes as C

import numpy as np
import pytest

import test_gpu_tiles
from emdee_gb300.emdee import MIXED
from mdrun import velocity_verlet
from test_gpu_tiles import compare, gpu, oracle, system  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pair", ["cut", "shifted", "sf", "smooth"])
@pytest.mark.parametrize("N,rho", [(4001, 0.8), (7001, 0.75)])
def test_one_thread_per_atom(gpu, oracle, monkeypatch, pair, N, rho):  # noqa: F811
    monkeypatch.setenv("EMDEE_TILE", "6")
    kw = dict(N=N, rho=rho, rc=3.0, skin=0.5, pair=pair)
    md = system(gpu, precision=MIXED, **kw)
    # blocks of at most 256 threads: with two threads per atom they would have 1024
    assert gpu.EmDee_tile_edge(md) == 6 and gpu.EmDee_tile_threads(md, 1) <= 256
    compare(gpu, oracle, 1e-5, **kw)


@pytest.mark.parametrize("pair", ["cut", "shifted", "sf"])
@pytest.mark.parametrize("N,ntypes,rc", [(500, 2, 2.5), (1001, 3, 2.5), (1500, 2, 4.0)])
def test_shifted_damped_coulomb(gpu, oracle, monkeypatch, pair, N, ntypes, rc):  # noqa: F811
    monkeypatch.setitem(test_gpu_tiles.COULOMB, "damped_shifted",
                        lambda lib: lib.EmDee_shifted(lib.EmDee_coul_damped(0.6)))
    compare(gpu, oracle, 3e-5, N=N, rho=0.85, rc=rc, skin=0.3, ntypes=ntypes, pair=pair, coul="damped_shifted")


@pytest.mark.parametrize("N", [300, 5000])
def test_polled_steps(gpu, oracle, N):  # noqa: F811
    out = []
    for lib, precision in ((gpu, MIXED), (oracle, None)):
        md = system(lib, N=N, rho=0.8, rc=2.5, skin=0.3, pair="sf", precision=precision)
        lib.EmDee_random_momenta(C.byref(md), 1.2, True, 86245)
        rows = []
        velocity_verlet(lib, md, 0.004, 20, 5, lambda k, m: rows.append((m.Energy.Potential, m.Virial.Total, m.Kinetic.Total))
                        if k % 5 == 0 else None)
        out.append((np.array(rows), md.Builds))
    (a, builds), (b, builds0) = out
    assert builds == builds0 and np.abs(a - b).max() <= 1e-5 * np.abs(b).max()
