"""Two droplets in boxes far larger than they are, where nearly all of up to 24 million cells
are empty: grids of tens to hundreds of thousands of tiles and cell blocks.  Against the CPU oracle
in the smallest box (the drops are out of each other's reach in all of them).  Coordinates
uploaded with and without a rebuild, then ordinary steps.  Bounds as in test_gpu_tiles."""
import ctypes as C

import numpy as np
import pytest

from emdee_gb300.emdee import FP64, MIXED
from mdrun import fcc_lattice, velocity_verlet
from test_gpu_tiles import gpu, oracle  # noqa: F401

pytestmark = pytest.mark.gpu


def droplet(lib, L, precision=None):
    N, rng = 400, np.random.default_rng(5)
    md = lib.system(1, 1, 2.5, 0.3, N)
    if precision is not None:
        lib.EmDee_set_precision(md, precision)
    lib.EmDee_set_pair_model(md, 1, 1, lib.EmDee_shifted_force(lib.EmDee_pair_lj_cut(1.0, 1.0)), 0.0)
    R = fcc_lattice(N, 8.0, 0.05, 1) - 4.0   # the first drop lies across the box's corner
    R[N // 2:] += 0.47 * L
    lib.upload(md, "box", np.array([L]))
    lib.upload(md, "coordinates", R)
    lib.upload(md, "momenta", rng.standard_normal((N, 3)))
    return md, R


def check(gpu, oracle, md, ref, N):  # noqa: F811
    assert md.Builds == ref.Builds
    assert np.array_equal(gpu.neighbor_pairs(md), oracle.neighbor_pairs(ref))
    F, G = gpu.download(md, "forces", (N, 3)), oracle.download(ref, "forces", (N, 3))
    assert np.sqrt(((F - G) ** 2).sum()) <= 1e-5 * np.sqrt((G ** 2).sum())
    scale = abs(ref.Energy.Potential) + abs(ref.Virial.Total)
    assert abs(md.Energy.Potential - ref.Energy.Potential) <= 1e-5 * scale
    assert abs(md.Virial.Total - ref.Virial.Total) <= 1e-5 * scale


@pytest.mark.parametrize("L", [60.0, 130.0, 400.0])
def test_droplets(gpu, oracle, monkeypatch, L):  # noqa: F811
    monkeypatch.setenv("EMDEE_AUTOTUNE", "0")
    (md, R), (ref, R0) = droplet(gpu, L, MIXED), droplet(oracle, 60.0)
    N = len(R)
    check(gpu, oracle, md, ref, N)
    for shift in (0.01, 1.5, -0.7):   # within the skin, then two rebuilds
        for lib, m, r in ((gpu, md, R), (oracle, ref, R0)):
            lib.upload(m, "coordinates", r + shift)
            lib.EmDee_compute_forces(C.byref(m))
        check(gpu, oracle, md, ref, N)
    for lib, m in ((gpu, md), (oracle, ref)):
        velocity_verlet(lib, m, 0.004, 12, 4)
    check(gpu, oracle, md, ref, N)
    gpu.EmDee_destroy(C.byref(md))


@pytest.mark.parametrize("L", [60.0, 130.0])
def test_fp64(gpu, oracle, L):  # noqa: F811
    """FP64 forces with many empty tiles, in blocks of every size: FP64 rounding, 1e-12"""
    (md, R), (ref, _) = droplet(gpu, L, FP64), droplet(oracle, 60.0)
    N = len(R)
    F, G = gpu.download(md, "forces", (N, 3)), oracle.download(ref, "forces", (N, 3))
    assert np.sqrt(((F - G) ** 2).sum()) <= 1e-12 * np.sqrt((G ** 2).sum())
    assert abs(md.Energy.Potential - ref.Energy.Potential) <= 1e-12 * abs(ref.Energy.Potential)
    gpu.EmDee_destroy(C.byref(md))


def test_types_and_charges(gpu, oracle):  # noqa: F811
    """Two types with damped charges, where most tiles have no atoms; bounds of test_gpu_tiles"""
    N, L, rng = 300, 80.0, np.random.default_rng(3)
    R = fcc_lattice(N, 7.5, 0.05, 2) - 3.0
    R[::2] += 0.4 * L * (np.arange(N // 2) % 2)[:, None]
    q, out = rng.uniform(-1, 1, N), []
    for lib, precision in ((gpu, MIXED), (oracle, None)):
        md = lib.system(1, 1, 2.5, 0.3, N, np.arange(N) % 2 + 1, [1.0, 2.0])
        if precision is not None:
            lib.EmDee_set_precision(md, precision)
        for t in (1, 2):
            lib.EmDee_set_pair_model(md, t, t, lib.EmDee_pair_lj_cut(0.5 * t, 1.0), 0.9)
        lib.EmDee_set_coul_model(md, lib.EmDee_shifted_force(lib.EmDee_coul_damped(0.6)))
        lib.upload(md, "charges", q)
        lib.upload(md, "box", np.array([L]))
        lib.upload(md, "coordinates", R)
        out.append((lib.download(md, "forces", (N, 3)), md.Energy.Potential, md.Energy.Coulomb, md.Virial.Total))
    (F, E, Q, W), (G, E0, Q0, W0) = out
    assert np.sqrt(((F - G) ** 2).sum()) <= 3e-5 * np.sqrt((G ** 2).sum())
    scale = abs(E0) + abs(Q0) + abs(W0)
    assert max(abs(E - E0), abs(Q - Q0), abs(W - W0)) <= 1e-5 * scale


def test_tuned(gpu, oracle):  # noqa: F811
    """The first forces time tile edges: none so small that 11 million cells get a tile each,
    which would take 41 GB (2 KB of halo layout and 1.7 KB of lists a tile); edge 3, the least
    they should try, has 405,000 tiles with 5.5 and 13 KB, 7.5 GB"""
    import torch
    free = torch.cuda.mem_get_info()[0]
    md, _ = droplet(gpu, 311.0, MIXED)
    used = free - torch.cuda.mem_get_info()[0]
    assert gpu.EmDee_tile_edge(md) >= 3 and used < 16 << 30, (gpu.EmDee_tile_edge(md), used)
    ref, _ = droplet(oracle, 60.0)
    F, G = gpu.download(md, "forces", (400, 3)), oracle.download(ref, "forces", (400, 3))
    assert np.sqrt(((F - G) ** 2).sum()) <= 1e-5 * np.sqrt((G ** 2).sum())
    gpu.EmDee_destroy(C.byref(md))
