"""Replica batches at the edges of their work split, against the CPU oracle: one to a few
atoms, boxes of five cells per edge and more, sizes around a warp and a block, atoms many
boxes away from the origin, one to three types, plain and force-shifted models; forces,
energies and virials of an evaluation, and a few steps (momenta, kinetic energies, rebuild
counts) in one run, in two and after a restored checkpoint.

Bounds: FP32 pair terms of a few 1e-7 (relative): 1e-5 of the RMS force, 1e-5 of the sums'
scale; over 30 steps of 0.004 the momenta separate by at most the force error times the
time, times the fluid's growth of about ten per 100 steps: 1e-5 of their RMS."""
import ctypes as C

import numpy as np
import pytest

from emdee_gb300.emdee import EmDee, MIXED
from mdrun import fcc_lattice, velocity_verlet

pytestmark = pytest.mark.gpu

# N, rho, rc, types, model, boxes away
SPECS = [(2, 0.05, 2.5, 1, "sf", 0), (31, 0.6, 1.4, 1, "sf", 3), (257, 0.8, 2.5, 2, "sf", -2), (1025, 0.85, 2.5, 1, "cut", 0),
         (900, 0.8, 1.7, 3, "sf", 40), (4000, 0.85, 2.5, 1, "sf", 1000)]


@pytest.fixture(scope="module")
def gpu():
    import emdee_gb300
    from emdee_gb300.build import build
    build()
    return emdee_gb300.load()


@pytest.fixture(scope="module")
def oracle(oracle_path):
    return EmDee(oracle_path)


def make(lib, spec, precision=None):
    N, rho, rc, nt, model, away = spec
    L = (N / rho) ** (1.0 / 3.0)
    md = lib.system(1, 1, rc, 0.3, N, np.arange(N) % nt + 1, [1.0 + t for t in range(nt)])
    if precision is not None:
        lib.EmDee_set_precision(md, precision)
    for t in range(1, nt + 1):
        p = lib.EmDee_pair_lj_cut(1.0 + 0.2 * t, 1.0 - 0.02 * t)
        lib.EmDee_set_pair_model(md, t, t, lib.EmDee_shifted_force(p) if model == "sf" else p, 0.0)
    for t in range(1, nt + 1):
        for u in range(t + 1, nt + 1):
            p = lib.EmDee_pair_lj_cut(0.9, 0.95)
            lib.EmDee_set_pair_model(md, t, u, lib.EmDee_shifted_force(p) if model == "sf" else p, 0.0)
    lib.upload(md, "box", np.array([L]))
    lib.upload(md, "coordinates", fcc_lattice(N, L, 0.03, N) + away * L)
    rng = np.random.default_rng(N)
    lib.upload(md, "momenta", rng.standard_normal((N, 3)))
    return md


def batch(gpu, mds):
    arr = (C.POINTER(type(mds[0])) * len(mds))(*[C.pointer(m) for m in mds])
    return gpu.lib.EmDee_replicas_create(len(mds), C.cast(arr, C.c_void_p)), arr


def rms(a, b):
    return np.sqrt(((a - b) ** 2).sum()) / np.sqrt((b ** 2).sum())


def check(gpu, oracle, mds, refs, momenta):
    for spec, md, ref in zip(SPECS, mds, refs):
        N = spec[0]
        F, G = gpu.download(md, "forces", (N, 3)), oracle.download(ref, "forces", (N, 3))
        assert np.sqrt(((F - G) ** 2).sum()) <= 1e-5 * np.sqrt((G ** 2).sum()) + 1e-12, spec
        scale = abs(ref.Energy.Potential) + abs(ref.Virial.Total) + 1e-12
        assert abs(md.Energy.Potential - ref.Energy.Potential) <= 1e-5 * scale, spec
        assert abs(md.Virial.Total - ref.Virial.Total) <= 1e-5 * scale, spec
        if momenta:
            assert md.Builds == ref.Builds, spec
            assert rms(gpu.download(md, "momenta", (N, 3)), oracle.download(ref, "momenta", (N, 3))) <= 1e-5, spec
            assert abs(md.Kinetic.Total - ref.Kinetic.Total) <= 1e-5 * ref.Kinetic.Total, spec


def test_evaluate(gpu, oracle):
    mds, refs = [make(gpu, s, MIXED) for s in SPECS], [make(oracle, s) for s in SPECS]
    b, keep = batch(gpu, mds)
    gpu.lib.EmDee_replicas_evaluate(b)
    check(gpu, oracle, mds, refs, False)
    gpu.lib.EmDee_replicas_destroy(b)


@pytest.mark.parametrize("runs", [(30,), (1, 29), (7, 23)])
def test_steps(gpu, oracle, runs):
    mds, refs = [make(gpu, s, MIXED) for s in SPECS], [make(oracle, s) for s in SPECS]
    b, keep = batch(gpu, mds)
    for n in runs:
        gpu.lib.EmDee_replicas_run(b, n, 0.004, n)
    for ref in refs:
        velocity_verlet(oracle, ref, 0.004, sum(runs), sum(runs))
    check(gpu, oracle, mds, refs, True)
    gpu.lib.EmDee_replicas_destroy(b)


def test_restored_positions_rebuild(gpu):
    """After a restore the lists of the abandoned path must not serve."""
    out = []
    for detour in (False, True):
        mds = [make(gpu, s, MIXED) for s in SPECS]
        b, keep = batch(gpu, mds)
        P = [gpu.download(m, "momenta", (s[0], 3)) for s, m in zip(SPECS, mds)]
        gpu.lib.EmDee_replicas_evaluate(b)
        gpu.lib.EmDee_replicas_checkpoint(b)
        if detour:
            gpu.lib.EmDee_replicas_run(b, 25, 0.004, 25)
            gpu.lib.EmDee_replicas_restore(b, (C.c_int * len(mds))(*[1] * len(mds)))
            for m, p in zip(mds, P):
                gpu.upload(m, "momenta", p)
        gpu.lib.EmDee_replicas_run(b, 10, 0.004, 10)
        out.append([(gpu.download(m, "coordinates", (s[0], 3)), gpu.download(m, "momenta", (s[0], 3)))
                    for s, m in zip(SPECS, mds)])
        gpu.lib.EmDee_replicas_destroy(b)
    for a, c in zip(*out):
        assert np.array_equal(a[0], c[0]) and np.array_equal(a[1], c[1])
