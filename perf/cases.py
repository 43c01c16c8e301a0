"""Timed cases of the library: what a user's program has it do, over the range of sizes.

Kinds
  lj         a Lennard-Jones fluid (rho 0.8442, rc 2.5, skin 0.3, T* 1.5, dt 0.005) advanced by
             velocity-Verlet steps: `stepper` "vv" is the boost / displace / boost loop of the
             reference's tests, "verlet" is EmDee_verlet_step; `model` "cut" is the plain
             truncated potential, "sf" the force-shifted one; energies every `nprop`-th step
  rerun      stored frames of such a fluid from host memory, in FP64 mode: coordinates up,
             energies, forces down, radial distribution function
  mixture    the 80:20 binary Lennard-Jones mixture (rho 1.2, T* 0.8), force-shifted
  water      rigid three-site water (exact rotation), damped force-shifted Coulomb, dt 1 fs
  ewald      the same molecules with coul_long and the Ewald sum
  flexible   the same molecules with harmonic bonds and angles instead, dt 0.5 fs, verlet_step
  replicas   many independent boxes of ragged sizes in one batch run
  proposal   the learned potential: a hybrid Monte Carlo proposal of a few steps, all chains
  training   the learned potential: one energy + force gradient of a batch of configurations

Every input is generated from the seed.  Results of the default mode, whose pair arithmetic is
FP32, are handed on as trajectory files hold them, in FP32 (the forces of that mode are FP32
values); those of the FP64 mode in FP64.  The force of the plain truncated potential jumps at the
cut-off, so a pair that lies there to the last bit changes two forces by 0.04: of "cut" runs the
frame holds coordinates and momenta, of "sf" runs the forces too.
"""
import ctypes as C
import math

import numpy as np
import torch

import emdee_gb300
from emdee_gb300.emdee import FP64, MIXED
from emdee_gb300.surrogate import Surrogate

# reduced Lennard-Jones units
LJ = dict(rho=0.8442, rc=2.5, skin=0.3, kT=1.5, dt=0.005)
MIX = dict(rho=1.2, rc=2.5, skin=0.3, kT=0.8, dt=0.004, eps=[[1.0, 1.5], [1.5, 0.5]], sig=[[1.0, 0.8], [0.8, 0.88]])
# water: Da, Angstrom, fs, e; SPC/E geometry and charges, SPC/Fw force constants
MVV2E, KB, KCOUL = 2390.057364, 8.3144621455e-07, 0.13893545755135628
WATER = dict(mass=[15.9994, 1.008], eps=0.1553 / MVV2E, sig=3.166, q=[-0.8476, 0.4238], roh=1.0, angle=109.47,
             rc=10.0, skin=1.0, damp=0.2, accuracy=1e-6, spacing=3.104, kT=KB * 300.0,
             kb=1059.162 / MVV2E, r0=1.012, ka=75.90 / MVV2E, theta0=math.radians(113.24))
NET = dict(rc=2.5, mu0=0.8, mu15=2.5, width=0.15, dt=0.002)


def listed():
    return [
        # a small sample as in the golden tests, energies once per report: launches and latency
        dict(name="lj_sf_800", kind="lj", N=800, model="sf", stepper="vv", steps=20, nprop=20),
        # the step that also gives the shadow Hamiltonian, energies at every step
        dict(name="lj_verlet_16001", kind="lj", N=16001, model="sf", stepper="verlet", steps=10, nprop=1),
        # an ordinary production run of a ragged size, energies once per report
        dict(name="lj_sf_100003", kind="lj", N=100003, model="sf", stepper="vv", steps=10, nprop=10),
        # the benchmark's box: energies and virial at every step
        dict(name="lj_cut_1048576", kind="lj", N=1048576, model="cut", stepper="vv", steps=10, nprop=1),
        # analysis of stored frames in the reference's own precision
        dict(name="lj_rerun_fp64_32003", kind="rerun", N=32003, bins=100),
        # two atom types: the general force kernel and list build
        dict(name="mixture_50021", kind="mixture", N=50021, steps=10, nprop=10),
        # the rigid-water box
        dict(name="water_rigid_4096", kind="water", nmol=4096, steps=5, nprop=5),
        # electrostatics with the Ewald sum, energies at every step
        dict(name="water_ewald_1000", kind="ewald", nmol=1000, steps=3, nprop=1),
        # bonds, angles and exclusions
        dict(name="water_flexible_512", kind="flexible", nmol=512, steps=10, nprop=1),
        # the replica benchmark: 256 boxes of 256 to 8192 atoms
        dict(name="replicas_256", kind="replicas", n=256, nmin=256, nmax=8192, steps=20),
        # hybrid Monte Carlo on the learned potential
        dict(name="proposal_8x8000", kind="proposal", chains=8, N=8000, steps=5),
        # its training step
        dict(name="training_8x8000", kind="training", chains=8, N=8000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lj", "lj", "lj", "lj", "rerun", "mixture", "water", "ewald", "flexible", "replicas", "proposal",
                       "training"])
    if kind == "lj":
        model = rng.choice(["cut", "sf"])
        stepper = rng.choice(["vv", "vv", "verlet"])
        steps = rng.randint(5, 10)
        return dict(kind=kind, N=_log(rng, 800, 1000000), model=model, stepper=stepper, steps=steps,
                    nprop=rng.choice([1, steps]))
    if kind == "rerun":
        return dict(kind=kind, N=_log(rng, 1000, 100000), bins=rng.randint(50, 200))
    if kind == "mixture":
        return dict(kind=kind, N=_log(rng, 1000, 200000), steps=rng.randint(5, 10), nprop=rng.choice([1, 5]))
    if kind == "water":
        return dict(kind=kind, nmol=_log(rng, 700, 6000), steps=rng.randint(2, 5), nprop=rng.choice([1, 2]))
    if kind == "ewald":
        return dict(kind=kind, nmol=_log(rng, 600, 1000), steps=rng.randint(1, 3), nprop=1)
    if kind == "flexible":
        return dict(kind=kind, nmol=_log(rng, 500, 1000), steps=rng.randint(3, 10), nprop=1)
    if kind == "replicas":
        return dict(kind=kind, n=rng.randint(16, 256), nmin=256, nmax=_log(rng, 1000, 8192), steps=rng.randint(5, 20))
    return dict(kind=kind, chains=rng.randint(1, 8), N=rng.randint(10, 20) ** 3,
                **(dict(steps=rng.randint(1, 5)) if kind == "proposal" else {}))


# ---- inputs -----------------------------------------------------------------------


def _sites(N):
    """The cubic lattice (simple, body- or face-centred) with the fewest sites >= N, in units of the box edge."""
    best = None
    for base in ([[0, 0, 0]], [[0, 0, 0], [.5, .5, .5]], [[0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]]):
        n = 1
        while len(base) * n ** 3 < N:
            n += 1
        if best is None or len(base) * n ** 3 < best[0]:
            best = (len(base) * n ** 3, n, base)
    _, n, base = best
    g = np.stack(np.meshgrid(np.arange(n), np.arange(n), np.arange(n), indexing="ij"), -1).reshape(-1, 3)
    return ((g[:, None, :] + np.array(base)[None, :, :]).reshape(-1, 3) + 0.25) / n


def _fluid(N, rho, kT, rng, jitter=0.05):
    """Coordinates (lattice sites with random vacancies, jittered), box edge, momenta (unit masses, no drift)."""
    L = (N / rho) ** (1.0 / 3.0)
    s = _sites(N)
    if len(s) > N:
        s = s[np.sort(rng.permutation(len(s))[:N])]
    R = s * L + rng.uniform(-jitter, jitter, size=(N, 3))
    P = rng.standard_normal((N, 3)) * math.sqrt(kT)
    return R, L, P - P.mean(0)


def _rotations(n, rng):
    u1, u2, u3 = rng.random(n), rng.random(n), rng.random(n)
    q = np.stack([np.sqrt(1 - u1) * np.sin(2 * np.pi * u2), np.sqrt(1 - u1) * np.cos(2 * np.pi * u2),
                  np.sqrt(u1) * np.sin(2 * np.pi * u3), np.sqrt(u1) * np.cos(2 * np.pi * u3)], -1)
    w, x, y, z = q.T
    return np.stack([np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)], -1),
                     np.stack([2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)], -1),
                     np.stack([2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1)], -2)


def _water(nmol, rng, rigid):
    """Molecules on a simple-cubic lattice (random vacancies), random orientations; rigid: momenta of rigid motion."""
    n = 1
    while n ** 3 < nmol:
        n += 1
    L = n * WATER["spacing"]
    g = np.stack(np.meshgrid(np.arange(n), np.arange(n), np.arange(n), indexing="ij"), -1).reshape(-1, 3)
    centre = (g[np.sort(rng.permutation(n ** 3)[:nmol])] + 0.5) * WATER["spacing"]
    half, roh = math.radians(WATER["angle"]) / 2, WATER["roh"]
    site = np.array([[0, 0, 0], [roh * math.sin(half), roh * math.cos(half), 0],
                     [-roh * math.sin(half), roh * math.cos(half), 0]])
    m = np.array([WATER["mass"][0], WATER["mass"][1], WATER["mass"][1]])
    site = site - (m[:, None] * site).sum(0) / m.sum()
    rot = _rotations(nmol, rng)
    delta = np.einsum("mij,sj->msi", rot, site)
    R = (centre[:, None, :] + delta).reshape(-1, 3)
    if rigid:
        inertia = np.array([(m * (site[:, 1] ** 2)).sum(), (m * (site[:, 0] ** 2)).sum(),
                            (m * (site ** 2).sum(1)).sum()])
        v = rng.standard_normal((nmol, 3)) * math.sqrt(WATER["kT"] / m.sum())
        w = np.einsum("mij,mj->mi", rot, rng.standard_normal((nmol, 3)) * np.sqrt(WATER["kT"] / inertia))
        P = (m[None, :, None] * (v[:, None, :] + np.cross(w[:, None, :], delta))).reshape(-1, 3)
    else:
        P = rng.standard_normal((3 * nmol, 3)) * np.sqrt(WATER["kT"] * np.tile(m, nmol))[:, None]
    return R, L, P, np.tile(m, nmol)


def _replica_sizes(case):
    """Atoms, density and temperature of every box: the benchmark's ranges."""
    rng = np.random.default_rng(86245)
    return [(int(rng.integers(case["nmin"], case["nmax"] + 1)), float(rng.uniform(0.70, 0.90)),
             float(rng.uniform(0.8, 2.0))) for _ in range(case["n"])]


def _chains(case, seed):
    """Configurations, species and parameters of the learned potential."""
    rng = np.random.default_rng([seed, 7])
    N, n = case["N"], round(case["N"] ** (1.0 / 3.0))
    L = (N / MIX["rho"]) ** (1.0 / 3.0)
    g = np.stack(np.meshgrid(np.arange(n), np.arange(n), np.arange(n), indexing="ij"), -1).reshape(-1, 3)
    R = ((g + 0.5) * (L / n))[None] + rng.uniform(-0.12, 0.12, size=(case["chains"], N, 3))
    types = np.where(rng.permutation(N) < int(0.8 * N), 1, 2).astype(np.int32)
    p = []
    for _ in range(2):   # W1[32][64], b1, W2[64][64], b2, w3, b3
        a, b = math.sqrt(6 / 96), math.sqrt(6 / 128)
        p += [rng.uniform(-a, a, 2048), rng.uniform(-.1, .1, 64), rng.uniform(-b, b, 4096), rng.uniform(-.1, .1, 64),
              rng.uniform(-0.1, 0.1, 64), [-6.0]]
    P = rng.standard_normal(R.shape) * math.sqrt(MIX["kT"])
    E = -6.0 * N + rng.standard_normal(case["chains"]) * 0.1 * N
    F = rng.standard_normal(R.shape) * 20.0
    return R, L, types, np.concatenate(p).astype(np.float32), P, E, F


# ---- states -----------------------------------------------------------------------


class _View:
    """A device array of the library as torch sees it, without a copy."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(ptr, False), version=3)


class _State:
    lib = None
    systems = ()
    batch = None
    model = None

    def __del__(self):
        if self.batch:
            self.lib.EmDee_replicas_destroy(self.batch)
        for md in self.systems:
            self.lib.EmDee_destroy(C.byref(md))
        if self.model is not None:
            self.model.close()


def _start(s, md, R, L, P):
    lib = s.lib
    s.systems = [md]
    s.md = md
    lib.upload(md, "box", np.array([L]))
    lib.upload(md, "coordinates", R)
    lib.upload(md, "momenta", P)
    s.items = [n for n in ("coordinates", "momenta", "forces") if n in s.frame]
    shape = (len(R), 3)
    s.stream = torch.cuda.ExternalStream(lib.EmDee_cuda_stream(md))
    s.out = {n: torch.empty(shape, dtype=torch.float32, device="cuda") for n in s.items}
    s.view = {n: torch.as_tensor(_View(lib.EmDee_device_pointer(md, n.encode()), shape), device="cuda")
              for n in s.items}
    torch.cuda.synchronize()
    return s


def prepare(case, seed):
    lib = emdee_gb300.load()
    s = _State()
    s.lib, s.case = lib, case
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("lj", "rerun"):
        N = case["N"]
        R, L, P = _fluid(N, LJ["rho"], LJ["kT"], rng)
        md = lib.system(1, 1, LJ["rc"], LJ["skin"], N)
        lib.EmDee_set_precision(md, FP64 if kind == "rerun" else MIXED)
        pair = lib.EmDee_pair_lj_cut(1.0, 1.0)
        if kind == "rerun" or case["model"] == "sf":
            pair = lib.EmDee_shifted_force(pair)
        lib.EmDee_set_pair_model(md, 1, 1, pair, 0.0)
        if kind == "rerun":
            s.systems, s.md = [md], md
            lib.upload(md, "box", np.array([L]))
            frames = [R, R + rng.uniform(-0.1, 0.1, size=(N, 3))]
            s.frames = [torch.from_numpy(f).pin_memory() for f in frames]
            s.forces = torch.empty((N, 3), dtype=torch.float64).pin_memory()
            s.g = np.zeros(case["bins"])
            s.one = (C.c_int * 1)(1)
            s.next = 0
            lib.upload(md, "coordinates", frames[1])
            return s
        s.dt = LJ["dt"]
        s.frame = ("coordinates", "momenta") + (("forces",) if case["model"] == "sf" else ())
        return _start(s, md, R, L, P)
    if kind == "mixture":
        N = case["N"]
        R, L, P = _fluid(N, MIX["rho"], MIX["kT"], rng)
        types = np.where(rng.permutation(N) < int(0.8 * N), 1, 2)
        md = lib.system(1, 1, MIX["rc"], MIX["skin"], N, types, [1.0, 1.0])
        lib.EmDee_set_precision(md, MIXED)
        for a, b in ((1, 1), (2, 2), (1, 2)):
            lib.EmDee_set_pair_model(md, a, b, lib.EmDee_shifted_force(
                lib.EmDee_pair_lj_cut(MIX["eps"][a - 1][b - 1], MIX["sig"][a - 1][b - 1])), 0.0)
        s.dt = MIX["dt"]
        s.frame = ("coordinates", "momenta", "forces")
        return _start(s, md, R, L, P)
    if kind in ("water", "ewald", "flexible"):
        nmol, rigid = case["nmol"], kind != "flexible"
        R, L, P, _ = _water(nmol, rng, rigid)
        bodies = np.repeat(np.arange(1, nmol + 1), 3) if rigid else None
        md = lib.system(1, 1, WATER["rc"], WATER["skin"], 3 * nmol, np.tile([1, 2, 2], nmol), WATER["mass"], bodies)
        lib.EmDee_set_precision(md, MIXED)
        lib.EmDee_set_pair_model(md, 1, 1, lib.EmDee_shifted_force(lib.EmDee_pair_lj_cut(WATER["eps"], WATER["sig"])),
                                 KCOUL)
        lib.EmDee_set_pair_model(md, 2, 2, lib.EmDee_pair_none(), KCOUL)
        if kind == "ewald":
            lib.EmDee_set_coul_model(md, lib.EmDee_coul_long())
            lib.EmDee_set_kspace_model(md, lib.EmDee_kspace_ewald(WATER["accuracy"]))
        else:
            lib.EmDee_set_coul_model(md, lib.EmDee_shifted_force(lib.EmDee_coul_damped(WATER["damp"])))
        if kind == "flexible":
            bond = lib.EmDee_bond_harmonic(WATER["kb"], WATER["r0"])
            angle = lib.EmDee_angle_harmonic(WATER["ka"], WATER["theta0"])
            for k in range(1, 3 * nmol, 3):
                lib.EmDee_add_bond(md, k, k + 1, bond)
                lib.EmDee_add_bond(md, k, k + 2, bond)
                lib.EmDee_add_angle(md, k + 1, k, k + 2, angle)
        lib.upload(md, "charges", np.tile([WATER["q"][0], WATER["q"][1], WATER["q"][1]], nmol))
        s.dt = 1.0 if rigid else 0.5
        # the momenta of rigid molecules live in the bodies
        s.frame = ("coordinates", "forces") if rigid else ("coordinates", "momenta", "forces")
        return _start(s, md, R, L, P)
    if kind == "replicas":
        s.systems = []
        for k, (N, rho, kT) in enumerate(_replica_sizes(case)):
            R, L, P = _fluid(N, rho, kT, np.random.default_rng([seed, k]))
            md = lib.system(1, 1, LJ["rc"], LJ["skin"], N)
            s.systems.append(md)
            lib.EmDee_set_precision(md, MIXED)
            lib.EmDee_set_pair_model(md, 1, 1, lib.EmDee_pair_lj_cut(1.0, 1.0), 0.0)
            lib.upload(md, "box", np.array([L]))
            lib.upload(md, "coordinates", R)
            lib.upload(md, "momenta", P)
        n = len(s.systems)
        s.arr = (C.POINTER(type(s.systems[0])) * n)(*[C.pointer(m) for m in s.systems])
        s.batch = lib.EmDee_replicas_create(n, C.cast(s.arr, C.c_void_p))
        s.sizes = [k[0] for k in _replica_sizes(case)]
        s.view = {i: [torch.as_tensor(_View(lib.EmDee_device_pointer(md, i.encode()), (N, 3)), device="cuda")
                      for md, N in zip(s.systems, s.sizes)] for i in ("coordinates", "momenta")}
        lib.EmDee_replicas_run(s.batch, 0, LJ["dt"], case["steps"])   # a program's first call: picks the block size
        torch.cuda.synchronize()
        return s
    R, L, types, params, P, E, F = _chains(case, seed)
    s.model = Surrogate(lib, case["chains"], case["N"], L, types)
    s.model.set_params(params)
    s.R, s.P, s.E, s.F = [torch.from_numpy(x).cuda() for x in (R, P, E, F)]
    torch.cuda.synchronize()
    return s


# ---- passes -----------------------------------------------------------------------


def _thermo(md):
    return [md.Energy.Potential, md.Virial.Total, md.Kinetic.Total]


def run(s):
    case, lib, kind = s.case, s.lib, s.case["kind"]
    if kind == "rerun":
        md, frame = s.md, s.frames[s.next]
        s.next ^= 1
        lib.EmDee_upload(C.byref(md), b"coordinates", C.c_void_p(frame.data_ptr()))
        lib.EmDee_compute_forces(C.byref(md))
        lib.EmDee_download(md, b"forces", C.c_void_p(s.forces.data_ptr()))
        lib.EmDee_rdf(md, case["bins"], LJ["rc"], 1, C.cast(s.one, C.c_void_p), C.cast(s.one, C.c_void_p),
                      s.g.ctypes.data_as(C.c_void_p))
        return dict(forces=s.forces, thermo=np.array([md.Energy.Potential, md.Virial.Total]), rdf=s.g)
    if kind == "replicas":
        lib.EmDee_replicas_run(s.batch, case["steps"], LJ["dt"], case["steps"])
        return dict({i: torch.cat(v).float() for i, v in s.view.items()},
                    thermo=np.array([_thermo(md) for md in s.systems], np.float32))
    if kind == "proposal":
        R, P = s.R.clone(), s.P.clone()
        _, F = s.model.forces(R, rebuild=True)
        E = s.model.trajectory(R, P, F, case["steps"], NET["dt"])
        return dict(R=R.float(), P=P.float(), F=F.float(), E=E.float())
    if kind == "training":
        lossE, lossF, grad = s.model.gradient(s.R, s.E, s.F)
        return dict(loss=np.array([lossE, lossF], np.float32), grad=grad)
    md, dt = s.md, s.dt
    ref, opts = C.byref(md), md.Options
    half, nprop = 0.5 * dt, case["nprop"]
    for k in range(1, case["steps"] + 1):
        opts.Compute = k % nprop == 0 or k == case["steps"]
        if kind == "flexible" or case.get("stepper") == "verlet":
            lib.EmDee_verlet_step(ref, dt)
        else:
            lib.EmDee_boost(ref, 1.0, 0.0, half)
            lib.EmDee_displace(ref, 1.0, 0.0, dt)
            lib.EmDee_boost(ref, 1.0, 0.0, half)
    for n in s.items:   # momenta: also applies kicks that are still due
        lib.EmDee_device_pointer(md, n.encode())
    with torch.cuda.stream(s.stream):
        for n in s.items:
            s.out[n].copy_(s.view[n])
    return dict(s.out, thermo=np.array(_thermo(md), np.float32))


# ---- work -------------------------------------------------------------------------


def _ewald_vectors(L):
    a, kmax = _ewald_alpha()
    n = math.ceil(kmax * L / (2 * math.pi))
    g = np.stack(np.meshgrid(*[np.arange(-n, n + 1)] * 3, indexing="ij"), -1).reshape(-1, 3)
    g = g[(g ** 2).sum(1) <= n * n]
    return a, g[((g[:, 0] > 0) | ((g[:, 0] == 0) & ((g[:, 1] > 0) | ((g[:, 1] == 0) & (g[:, 2] > 0)))))]


def _ewald_alpha():
    y = -math.log(WATER["accuracy"])
    x = y
    for _ in range(60):
        x = x * (y + 1.0 - math.log(x)) / (x + 1.0)
    s = math.sqrt(x)
    return s / WATER["rc"], 2.0 * s * s / WATER["rc"]


def work(case):
    """Bytes: the state read once and the frame and new state written once.  Operations: about 30 for a Lennard-Jones
    pair within the cut-off, 60 with Coulomb, each pair once; 16 per atom and wave vector; 12.4 k multiply-adds per
    atom and pass of the network, forward and back, 80 per neighbour for its descriptors and again for their
    adjoint."""
    kind, steps = case["kind"], case.get("steps", 1)
    sphere = lambda rc: 4.0 / 3.0 * math.pi * rc ** 3  # noqa: E731
    if kind == "lj":
        return dict(bytes=132.0 * case["N"], flops=30.0 * steps * case["N"] * sphere(2.5) * LJ["rho"] / 2)
    if kind == "rerun":
        return dict(bytes=48.0 * case["N"], flops=38.0 * case["N"] * sphere(2.5) * LJ["rho"] / 2)
    if kind == "mixture":
        return dict(bytes=132.0 * case["N"], flops=30.0 * steps * case["N"] * sphere(2.5) * MIX["rho"] / 2)
    if kind in ("water", "ewald", "flexible"):
        n = 1
        while n ** 3 < case["nmol"]:
            n += 1
        N, L = 3 * case["nmol"], n * WATER["spacing"]
        flops = 60.0 * N * sphere(WATER["rc"]) * N / L ** 3 / 2
        if kind == "ewald":
            flops += 16.0 * N * len(_ewald_vectors(L)[1])
        return dict(bytes=132.0 * N, flops=steps * flops)
    if kind == "replicas":
        N = case["n"] * (case["nmin"] + case["nmax"]) / 2
        return dict(bytes=120.0 * N, flops=30.0 * steps * N * sphere(2.5) * 0.8 / 2)
    N, pairs = case["chains"] * case["N"], sphere(2.5) * MIX["rho"]
    one = 2 * 12400.0 + 160.0 * pairs
    if kind == "proposal":
        return dict(bytes=(48 + 36) * N, flops=N * one * (1 + steps))
    return dict(bytes=(48 + 24) * N, flops=N * (one + 6 * 6200.0 + 80.0 * pairs))


# ---- the same in 64 bits, in plain torch -----------------------------------------------


def _pairs(R, L, rmax):
    """Half list (i, j) of all pairs within rmax (minimum image), by cells of edge >= rmax."""
    N, n = len(R), int(L / rmax)
    dev = R.device
    if n < 4:
        out = []
        for a in range(0, N, 1024):
            d = R[a:a + 1024, None, :] - R[None]
            d = d - L * torch.round(d / L)
            i, j = torch.nonzero((d * d).sum(-1) < rmax * rmax, as_tuple=True)
            out.append(torch.stack([i + a, j])[:, i + a < j])
        return torch.cat(out, 1)
    c = torch.floor((R / L - torch.floor(R / L)) * n).long().clamp(0, n - 1)
    cell = c[:, 0] + n * (c[:, 1] + n * c[:, 2])
    order = torch.argsort(cell)
    count = torch.bincount(cell, minlength=n ** 3)
    start = torch.cumsum(count, 0) - count
    out = []
    for o in range(14):
        dx, dy, dz = (o + 13) % 3 - 1, (o + 13) // 3 % 3 - 1, (o + 13) // 9 - 1
        nc = (c[:, 0] + dx) % n + n * ((c[:, 1] + dy) % n + n * ((c[:, 2] + dz) % n))
        m = count[nc]
        i = torch.repeat_interleave(torch.arange(N, device=dev), m)
        j = order[start[nc][i] + torch.arange(len(i), device=dev) - torch.repeat_interleave(torch.cumsum(m, 0) - m, m)]
        d = R[i] - R[j]
        d = d - L * torch.round(d / L)
        keep = (d * d).sum(-1) < rmax * rmax
        if o == 0:
            keep &= i < j
        out.append(torch.stack([i[keep], j[keep]]))
    return torch.cat(out, 1)


class _Lists:
    """Pairs within rc of moving atoms: a half list of radius rc + margin, kept while nothing has moved margin / 2."""

    def __init__(self, L, rc, margin, drop=None):
        self.L, self.rc, self.margin, self.R0, self.drop = L, rc, margin, None, drop

    def __call__(self, R):
        if self.R0 is None or (R - self.R0).norm(dim=1).max() > 0.49 * self.margin:
            self.R0 = R.clone()
            self.ij = _pairs(R, self.L, self.rc + self.margin)
            if self.drop is not None:   # pairs of the same molecule
                self.ij = self.ij[:, self.drop[self.ij[0]] != self.drop[self.ij[1]]]
        i, j = self.ij
        d = R[i] - R[j]
        d = d - self.L * torch.round(d / self.L)
        r2 = (d * d).sum(-1)
        k = r2 < self.rc * self.rc
        return i[k], j[k], d[k], r2[k]


def _sum_forces(n, i, j, d, s):
    f = s[:, None] * d
    return torch.zeros((n, 3), dtype=torch.float64, device=d.device).index_add_(0, i, f).index_add_(0, j, -f)


def _lj(r2, eps, sig, rc, shifted):
    """Energy and virial (-r dE/dr) of Lennard-Jones pairs, force-shifted or plain."""
    s6 = (sig * sig / r2) ** 3
    E, W = 4 * eps * (s6 * s6 - s6), 24 * eps * (2 * s6 * s6 - s6)
    if shifted:
        c6 = (sig / rc) ** 6
        Ec, Wc, r = 4 * eps * (c6 * c6 - c6), 24 * eps * (2 * c6 * c6 - c6), torch.sqrt(r2)
        E, W = E - (Ec + Wc) + Wc / rc * r, W - Wc / rc * r
    return E, W


def _erfc(x):
    """Abramowitz and Stegun 7.1.26, which defines the damped models."""
    t = 1.0 / (1.0 + 0.3275911 * x)
    return t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (-1.453152027 + t * 1.061405429)))) \
        * torch.exp(-x * x)


def _damped(r, alpha):
    E = _erfc(alpha * r) / r
    return E, E + 2 * alpha / math.sqrt(math.pi) * torch.exp(-(alpha * r) ** 2)


def _lj_force(L, shifted, eps=None, sig=None, types=None, rc=2.5):
    lists = _Lists(L, rc, 0.35)

    def force(R):
        i, j, d, r2 = lists(R)
        e = 1.0 if eps is None else eps[types[i], types[j]]
        g = 1.0 if sig is None else sig[types[i], types[j]]
        E, W = _lj(r2, e, g, rc, shifted)
        return _sum_forces(len(R), i, j, d, W / r2), float(E.sum()), float(W.sum())
    return force


def _water_force(case, L, dev):
    nmol, w = case["nmol"], WATER
    q = torch.tensor([w["q"][0], w["q"][1], w["q"][1]] * nmol, dtype=torch.float64, device=dev)
    mol = torch.arange(nmol, device=dev).repeat_interleave(3)
    oxygen = torch.arange(3 * nmol, device=dev) % 3 == 0
    lists = _Lists(L, w["rc"], 0.5, mol)
    ewald = case["kind"] == "ewald"
    if ewald:
        alpha, g = _ewald_vectors(L)
        k = torch.tensor(g * (2 * math.pi / L), dtype=torch.float64, device=dev)
        k2 = (k * k).sum(1)
        pre = 4 * math.pi / L ** 3 * torch.exp(-k2 / (4 * alpha * alpha)) / k2

    def force(R):
        i, j, d, r2 = lists(R)
        r = torch.sqrt(r2)
        qq = KCOUL * q[i] * q[j]
        if ewald:
            E, W = _damped(r, alpha)
        else:
            E, W = _damped(r, w["damp"])
            Ec, Wc = [float(x) for x in _damped(torch.tensor(w["rc"], dtype=torch.float64), w["damp"])]
            E, W = E - (Ec + Wc) + Wc / w["rc"] * r, W - Wc / w["rc"] * r
        Ecoul, Wcoul, W = float((qq * E).sum()), float((qq * W).sum()), qq * W
        o = oxygen[i] & oxygen[j]
        Elj, Wlj = _lj(r2[o], w["eps"], w["sig"], w["rc"], True)
        W[o] += Wlj
        F = _sum_forces(len(R), i, j, d, W / r2)
        Elj, Wlj = float(Elj.sum()), float(Wlj.sum())
        if ewald:
            for a in range(0, len(k), 512):
                ph = R @ k[a:a + 512].T
                cs, sn = torch.cos(ph) * q[:, None], torch.sin(ph) * q[:, None]
                C0, S0 = cs.sum(0), sn.sum(0)
                Ecoul += KCOUL * float((pre[a:a + 512] * (C0 * C0 + S0 * S0)).sum())
                F += 2 * KCOUL * ((sn * C0 - cs * S0) * pre[a:a + 512]) @ k[a:a + 512]
            Ecoul -= KCOUL * alpha / math.sqrt(math.pi) * float((q * q).sum())
            for a, b in ((0, 1), (0, 2), (1, 2)):   # the pairs inside the molecules, from the k-space sum
                r = (R0[a::3] - R0[b::3]).norm(dim=1)
                Ecoul -= KCOUL * float((q[a::3] * q[b::3] * (1 - _erfc(alpha * r)) / r).sum())
            Wcoul = Ecoul
        return F, Elj + Ecoul, Wlj + Wcoul
    R0 = None

    def first(R):
        nonlocal R0
        R0 = R.clone() if R0 is None else R0
        return force(R)
    return first


def _bonded(R, L):
    """Forces, energy and virial of the harmonic bonds and angles."""
    w = WATER
    F = torch.zeros_like(R)
    E = W = 0.0
    O, H = R[0::3], (R[1::3], R[2::3])
    a = []
    for h in range(2):
        d = H[h] - O
        d = d - L * torch.round(d / L)
        r = d.norm(dim=1)
        f = (-w["kb"] * (r - w["r0"]) / r)[:, None] * d
        F[1 + h::3] += f
        F[0::3] -= f
        E += float((0.5 * w["kb"] * (r - w["r0"]) ** 2).sum())
        W += float((f * d).sum())
        a.append(d)
    u, v = a
    uu, vv, uv = (u * u).sum(1), (v * v).sum(1), (u * v).sum(1)
    th = torch.acos(uv / torch.sqrt(uu * vv))
    fac = (-w["ka"] * (th - w["theta0"]) / torch.sqrt(uu * vv - uv * uv))[:, None]
    fu, fv = ((uv / uu)[:, None] * u - v) * fac, ((uv / vv)[:, None] * v - u) * fac
    F[1::3] += fu
    F[2::3] += fv
    F[0::3] -= fu + fv
    E += float((0.5 * w["ka"] * (th - w["theta0"]) ** 2).sum())
    return F, E, W + float((fu * u + fv * v).sum())


def _steps(force, R, P, m, dt, steps):
    """Velocity Verlet of free atoms."""
    F, E, W = force(R)
    for _ in range(steps):
        P = P + 0.5 * dt * F
        R = R + dt * P / m
        F, E, W = force(R)
        P = P + 0.5 * dt * F
    return R, P, F, [E, W, 0.5 * float((P * P / m).sum())]


def _rigid_steps(force, R, P, m, dt, steps):
    """The same for rigid three-atom molecules: the free rotation by Runge-Kutta in 40 parts per step."""
    mm = m.reshape(-1, 3, 1)
    M = mm.sum(1)
    R, P = R.reshape(-1, 3, 3), P.reshape(-1, 3, 3)
    c = (mm * R).sum(1) / M
    X = R - c[:, None]
    p = P.sum(1)
    J = torch.cross(X, P, dim=2).sum(1)

    def inertia(X):
        return ((mm * (X * X).sum(2, keepdim=True)).sum(1)[..., None] * torch.eye(3, dtype=X.dtype, device=X.device)
                - torch.einsum("maz,mai,maj->mij", mm, X, X))

    def rate(X, J):
        w = torch.linalg.solve(inertia(X), J)
        return torch.cross(w[:, None].expand_as(X), X, dim=2)

    def kick(F, p, J):
        f = F.reshape(-1, 3, 3)
        return p + 0.5 * dt * f.sum(1), J + 0.5 * dt * torch.cross(X, f, dim=2).sum(1)

    F, E, W = force((c[:, None] + X).reshape(-1, 3))
    for _ in range(steps):
        p, J = kick(F, p, J)
        c = c + dt * p / M
        h = dt / 40
        for _ in range(40):
            k1 = rate(X, J)
            k2 = rate(X + 0.5 * h * k1, J)
            k3 = rate(X + 0.5 * h * k2, J)
            k4 = rate(X + h * k3, J)
            X = X + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
        F, E, W = force((c[:, None] + X).reshape(-1, 3))
        p, J = kick(F, p, J)
    W -= float((F.reshape(-1, 3, 3) * X).sum())
    K = 0.5 * float((p * p / M).sum()) + 0.5 * float((J * torch.linalg.solve(inertia(X), J)).sum())
    return (c[:, None] + X).reshape(-1, 3), F, [E, W, K]


def _net_energy(R, L, species, params):
    """Energy of one configuration of the learned potential (differentiable in R and params)."""
    i, j = _pairs(R.detach(), L, NET["rc"])
    i, j = torch.cat([i, j]), torch.cat([j, i])
    d = R[i] - R[j]
    d = d - L * torch.round(d / L)
    r = torch.sqrt((d * d).sum(1))
    mu = NET["mu0"] + torch.arange(16, dtype=R.dtype, device=R.device) * (NET["mu15"] - NET["mu0"]) / 15.0
    h = torch.exp(-((r[:, None] - mu) ** 2) / (2 * NET["width"] ** 2)) * (0.5 * (torch.cos(math.pi * r / NET["rc"])
                                                                          + 1))[:, None]
    G = torch.zeros((2 * len(R), 16), dtype=R.dtype, device=R.device).index_add(0, 2 * i + species[j], h).reshape(-1, 32)
    E = 0.0
    for s in range(2):
        p = params[s * (len(params) // 2):(s + 1) * (len(params) // 2)]
        x = torch.nn.functional.silu(G[species == s] @ p[:2048].reshape(32, 64) + p[2048:2112])
        x = torch.nn.functional.silu(x @ p[2112:6208].reshape(64, 64) + p[6208:6272])
        E = E + (x @ p[6272:6336] + p[6336]).sum()
    return E


def exact(case, seed):
    kind, dev = case["kind"], "cuda"
    rng = np.random.default_rng(seed)
    up = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(dev)  # noqa: E731
    one = torch.ones((1, 1), dtype=torch.float64, device=dev)
    if kind == "lj":
        R, L, P = _fluid(case["N"], LJ["rho"], LJ["kT"], rng)
        R, P, F, t = _steps(_lj_force(L, case["model"] == "sf"), up(R), up(P), one, LJ["dt"], case["steps"])
        return dict(coordinates=R, momenta=P, forces=F if case["model"] == "sf" else None, thermo=np.array(t))
    if kind == "rerun":
        R, L, _ = _fluid(case["N"], LJ["rho"], LJ["kT"], rng)
        R = up(R)
        F, E, W = _lj_force(L, True)(R)
        r = torch.sqrt(_Lists(L, LJ["rc"], 0.1)(R)[3])
        bins, N = case["bins"], case["N"]
        n = torch.bincount((r / LJ["rc"] * bins).long().clamp(max=bins - 1), minlength=bins).cpu().numpy()
        b = np.arange(1, bins + 1)
        g = 2.0 * n / (4.0 / 3.0 * math.pi * (LJ["rc"] / L / bins) ** 3) / (3 * b * (b - 1) + 1) / (float(N) * N)
        return dict(forces=F, thermo=np.array([E, W]), rdf=g)
    if kind == "mixture":
        N = case["N"]
        R, L, P = _fluid(N, MIX["rho"], MIX["kT"], rng)
        types = up(np.where(rng.permutation(N) < int(0.8 * N), 0, 1))
        f = _lj_force(L, True, up(np.array(MIX["eps"])), up(np.array(MIX["sig"])), types)
        R, P, F, t = _steps(f, up(R), up(P), one, MIX["dt"], case["steps"])
        return dict(coordinates=R, momenta=P, forces=F, thermo=np.array(t))
    if kind in ("water", "ewald", "flexible"):
        R, L, P, m = _water(case["nmol"], rng, kind != "flexible")
        f, m = _water_force(case, L, dev), up(m)
        if kind == "flexible":
            def both(R):
                return tuple(x + y for x, y in zip(f(R), _bonded(R, L)))
            R, P, F, t = _steps(both, up(R), up(P), m[:, None], 0.5, case["steps"])
            return dict(coordinates=R, momenta=P, forces=F, thermo=np.array(t))
        R, F, t = _rigid_steps(f, up(R), up(P), m, 1.0, case["steps"])
        return dict(coordinates=R, forces=F, thermo=np.array(t))
    if kind == "replicas":
        got = []
        for k, (N, rho, kT) in enumerate(_replica_sizes(case)):
            R, L, P = _fluid(N, rho, kT, np.random.default_rng([seed, k]))
            got.append(_steps(_lj_force(L, False), up(R), up(P), one, LJ["dt"], case["steps"]))
        return dict(coordinates=torch.cat([x[0] for x in got]), momenta=torch.cat([x[1] for x in got]),
                    thermo=np.array([x[3] for x in got]))
    R, L, types, params, P, E, F = _chains(case, seed)
    species, params = up(types.astype(np.int64) - 1), up(params.astype(np.float64))
    R, P, E, F = up(R), up(P), up(E), up(F)
    Cn, N = R.shape[:2]
    if kind == "proposal":
        out = []
        for c in range(Cn):
            def force(x):
                x = x.detach().requires_grad_(True)
                e = _net_energy(x, L, species, params)
                return -torch.autograd.grad(e, x)[0], float(e), 0.0
            out.append(_steps(force, R[c], P[c], one, NET["dt"], case["steps"]))
        return dict(R=torch.stack([o[0] for o in out]), P=torch.stack([o[1] for o in out]),
                    F=torch.stack([o[2] for o in out]), E=np.array([o[3][0] for o in out]))
    params.requires_grad_(True)
    lossE = lossF = 0.0
    grad = torch.zeros_like(params)
    for c in range(Cn):
        x = R[c].detach().requires_grad_(True)
        e = _net_energy(x, L, species, params)
        g, = torch.autograd.grad(e, x, create_graph=True)
        lE, lF = (e - E[c]) ** 2 / (N * N * Cn), ((g + F[c]) ** 2).sum() / (3 * N * Cn)
        grad += torch.autograd.grad(lE + lF, params)[0]
        lossE, lossF = lossE + float(lE.detach()), lossF + float(lF.detach())
    return dict(loss=np.array([lossE, lossF]), grad=grad)
