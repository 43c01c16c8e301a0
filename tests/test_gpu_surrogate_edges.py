"""Descriptors, forces and training gradient of the surrogate at the edges of their work
split, against the CPU reference: boxes of one cell, of two cells per edge (the whole
chain is one neighbourhood) and of three or more, chains with odd atom counts, one
species only, fewer tiles than blocks.  Bounds as in test_gpu_surrogate.py: FP32
descriptors 1e-4 relative; BF16 network gradients within a few percent of FP64 ones."""
import os
import sys

import numpy as np
import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "oracle"))

pytestmark = pytest.mark.gpu

DESC = dict(rc=2.5, mu0=0.8, mu15=2.5, width=0.15)


@pytest.fixture(scope="module")
def gpu():
    import emdee_gb300
    from emdee_gb300.build import build
    build()
    return emdee_gb300.load()


@pytest.mark.parametrize("C,n,drop,species", [(1, 3, 0, "mixed"), (3, 5, 7, "mixed"), (1, 7, 1, "first"),
                                              (2, 9, 0, "mixed"), (5, 9, 40, "second"), (1, 13, 3, "mixed")])
def test_edges(gpu, C, n, drop, species):
    import surrogate_oracle as so
    from emdee_gb300.surrogate import BINARY, Surrogate, simple_cubic
    L = (n ** 3 / BINARY["rho"]) ** (1.0 / 3.0)
    N = n ** 3 - drop
    rng = np.random.default_rng(n)
    types = {"mixed": np.where(rng.random(N) < 0.8, 1, 2), "first": np.ones(N, int), "second": np.full(N, 2)}[species]
    R = np.stack([simple_cubic(n ** 3, L, n + c, jitter=0.2)[:N] for c in range(C)])
    m = Surrogate(gpu, C, N, L, types)
    p = rng.normal(0, 0.2, m.nparam).astype(np.float32)
    m.set_params(p)
    Rt = torch.tensor(R, device="cuda")
    G = m.descriptors(Rt).cpu().double().reshape(C, N, 32)
    t = torch.tensor(types - 1)
    for c in range(C):
        ref = so.descriptors(torch.tensor(R[c]), L, t, **DESC)
        assert torch.allclose(G[c], ref, rtol=1e-4, atol=1e-5), (G[c] - ref).abs().max()
    E, F = m.forces(Rt)
    E0, F0 = zip(*[so.forces(torch.tensor(R[c]), L, t, torch.tensor(p, dtype=torch.float64), **DESC) for c in range(C)])
    E0, F0 = torch.stack(E0), torch.stack(F0)
    assert ((F.cpu() - F0).norm() / F0.norm()).item() < 0.05
    Et = E0 + torch.tensor(rng.normal(0, 0.1 * N, C))
    Ft = F0 + torch.tensor(rng.normal(0, 1.0, F0.shape)) * F0.std()
    lE, lF, grad = m.gradient(Rt, Et.cuda(), Ft.cuda())
    # the losses follow from the model's own energies and forces
    dE, dF = E.cpu() - Et, F.cpu() - Ft
    assert abs(lE - (dE ** 2).sum().item() / (N * N * C)) < 1e-12 * lE
    assert abs(lF - (dF ** 2).sum().item() / (3 * N * C)) < 1e-12 * lF
    # the gradient against the reference's for the same residuals
    _, _, g0 = so.loss_gradient(torch.tensor(R), L, t, torch.tensor(p, dtype=torch.float64), *DESC.values(), E0 - dE,
                                F0 - dF, 1.0, 1.0)
    g = grad.cpu().double()
    assert (g @ g0 / (g.norm() * g0.norm())).item() > 0.99
    assert abs(g.norm() / g0.norm() - 1).item() < 0.05
    m.close()
