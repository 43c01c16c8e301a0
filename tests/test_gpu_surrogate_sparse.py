"""Surrogate lists of chains with more cells than atoms (their blocks go by atoms instead of
cells), with just as many, and with fewer: clusters across the box's corner and inside it,
against the CPU reference.  Bounds as in test_gpu_surrogate_edges."""
import os
import sys

import numpy as np
import pytest
import torch

from test_gpu_surrogate_edges import DESC, ROOT, gpu  # noqa: F401

sys.path.insert(0, os.path.join(ROOT, "oracle"))
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,N,L", [(1, 2, 30.0), (2, 61, 60.0), (3, 216, 20.0), (1, 217, 20.0), (2, 215, 20.0)])
def test_clusters(gpu, C, N, L):  # noqa: F811
    import surrogate_oracle as so
    from emdee_gb300.surrogate import Surrogate
    rng = np.random.default_rng(N)
    side = int(np.ceil(N ** (1.0 / 3.0)))
    # (1.6 apart: within the lists' room, which follows the mean density)
    sites = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:N] * 1.6
    R = np.stack([sites + rng.uniform(-0.2, 0.2, (N, 3)) - 2.0 + c * 0.3 * L for c in range(C)])
    types = np.where(rng.random(N) < 0.7, 1, 2)
    m = Surrogate(gpu, C, N, L, types)
    p = rng.normal(0, 0.2, m.nparam).astype(np.float32)
    m.set_params(p)
    Rt = torch.tensor(R, device="cuda")
    G = m.descriptors(Rt).cpu().double().reshape(C, N, 32)
    t = torch.tensor(types - 1)
    for c in range(C):
        ref = so.descriptors(torch.tensor(R[c]), L, t, **DESC)
        assert torch.allclose(G[c], ref, rtol=1e-4, atol=1e-5), (G[c] - ref).abs().max()
    m.close()
