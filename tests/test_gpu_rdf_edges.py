"""EmDee_rdf at the edges of its work split: few atoms, lists of other lengths than a
multiple of 32, halos staged as atoms and as slots only (large tiles of dense cells),
histograms in shared and in global memory.  Pair counts are whole numbers, so g(r) equals
the oracle's bit for bit."""
import ctypes as C

import numpy as np
import pytest

from emdee_gb300.emdee import EmDee, FP64, MIXED
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


def rdf(lib, N, rc, bins, precision=None):
    L = (N / 0.85) ** (1.0 / 3.0)
    md = lib.system(1, 1, rc, 0.3, N, np.arange(N) % 2 + 1, [1.0, 1.0])
    if precision is not None:
        lib.EmDee_set_precision(md, precision)
    for t in (1, 2):
        lib.EmDee_set_pair_model(md, t, t, lib.EmDee_pair_lj_cut(1.0, 1.0), 0.0)
    lib.upload(md, "box", np.array([L]))
    lib.upload(md, "coordinates", fcc_lattice(N, L, 0.07, N) + 3 * L)
    pairs = np.array([[1, 2, 1], [1, 2, 2]], dtype=np.int32)
    g = np.zeros((3, bins))
    lib.EmDee_rdf(md, bins, rc, 3, pairs[0].ctypes.data_as(C.c_void_p), pairs[1].ctypes.data_as(C.c_void_p),
                  g.ctypes.data_as(C.c_void_p))
    return g


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("N,rc,bins,tile", [(2, 2.5, 7, None), (37, 2.5, 33, None), (1000, 2.5, 5000, None),
                                            (4001, 2.2, 64, "1"), (4001, 4.5, 100, "6"), (20001, 2.5, 100, None)])
def test_rdf_edges(gpu, oracle, monkeypatch, N, rc, bins, tile, precision):
    if tile:
        monkeypatch.setenv("EMDEE_TILE", tile)
    assert np.array_equal(rdf(gpu, N, rc, bins, precision), rdf(oracle, N, rc, bins))
