"""Single-type Lennard-Jones with each modifier, with one thread per atom and with split
lists: the packed loop (plain, shifted, force-shifted) takes entries two at a time and
removes those beyond the cut-off by zero reciprocals, the others run one at a time.
Bounds as in test_gpu_tiles: 1e-5 of the RMS force, 1e-5 of the energy scale."""
import pytest

from test_gpu_tiles import compare, gpu, oracle  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pair", ["cut", "shifted", "sf", "smooth"])
@pytest.mark.parametrize("N,tile,threads", [(251, 2, 0), (4001, 3, 0), (4001, 8, 1)])
def test_modifiers(gpu, oracle, monkeypatch, pair, N, tile, threads):  # noqa: F811
    # an edge of 8 cells holds more atoms than a block could split (one thread per atom)
    monkeypatch.setenv("EMDEE_TILE", str(tile))
    compare(gpu, oracle, 1e-5, N=N, rho=0.8, rc=2.5, skin=0.3, pair=pair)
