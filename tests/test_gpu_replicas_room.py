"""A replica whose lists outgrow their room stops with the message, whichever call builds
them: a cold crystalline drop in a large box has up to 140 neighbors per atom where the
room follows the mean density (64).  Each case runs in a child process."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

DROP = """
import ctypes as C
import sys
sys.path[:0] = [%r, %r]
import numpy as np
import emdee_gb300
from mdrun import fcc_lattice
lib, N, L = emdee_gb300.load(), 500, 38.0
md = lib.system(1, 1, 2.5, 0.3, N)
lib.EmDee_set_pair_model(md, 1, 1, lib.EmDee_pair_lj_cut(1.0, 1.0), 0.0)
lib.upload(md, "box", np.array([L]))
lib.upload(md, "coordinates", fcc_lattice(N, 5 * 1.55, 0.0, 0) + 15.0)
lib.upload(md, "momenta", np.zeros((N, 3)))
mds = (C.POINTER(type(md)) * 1)(C.pointer(md))
b = lib.EmDee_replicas_create(1, C.cast(mds, C.c_void_p))
""" % (ROOT, os.path.join(ROOT, "tests"))


@pytest.fixture(scope="module", autouse=True)
def built():
    from emdee_gb300.build import build
    build()


@pytest.mark.parametrize("calls", ["lib.EmDee_replicas_run(b, 5, 1e-5, 5)",
                                   "lib.EmDee_replicas_run(b, 0, 1e-5, 5); lib.EmDee_replicas_run(b, 5, 1e-5, 5)",
                                   "lib.EmDee_replicas_run(b, 0, 1e-5, 5); lib.EmDee_replicas_evaluate(b)",
                                   "lib.EmDee_replicas_evaluate(b)"])
def test_outgrown_lists_are_reported(calls):
    r = subprocess.run([sys.executable, "-c", DROP + calls], capture_output=True, text=True, timeout=300)
    assert r.returncode == 1 and "a neighbor list outgrew its capacity" in r.stderr, r.stderr
