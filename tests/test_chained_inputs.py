"""CPU check of the chained kernels' sources (csrc/chain.cuh): a grid launched by
launch_chained starts while the grid before it still writes, so nothing that a kernel
writes may be declared read-only for the kernel's whole run (`const T* __restrict__`, __ldg)."""
import glob
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "emdee_gb300", "csrc")
CONSTANT = {"invMass", "charge", "species"}   # written by the host only
HELPERS = ["for_neighbors", "each_neighbor", "masked_entries", "stage_marked", "stage_frame_saved", "saved_slot"]


def definitions():
    """(file, name, parameters, body) of every kernel that waits for the grid before it and of
    the device functions that read its inputs"""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"__(launch_bounds|maxnreg)__\((?:[^()]|\([^()]*\))*\)", "", open(path).read())
        for m in re.finditer(r"^(__global__|__device__ __forceinline__)[^;{}]*?\b(\w+)\(([^;{}]*)\)\s*\{", text, re.M):
            body = text[m.end():text.index("\n}\n", m.end())]
            if "chain_wait();" in body if m.group(1) == "__global__" else m.group(2) in HELPERS:
                yield os.path.basename(path), m.group(2), m.group(3), body


def test_found():
    names = {n for _, n, _, _ in definitions()}
    assert names >= {"k_skin", "k_build", "k_pair_mixed", "k_pair_types", "k_sg_force", "k_body_boost"} | set(HELPERS)


@pytest.mark.parametrize("file,name,params,body", [pytest.param(*d, id=d[1]) for d in definitions()])
def test_inputs_are_plain(file, name, params, body):
    readonly = set(re.findall(r"const \w+\* __restrict__ (\w+)", params)) - CONSTANT
    assert not readonly, (file, name, readonly)
    assert "__ldg" not in body, (file, name)


def test_replica_lists_are_plain():
    """k_replicas rebuilds its lists between its own reads of them"""
    assert "__ldg" not in open(os.path.join(CSRC, "replicas.cu")).read()
