"""A block's shared memory exists for its cluster once the block runs, which the
cluster's barrier alone guarantees: no kernel may reach into another block's
shared memory before a cluster barrier of its own. Read from the source, since a
run shows nothing while the hardware happens to start a cluster's blocks together."""
from __future__ import annotations

import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "3d-ray_b200", "csrc")


def functions_with_remote_access():
    """(file:name, body) of every function that maps another block's shared memory."""
    out = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cuh", ".cu")):
            continue
        with open(os.path.join(CSRC, f)) as fh:
            text = re.sub(r"//[^\n]*", "", fh.read())
        for body in re.split(r"\n(?=(?:RT_D|RT_NI|__global__|template|__device__)\b)", text):
            if "map_shared_rank" in body:
                out.append(pytest.param(body, id=f"{f}:{re.search(r'(\w+)\s*\(const __grid|(\w+)\(', body).group(0)}"))
    return out


def test_the_cluster_kernels_are_found():
    assert len(functions_with_remote_access()) >= 2


@pytest.mark.parametrize("body", functions_with_remote_access())
def test_a_cluster_barrier_precedes_the_first_remote_access(body):
    before = body[: body.index("map_shared_rank")]
    assert "cluster.sync()" in before or ("barrier_arrive()" in before and "barrier_wait()" in before)


@pytest.mark.parametrize("body", functions_with_remote_access())
def test_a_cluster_barrier_follows_the_last_remote_access(body):
    """A block may not leave while another still reaches into its shared memory."""
    assert "cluster.sync()" in body[body.rindex("map_shared_rank"):]
