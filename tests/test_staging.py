"""The staged host copies (staging.h) against a CPU stand-in of the runtime whose
copies run only when someone waits for their stream: what a copy returns with is
in place, at the edges of chunks and windows, on an ordinary stream and on
cudaStreamPerThread, for one caller and for several."""
from __future__ import annotations

import os
import subprocess

import pytest

from conftest import ROOT

HERE = os.path.join(ROOT, "tests", "staging")


@pytest.fixture(scope="module")
def binary(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("staging") / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", HERE, "-I", os.path.join(ROOT, "3d-ray_b200", "csrc"),
                    os.path.join(HERE, "staging_check.cpp"), "-o", out], check=True)
    return out


def test_copies_are_done_when_they_return(binary):
    r = subprocess.run([binary], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("events", [0, 1, 31])
def test_without_events_copies_go_the_plain_way(binary, events):
    r = subprocess.run([binary, str(events)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
