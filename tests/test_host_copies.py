"""Copies between host arrays and the device (csrc/fs_stage.cpp), their CUDA calls
replaced by a stand-in that can fail (tests/stage_harness.cpp)."""
import os
import subprocess

import pytest

from multi_species_b200 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("stage") / "stage_harness")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(B.nvcc()))), "include")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", cuda, "-I", os.path.join(B.ROOT, "include"),
                    os.path.join(HERE, "stage_harness.cpp"), "-o", exe, "-lpthread", "-ldl"], check=True)
    return exe


@pytest.mark.parametrize("scenario", ["failing copies", "refused", "short lives"])
def test_host_copies(harness, scenario):
    r = subprocess.run([harness, scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
