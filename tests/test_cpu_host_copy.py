"""The transfers of fields and distributions (host_copy.cpp) on the CPU, over an
implementation of the CUDA calls they make (tests/cpp/host_copy_main.cpp)."""

import os
import subprocess

import pytest

from conftest import ROOT
from hemepure_b200.build import CSRC, CUDA


@pytest.fixture(scope="module")
def host_copy(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("cpp") / "host_copy_main")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-Wall", "-pthread", "-I" + os.path.join(CUDA, "include"),
                           os.path.join(ROOT, "tests", "cpp", "host_copy_main.cpp"), os.path.join(CSRC, "host_copy.cpp"),
                           "-o", exe])
    return exe


@pytest.mark.parametrize("scenario", ["other_device", "event_failure", "own_buffers", "shared_pieces", "scratch_given_back", "one_order",
                                      "small_copies", "no_device_memory", "fork_safe", "sets_in_turn"])
def test_host_copy(host_copy, scenario):
    r = subprocess.run([host_copy, scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
