"""The weight of an FP64 history after a segment, E exp(-y), against extended
precision over the values that y = sigma_a f d takes.

Bound, in units of 2^-53 of the weight (of the least normal number where the
weight is below it): where exp(-y) - 1 is above -1/2, its error (1.01 units in
the last place of at most 1/2) is at most 1.01 of the weight, and the sum E + E
(exp(-y) - 1) rounds once (1).  Beyond, exp(-y) itself is off by 0.51 units in
its last place (1.02), and the product rounds once (1).  Below 0, exp(-y) - 1 is
CUDA's, one unit in its last place (2), and the sum rounds once (1)."""
import os
import subprocess

import pytest

from conftest import REPO

SRC = os.path.join(REPO, "tests", "native", "attenuate_check.cu")
BIN = os.path.join(REPO, "tests", "native", "_build", "attenuate_check")
RANGES = ["tiny", "thin", "near_half", "near_one", "to_two", "cutoff", "deep", "far", "past_census", "negative"]


def bound(name):
    return 3.0 if name in ("past_census", "negative") else 2.1


@pytest.fixture(scope="module")
def tool():
    os.makedirs(os.path.dirname(BIN), exist_ok=True)
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc if os.path.exists(nvcc) else "nvcc", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-std=c++17", "-O2", "--fmad=false", "-Xcompiler", "-ffp-contract=off", SRC, "-o", BIN], check=True)

    def ask(mode):
        out = subprocess.run([BIN, mode], capture_output=True, text=True, check=True).stdout
        return dict(line.split() for line in out.strip().split("\n"))
    return ask


@pytest.fixture(scope="module")
def host(tool):
    return tool("host")


@pytest.mark.parametrize("name", RANGES)
def test_weight_within_bound(host, name):
    assert float(host[name]) <= bound(name)


@pytest.fixture(scope="module")
def device(tool):
    return tool("device")


@pytest.mark.gpu
@pytest.mark.parametrize("name", RANGES)
def test_device_weight_within_bound(device, name):
    assert float(device[name]) <= bound(name)


@pytest.mark.gpu
def test_device_weight_is_the_hosts(device):
    assert device["differ"] == "0"
