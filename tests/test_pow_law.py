"""x^p of the opacity laws for small whole p, against extended precision.

Bound, in units in the last place: the result rounds once (1/2); the error terms
that are carried along are below 2^-50 of it and wrong by 2^-52 of themselves,
the extended product by a few 2^-64: 0.51.  Beyond the range of the products,
and for zeros, infinities and NaN, it is pow's value to the bit."""
import os
import subprocess

import pytest

from conftest import REPO

SRC = os.path.join(REPO, "tests", "native", "pow_law_check.cu")
BIN = os.path.join(REPO, "tests", "native", "_build", "pow_law_check")
POWERS = ["-3", "-2", "-1", "0", "1", "2", "3"]


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


@pytest.fixture(scope="module")
def device(tool):
    return tool("device")


@pytest.mark.parametrize("power", POWERS)
def test_host_power(host, power):
    assert float(host[power]) <= 0.51


def test_host_limits(host):
    assert host["limits"] == "0"


@pytest.mark.gpu
@pytest.mark.parametrize("power", POWERS)
def test_device_power(device, power):
    assert float(device[power]) <= 0.51


@pytest.mark.gpu
def test_device_limits(device):
    assert device["limits"] == "0"
