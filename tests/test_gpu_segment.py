"""The FP32 segment's building blocks (imc_device.cuh): the shift register of
stream words against the stream itself, and on the GPU the reciprocals and
quotients against the IEEE division and the FP64 functions of imc_math64.cuh
against their host path.  All are exact, no mismatch is allowed, but the FP64
reciprocal: off by 1/2 + 1/32 units in the last place at most, it is the IEEE
quotient or its neighbour."""
import os
import subprocess

import pytest

from conftest import REPO

SRC = os.path.join(REPO, "tests", "native", "segment_check.cu")
BIN = os.path.join(REPO, "tests", "native", "_build", "segment_check")


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


def test_word_register_hands_out_the_stream(tool):
    assert tool("words") == {"words5": "0", "words7": "0"}


@pytest.fixture(scope="module")
def device(tool):
    return tool("device")


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["rcp_mid", "rcp_any", "div_mid", "neglog_k53", "expm1_neg", "rcp64"])
def test_device_arithmetic(device, name):
    assert device[name] == "0"
