"""The 128-bit sum of a cell's FP64 deposits before its flush, on the CPU: at
2^94 units of the tally and beyond it is refused, as one value of that size is,
since the flush's accumulator words hold no more; below, it is handed on exactly."""
import os
import subprocess

import pytest

from conftest import REPO

SRC = os.path.join(REPO, "tests", "native", "sum128_check.cpp")
BIN = os.path.join(REPO, "tests", "native", "_build", "sum128_check")


@pytest.fixture(scope="module")
def found():
    os.makedirs(os.path.dirname(BIN), exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", SRC, "-o", BIN], check=True)
    out = subprocess.run([BIN], capture_output=True, text=True, check=True).stdout
    return dict(line.split() for line in out.strip().split("\n"))


@pytest.mark.parametrize("name", ["refused", "kept"])
def test_sum_range(found, name):
    assert found[name] == "1"
