"""FP64 quotients by the reciprocals of rcp64, which may be the neighbour of
the rounded reciprocal, on the CPU: the sum that is rounded to the quotient is
then off by less than 2^-52 units in the last place, and none of the quotients
drawn here, a third of them next to a tie, is closer to one than that."""
import os
import subprocess

import pytest

from conftest import REPO

SRC = os.path.join(REPO, "tests", "native", "div64_check.cpp")
BIN = os.path.join(REPO, "tests", "native", "_build", "div64_check")


@pytest.fixture(scope="module")
def wrong():
    os.makedirs(os.path.dirname(BIN), exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", SRC, "-o", BIN], check=True)
    out = subprocess.run([BIN], capture_output=True, text=True, check=True).stdout
    return dict(line.split() for line in out.strip().split("\n"))


@pytest.mark.parametrize("name", ["any", "near_tie"])
def test_quotients_are_the_ieee_ones(wrong, name):
    assert wrong[name] == "0"
