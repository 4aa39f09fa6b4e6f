"""The FP64 functions of a transport segment (imc_math64.cuh), on the CPU
against extended precision.

Bounds, in units in the last place.  -log(k 2^-53): the conversion of the
fixed-point value rounds once (1/2); next to 1 the series' last sum rounds once
and its correction term is below 2^-8 of the result: 3/4.  exp(-y) - 1: from 1
on the remainder r, exp(-r) - 1, its product with the table value and the last
sum round once each, the first three on terms no larger than the result: 2, the
error CUDA's exp and expm1 together may have in the two results they replace.
The reciprocal's two Newton steps are exact to 2^-59 before their rounding:
1/2 + 1/32.  A 128-bit sum's addends are rounded to its unit (1/2 each, three
of them at most) or cut after 64 bits, 2^-63 of an addend: 2 of the larger of
the unit and 2^-60 of the sum.  The quotient and the uniforms are exact."""
import os
import subprocess

import pytest

from conftest import REPO

SRC = os.path.join(REPO, "tests", "native", "math64_check.cpp")
BIN = os.path.join(REPO, "tests", "native", "_build", "math64_check")


@pytest.fixture(scope="module")
def worst():
    os.makedirs(os.path.dirname(BIN), exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", SRC, "-o", BIN], check=True)
    out = subprocess.run([BIN], capture_output=True, text=True, check=True).stdout
    return dict(line.split() for line in out.strip().split("\n"))


@pytest.mark.parametrize("name,bound", [("log", 0.75), ("expm1", 2.0), ("div", 0), ("uniform", 0),
                                        ("reciprocal", 0.53125), ("sum", 2.0)])
def test_math64_within_bounds(worst, name, bound):
    assert float(worst[name]) <= bound


def test_math64_limits(worst):
    assert worst["limits"] == "1"
    assert worst["refused"] == "1"
