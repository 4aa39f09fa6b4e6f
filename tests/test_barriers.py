"""Block barriers stand where every thread of the block meets them: no
__syncthreads() under a condition on the thread, whose two branches would have
to hold the same number of barriers without anything that ties them together
(CUDA C++ defines a barrier in conditional code only for a condition that is the
same for the whole block; one barrier too many in a branch hangs the GPU)."""
import glob
import os
import re

import pytest

from conftest import PKG

FILES = sorted(glob.glob(os.path.join(PKG, "csrc", "*.cu")) + glob.glob(os.path.join(PKG, "csrc", "*.cuh")))
THREAD = re.compile(r"\b(threadIdx|lane|warp)\b")


def conditional_barriers(text):
    """Lines of the barriers inside an `if` on the thread or its `else`."""
    text = re.sub(r"//[^\n]*", "", text)
    blocks, closed, head, found = [], False, "", []
    for m in re.finditer(r"[{};]|__syncthreads\(\)|[^{};_]+|_", text):
        s = m.group()
        if s == "{":
            h = head.strip()
            under = bool(re.match(r"(else\s+)?if\b", h) and THREAD.search(h)) or (h.startswith("else") and closed)
            blocks.append(under)
            head, closed = "", False
        elif s == "}":
            closed = blocks.pop()
            head = ""
        elif s == ";":
            head, closed = "", False
        elif s == "__syncthreads()":
            if any(blocks) or (re.search(r"\bif\b", head) and THREAD.search(head)):
                found.append(text.count("\n", 0, m.start()) + 1)
            head += s
        else:
            head += s
    return found


def test_the_search_finds_them():
    assert conditional_barriers("void f() { if (threadIdx.x < 8) { a(); __syncthreads(); } else { b(); } }") == [1]
    assert conditional_barriers("void f() { if (threadIdx.x < 8) { a(); }\nelse { for (;;) __syncthreads(); } }") == [2]
    assert conditional_barriers("void f() { if (lane == 0) __syncthreads(); }") == [1]
    assert conditional_barriers("void f() { if (lane == 0) { a(); } __syncthreads(); if (last) { __syncthreads(); } }") == []


@pytest.mark.parametrize("path", FILES, ids=[os.path.basename(f) for f in FILES])
def test_no_barrier_under_a_thread_condition(path):
    with open(path) as f:
        assert conditional_barriers(f.read()) == []
