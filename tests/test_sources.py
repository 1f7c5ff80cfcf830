"""What the CUDA sources must not contain: they are compiled into one library
that every rank of a multi-GPU run loads."""
import glob
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = sorted(glob.glob(os.path.join(ROOT, "main_gb300", "csrc", "*")))


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_tma_multicast(path):
    # a load into several CTAs' shared memory is for code that single-GPU runs alone use
    with open(path) as f:
        assert ".multicast" not in f.read()


def kernels(text):
    """(name, body) of every __global__ function."""
    for m in re.finditer(r"__global__\s+void\b", text):
        at = text.index("{", text.index(") {", m.end()))
        depth, i = 0, at
        while True:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
            if depth == 0:
                break
        yield re.search(r"\b(k_\w+)\s*\(", text[m.end():]).group(1), text[at:i]


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_chained_kernels_wait_before_they_let_the_next_one_start(path):
    # a kernel may then read, ahead of its own wait, whatever the one right before it does not write
    with open(path) as f:
        for name, body in kernels(f.read()):
            let = body.find("let_next_start()")
            assert let < 0 or body.find("wait_for_previous()", let) < 0, name


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_state_read_before_the_wait_comes_from_l2(path):
    # until a kernel has waited, its SM's L1 may hold lines that an earlier kernel of the chain has changed since
    with open(path) as f:
        for name, body in kernels(f.read()):
            ahead = body[:max(body.find("after_previous()"), body.find("wait_for_previous()"), 0)]
            assert not re.findall(r"(?<!&)\bd(?:\.\w+)+(?:->|\s*\[)", ahead), name
