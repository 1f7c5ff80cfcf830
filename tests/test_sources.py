"""What the CUDA sources must not contain: they are compiled into one library
that every rank of a multi-GPU run loads."""
import glob
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = sorted(glob.glob(os.path.join(ROOT, "main_gb300", "csrc", "*")))


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_tma_multicast(path):
    # a load into several CTAs' shared memory is for code that single-GPU runs alone use
    with open(path) as f:
        assert ".multicast" not in f.read()
