"""Kernels that may be launched while the kernel before them still writes (they call wait_for_previous()) read no
memory through the read-only path: __ldg asks for memory that stays unchanged for as long as the kernel runs,
which begins before its wait."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "iqm_b200", "csrc")


def _early_kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            parts = re.split(r"(?m)^(?=__global__)", f.read())[1:]
        for part in parts:
            body = part.split("\n}\n")[0]
            name = re.search(r"(\w+)\(FsimGroup", part)
            if "wait_for_previous();" in body:
                yield pytest.param(body, id=name.group(1) if name else os.path.basename(path))


def test_the_chain_is_found():
    assert len(list(_early_kernels())) >= 6


@pytest.mark.parametrize("body", list(_early_kernels()))
def test_no_read_only_loads(body):
    assert "__ldg(" not in body and "ld.global.nc" not in body
