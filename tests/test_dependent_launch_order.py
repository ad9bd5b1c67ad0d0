"""Kernels that hold tensor memory let their dependents start only once they have it.

A CTA of a dependent kernel may take tensor memory and then wait for its predecessor; a predecessor whose CTA still waits for
the columns that it holds would never finish.  Which kernels share an SM is a matter of sizes, so the order is read from the
sources instead of being provoked.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc")


def kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "**", "*.cu"), recursive=True)):
        with open(path) as f:
            code = re.sub(r"//[^\n]*", "", f.read())
        for body in re.split(r"\b__global__\b", code)[1:]:
            if "tcgen05.alloc" in body and "pdl_trigger()" in body:
                yield pytest.param(body, id=f"{os.path.basename(path)}:{re.search(r'(\w+_kernel)', body).group(1)}")


def test_there_are_such_kernels():
    assert len(list(kernels())) >= 5


@pytest.mark.parametrize("body", list(kernels()))
def test_trigger_follows_the_allocation(body):
    assert body.index("tcgen05.alloc") < body.index("pdl_trigger()")
