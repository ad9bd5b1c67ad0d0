"""Kernels that give up on a bounded wait must not leave other warps of theirs at a barrier that only some warps still reach: a named
barrier has no limit, so no kernel that waits with an abort flag meets at one."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc")
FILES = sorted(os.path.join(d, f) for d, _, fs in os.walk(CSRC) for f in fs if f.endswith((".cu", ".cuh")))


@pytest.mark.parametrize("path", FILES, ids=[os.path.relpath(f, CSRC) for f in FILES])
def test_no_named_barrier_beside_bounded_waits(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    if "abort_flag" not in text:
        return
    assert not re.search(r"\b(bar|barrier)\.(cta\.)?sync(\.aligned)?\s+[%\w]+\s*,", text), "a wait without a limit"
