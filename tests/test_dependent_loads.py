"""Kernels of a pass start before the one ahead of them has ended, so what that
one writes is not read-only while they run."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpuseed_gb300", "csrc")


@pytest.mark.parametrize("name,read_only", [
    # the index, which no kernel of a pass writes
    ("gs_post.cu", {"&I"}),
    # ... and the bases of the reads, there before a pass's first kernel
    ("gs_search.cu", {"&I", "(const uint32_t *)(a0 - (uintptr_t)d) + lane", "wp + k"}),
    ("gs_scan.cuh", set()),
])
def test_read_only_loads(name, read_only):
    """Read-only loads are of what no kernel of a pass writes."""
    text = open(os.path.join(CSRC, name)).read()
    loads = [m.group(1) for m in re.finditer(r"__ldg\((.*)\)", text)]
    for load in loads:
        assert any(load.startswith(r) for r in read_only), f"{name}: __ldg({load})"
