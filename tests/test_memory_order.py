"""CPU tests of ordering rules that the kernels' sources have to keep and that a run on the GPU shows
only by luck of timing.
"""
from __future__ import annotations

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "onefft_b200", "csrc")


def sources() -> dict[str, str]:
    """Every kernel source without its comments."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(path) as f:
            out[os.path.basename(path)] = re.sub(r"//[^\n]*", "", f.read())
    return out


def test_relaxed_cluster_arrivals_follow_a_release_fence():
    """A relaxed arrival at a cluster barrier orders no memory access: before a peer overwrites what this
    thread read, the arrival needs a release fence directly before it."""
    found = 0
    for name, src in sources().items():
        statements = re.findall(r'asm volatile\(\s*"([^"]*)', src)
        for i, s in enumerate(statements):
            if "barrier.cluster.arrive.relaxed" in s:
                found += 1
                assert i > 0 and re.match(r"fence\.(release|acq_rel)\.", statements[i - 1]), (name, s)
    assert found == 1
