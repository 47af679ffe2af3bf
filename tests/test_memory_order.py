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


def test_early_started_kernels_read_caller_data_through_l2():
    """A kernel that may start while its predecessor runs (launch_kernel<true>) reads the caller's data
    through L2 only. Loads through L1 are left to the plan's tables, to weights of one-kernel transforms, whose
    weighted kernels are ordinary launches, and to ld_cached in the kernels named here, which are ordinary launches or (the
    uneven kernel) fence after their wait."""
    tables = ("tw", "stw", "lo", "hi", "a.tw_lo", "a.tw_hi")
    src = sources()
    weighted = set()
    for name, text in src.items():
        for args in re.findall(r"__ldg\(\(?([\w.]+)", text):
            assert args in tables + ("pre", "post") or (name == "fft_fused.cu" and args == "w"), (name, args)
            if args in ("pre", "post"):
                weighted.add(name)
        # every explicit global load but ld_cached's is an L2 one
        for function, body in re.findall(r"float[24] (\w+)\(const float2\* p\) \{(.*?)\n\}", text, flags=re.S):
            assert ("ld.global.cg" in body) == (function != "ld_cached"), (name, function)
        assert len(re.findall(r'"ld\.global\.v\d', text)) == (name == "fft_tiles.cuh"), name
        uses = len(re.findall(r"\bld_cached\(", text))
        assert uses == {"fft_tiles.cuh": 3, "fft_fused.cu": 1}.get(name, 0), (name, uses)
        # launches that read weights, or the batched tiles through L1, are ordinary ones
        for dependent, kernel in re.findall(r"launch_kernel<([^>]*)>\(([\w<>, ]+?), ", text):
            assert dependent in ("!W", "!L1", "true", "false"), (name, dependent)
            if dependent == "true":
                assert name in ("fft_kernels.cu", "fft_tma.cu", "fft_wide.cu"), (name, kernel)
    assert weighted == {"fft_tiles.cuh", "fft_kernels.cu", "fft_cluster.cu", "fft_long.cu"}
    assert "launch_kernel" not in src["fft_fused.cu"] + src["fft_tc.cu"]
    assert re.search(r"L1 \? ld_cached\(", src["fft_tiles.cuh"])
    assert re.search(r"launch_kernel<!L1>\(kernel, dim3\(\(unsigned\)now\), THREADS", src["fft_kernels.cu"])
    assert re.search(r"dependent_wait\(\);\s*if \(tid == 0\) \{\s*__threadfence\(\);.*?__syncthreads\(\);", src["uneven.cu"], flags=re.S)
