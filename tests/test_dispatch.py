"""CPU tests of which kernels a call is routed to: the library's host code compiled against a stand-in for
the CUDA runtime and the kernel launchers (tests/c_api/check_dispatch.cpp), which prints every launch.
"""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_HOME = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def launches(tmp_path_factory):
    cxx = next((c for c in map(shutil.which, ("c++", "g++")) if c), None)
    inc = os.path.join(CUDA_HOME, "include")
    if cxx is None or not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("no C++ compiler or no CUDA runtime headers")
    csrc = os.path.join(ROOT, "onefft_b200", "csrc")
    exe = str(tmp_path_factory.mktemp("dispatch") / "check_dispatch")
    cmd = [cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), "-I", csrc, "-I", inc, "-x", "c++",
           os.path.join(csrc, "onefft_api.cu"), os.path.join(ROOT, "tests", "c_api", "check_dispatch.cpp"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(*args) -> list[str]:
        r = subprocess.run([exe, *map(str, args)], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout.splitlines()
    return run


def test_uneven_batch_runs_on_its_own_device(launches):
    """A batch made on device 0 runs there whatever device is current, below and beyond the span from which
    on its kernel is launched directly."""
    assert launches("uneven_device") == ["graph on device 0", "graph on device 0", "kernel on device 0", "graph on device 0"]


@pytest.mark.parametrize("log2n,width,kernel", [(13, None, "long"), (13, -1, "long"), (13, 15, "long"), (13, 0, "batched"),
                                                (14, None, "long"), (14, -1, "long"), (14, 0, "batched"), (12, None, "batched"),
                                                (12, 15, "pipe"), (12, 0, "batched"), (12, 1, "batched"), (14, 15, None), (13, 1, None)])
@pytest.mark.parametrize("shift", [0, 1])  # offset of the buffers in complex values: 1 = not 16-byte aligned
def test_explicit_width_selects_its_kernel(launches, log2n, width, kernel, shift):
    """onefft_plan_create_tiles with one kernel: a width given runs k_batched with it, the pipelined choice
    and the tuned one (NULL or -1) the pipelined kernels where the input is aligned."""
    got = launches("widths", log2n, shift, *([] if width is None else [width]))
    if kernel is None:
        assert got == [f"invalid pass split for n={1 << log2n}"]
        return
    assert len(got) == 1
    words = got[0].split()
    assert words[0] == (kernel if shift == 0 else "batched")
    if kernel == "batched" and width is not None and width >= 0:
        assert words[2] == str(width)  # (the stand-in prints the width as the mode)


@pytest.mark.parametrize("log2n", [15, 16, 17, 20])
def test_batches_beyond_a_launch_keep_their_kernels(launches, log2n):
    """Aligned batches of more than 65535 transforms go through the same kernels as smaller ones, in slices
    (so a transform's bits do not depend on its batch); unaligned ones are one call of the plain passes."""
    small = [line.split() for line in launches("default", log2n, 60000, 0)]
    for batch, sizes in ((65535, [65535]), (65536, [65535, 1]), (131471, [65535, 65535, 401])):
        got = [line.split() for line in launches("default", log2n, batch, 0)]
        first = 0
        for size in sizes:
            # the last slice of 2^15 may be short of the cluster kernel's line
            want = [line.split() for line in launches("default", log2n, size, 0)]
            for words in want:
                mine = got.pop(0)
                assert mine[:7] == words[:7]
                assert int(mine[8]) - int(words[8]) == int(mine[10]) - int(words[10]) == first << log2n
            if size == 65535:
                assert [w[:5] for w in want] == [w[:5] for w in small]
            first += size
        assert got == []
    assert {line.split()[0] for line in launches("default", log2n, 65536, 1)} == {"pass"}
