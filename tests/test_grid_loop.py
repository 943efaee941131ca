"""The loop that kernels take over vertices ends, and meets every vertex once, up to 2^32 - 1 of them (on the CPU)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "comm-avoiding-cuts-cc_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "grid_loop.cuh"
// steps of the threads `first` of a grid of `stride` threads; more than any ending loop takes: exit 1
int main(int argc, char **argv) {
    const uint32_t stride = strtoul(argv[1], 0, 10), n = strtoul(argv[2], 0, 10);
    const uint32_t firsts[] = {0, 1, stride / 2, stride - 1};
    for (uint32_t first : firsts) {
        const uint64_t want = first < n ? ((uint64_t)n - first + stride - 1) / stride : 0;
        uint64_t steps = 0, last = first;
        cac::strided(first, stride, n, [&](uint32_t i) {
            if (++steps > want) exit(1);
            if (i != first + (steps - 1) * (uint64_t)stride) exit(2);
            last = i;
        });
        if (steps != want) exit(3);
        if (want && !(last < n && last + (uint64_t)stride >= n)) exit(4);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("grid_loop")
    src = d / "loop.cpp"
    src.write_text(PROGRAM)
    exe = str(d / "loop")
    subprocess.run([os.environ.get("CXX", shutil.which("g++") or "g++"), "-std=c++17", "-O1", "-I" + CSRC, str(src),
                    "-o", exe], check=True)
    return exe


# 152 SMs of 8 CTAs of 256 threads, and four times that (a thread's step in the labelling)
@pytest.mark.parametrize("stride", [152 * 8 * 256, 4 * 152 * 8 * 256])
@pytest.mark.parametrize("n", [1, 1000, 311295, 311296, 311297, 2**31 + 5, 2**32 - 1300000, 2**32 - 1245184,
                               2**32 - 1245183, 2**32 - 311296, 2**32 - 311295, 2**32 - 2, 2**32 - 1])
def test_loop_ends_below_2_32(program, stride, n):
    assert subprocess.run([program, str(stride), str(n)], timeout=60).returncode == 0
