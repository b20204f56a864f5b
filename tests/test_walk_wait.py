"""The bound on a walk's waits (csrc/walk_wait.h, compiled for the host) grows with what the options let a block's
search evaluate and covers a chain of as many blocks as are in work at a time."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "open-svpflow_b200", "csrc")
PROGRAM = r"""
#include <stdio.h>
#include <initializer_list>
#include "walk_wait.h"
using namespace svpf;
#define CHECK(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main() {
    // candidates counted step by step, against the formula
    for (int r = 0; r <= 100; r++) {
        int umh = 2 * (r / 2) * 2 + 16 * (r / 4 > 1 ? r / 4 : 1), hex = 6 + 3 * (r / 2) + 8, rings = 0;
        for (int k = 1; k < r; k++) rings += 4 * ((2 * k - 1) / 1) + 4;
        CHECK(most_candidates(4, r, false, 0) >= 13 + (2 * r + 1) * (2 * r + 1));
        CHECK(most_candidates(3, r, false, 0) >= 13 + umh + hex);
        CHECK(most_candidates(2, r, true, -r) >= 13 + hex + rings + 8);
        CHECK(most_candidates(2, r, true, r) >= 13 + hex + umh + hex + 8);
    }
    // the chain's blocks one after another, each searched ten times, 5000 cycles a candidate, fit threefold
    for (int r : {2, 8, 16, 24}) {
        const double n = (2.0 * r + 1) * (2.0 * r + 1);
        CHECK(wait_cycles(most_candidates(4, r, false, 0)) >= 3 * kMaxWalkers * 10 * 5000.0 * n);
    }
    // a wide search of large blocks, whose chain passes half a second
    CHECK(wait_cycles(most_candidates(4, 64, false, 0)) >= 64 * 10 * 5000.0 * 129 * 129);
    for (int r = 1; r < 4096; r *= 2) CHECK(wait_cycles(most_candidates(4, r, false, 0)) <= wait_cycles(most_candidates(4, 2 * r, false, 0)));
    CHECK(wait_cycles(0) == kWaitCycles && wait_cycles(1e30) == kMostWaitCycles);
    CHECK(wait_cycles(most_candidates(4, 2147483647, true, -2147483647)) == kMostWaitCycles);
    return 0;
}
"""


def test_waits_outlast_the_chain_they_wait_for(tmp_path):
    src, exe = tmp_path / "t.cpp", str(tmp_path / "t")
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_residency_is_asked_of_the_kernel_that_is_launched():
    # a walk's CTAs wait on one another, so its grid is sized by the occupancy of the very kernel it launches: the shape
    # that holds the answer holds the kernel too, and the plain and the batch's walks each make their own
    with open(os.path.join(CSRC, "analyse_body.cuh")) as f:
        src = f.read()
    assert src.count("cudaLaunchKernelEx(&cfg, w.kernel, args...)") == src.count("cudaLaunchKernelEx(") == 1
    for name in ("analyse", "batch"):
        assert f"walk_shape({name}_walk_kernel<kWalkPerSM>, {name}_walk_kernel<kDensePerSM>" in src
        assert f"cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, {name}_walk_kernel" not in src
