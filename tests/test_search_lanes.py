"""A block's search state is one copy per warp, moved on by all lanes alike. On the host: 32 threads that share
one copy and run out of step take the same steps, to the same result, as a single one (csrc/search_steps.cuh,
the code that the kernels run)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "open-svpflow_b200", "csrc")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("lanes") / "search_lanes")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, os.path.join(HERE, "search_lanes.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("seed", [1, 2])
def test_lanes_out_of_step_take_the_steps_of_one(program, seed):
    run = lambda lanes: subprocess.run([program, str(lanes), str(seed)], capture_output=True, text=True, timeout=120)
    one, warp = run(1), run(32)
    assert one.returncode == 0 and one.stdout.count("=") == 6 and len(one.stdout.splitlines()) > 60
    assert warp.returncode == 0, warp.stdout[-200:]
    assert warp.stdout == one.stdout


def test_words_of_other_warps_decide_for_the_whole_warp():
    # a direction's words (CTL_*) change under a walk: a branch into votes and shuffles takes one load of them,
    # broadcast (ld_warp_word), never each lane's own
    with open(os.path.join(CSRC, "analyse_body.cuh")) as f:
        src = f.read()
    assert "ld_word(ctl" not in src
    assert src.count("ld_warp_word(ctl + CTL_BAD)") == 3
