"""Super's path for packed frames: a tile of level-0 chunks (csrc/flat_tiles.cuh, the loop the kernel runs, compiled
for the host) does every chunk of a plane once, whatever the tile's size and whichever pairs can be taken together;
frame counts around the line between its two ways to the last levels, against the oracle."""
import os
import subprocess

import numpy as np
import pytest

from oracle import oracle as orc
from test_px16 import clip10

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "open-svpflow_b200", "csrc")
PROGRAM = r"""
#include <stdint.h>
#include <stdio.h>
#include <vector>
#define __device__
#define __forceinline__ inline
#include "flat_tiles.cuh"
int main() {
    const uint32_t threads = 256;
    for (uint32_t tile : {256u, 512u, 768u, 1024u})
        for (uint32_t chunks : {1u, 255u, 256u, 257u, 1024u, 14400u}) {
            const uint32_t tiles = (chunks + tile) / tile;
            std::vector<int> done(tiles * tile, 0);
            for (uint32_t e = 0; e < tiles; e++)
                for (uint32_t t = 0; t < threads; t++)
                    tile_chunks(e, tile, t, threads,
                        [&](uint32_t a, uint32_t b) { if (a % 7 == 0 || b >= chunks) return false; done.at(a)++; done.at(b)++; return true; },
                        [&](uint32_t c) { done.at(c)++; });
            for (uint32_t c = 0; c < tiles * tile; c++)
                if (done[c] != 1) { printf("tile %u, %u chunks: chunk %u done %d times\n", tile, chunks, c, done[c]); return 1; }
        }
    return 0;
}
"""


def test_every_chunk_is_done_once(tmp_path):
    src, exe = tmp_path / "t.cpp", str(tmp_path / "t")
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [8, 10])
@pytest.mark.parametrize("frames", [4, 5, 6])
def test_super_around_the_most_frames_of_the_tail(frames, bits):
    # the last levels go to clusters that are all resident at once (5 frames on 148 SMs), else to a launch each
    import svpflow_b200 as sv

    w, h, opt = 326, 182, "{pel:2}"
    if bits > 8:
        clip = clip10(w, h, frames, 60 + frames)
    else:
        from svpflow_b200.synth import make_clip

        clip = make_clip(w, h, frames, seed=60 + frames)
    so = orc.super_opts(w, h, opt)
    want = orc.build_super_many16(so, clip) if bits > 8 else orc.build_super_many(so, clip, os.cpu_count() or 1)
    assert np.array_equal(sv.Super(w, h, opt, bits=bits).build_many(clip), want)
