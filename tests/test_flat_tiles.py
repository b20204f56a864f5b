"""A tile of Super's level-0 chunks (csrc/flat_tiles.cuh, the loop the kernel runs, compiled for the host): every
chunk of a plane is done once, whatever the tile's size and whichever pairs can be taken together."""
import os
import subprocess

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
