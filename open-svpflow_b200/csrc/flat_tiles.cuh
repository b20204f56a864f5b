// flat_tiles.cuh -- how a CTA goes through a tile of a plane's chunks (included by super.cu; compiles for the host too).

// Chunks e * tile .. (e + 1) * tile - 1, each of them once: a thread takes two that lie `threads` apart in one go
// where the tile holds both and two() takes them, else one at a time.
template <class TWO, class ONE>
__device__ __forceinline__ void tile_chunks(uint32_t e, uint32_t tile, uint32_t thread, uint32_t threads, TWO two, ONE one) {
    const uint32_t end = (e + 1) * tile;
    for (uint32_t c = e * tile + thread; c < end; c += 2 * threads) {
        const bool both = c + threads < end;
        if (both && two(c, c + threads)) continue;
        one(c);
        if (both) one(c + threads);
    }
}
