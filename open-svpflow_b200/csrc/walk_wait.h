// walk_wait.h -- how long a warp of a walk (walk_level in analyse_body.cuh) waits for another one.
//
// The blocks of a direction form a chain: a block waits for its neighbours, they for theirs, and kMaxWalkers of
// them (one per warp) are in work at a time. So the bound on a wait is the time that many blocks take one after
// another with the widest search that the level's options allow. (A bound of one block, started anew whenever
// one finishes, would be tighter; counting them costs 1.7 % of 32 frames of 640x360 by an addition per block and
// 3 to 5 % by a look at the level's words during the wait.)
#pragma once
#include <stdint.h>

namespace svpf {

constexpr int kMaxWalkers = 64;                        // warps of a direction that may walk a level
constexpr int64_t kWaitCycles = 1000000000;            // SM cycles, about 0.5 s at 1.9 GHz: what any wait may take
constexpr int64_t kMostWaitCycles = (int64_t)1 << 36;  // about 35 s, whatever the options ask for
// A candidate by one warp: on the general path, with 20 warps per SM, a 32x32 block with chroma is some 3,000
// instructions of which an SM issues one per warp every 5 cycles.
constexpr int64_t kCandidateCycles = 1 << 14;
// Searches of one block: the first, one for each of up to 8 neighbours whose vector changes, rounded up.
constexpr int64_t kBlockSearches = 10;

// The candidates of one search of a block, at most: special ones, the refinement of `type` (4 exhaustive, 3 UMH,
// 2 hexagons) and radius `radius`, the bad-SAD expansion of range `bad_range` where `expands`.
inline double most_candidates(int32_t type, int32_t radius, bool expands, int32_t bad_range) {
    const auto hex = [](double r) { return 6 + 3 * (r / 2) + 8; };
    const auto umh = [](double r) { return 4 * (r / 2) + 16 * (r / 4 > 1 ? r / 4 : 1); };
    const double r = (double)(radius < 0 ? 0 : radius) + 1;  // the adaptive radius reaches one more
    double n = 13;
    if (type == 4) n += (2 * r + 1) * (2 * r + 1);
    if (type == 3) n += umh(r);
    if (type == 3 || type == 2) n += hex(r);
    if (expands) {
        const double b = bad_range < 0 ? -(double)bad_range : (double)bad_range;
        n += bad_range < 0 ? 4 * b * b + 4 * b : umh(b) + hex(b);
        n += 8;
    }
    return n;
}
// The cycles after which a wait gives up.
inline int64_t wait_cycles(double candidates) {
    const double c = (double)kWaitCycles + (double)(kMaxWalkers * kBlockSearches * kCandidateCycles) * candidates;
    return c < (double)kMostWaitCycles ? (int64_t)c : kMostWaitCycles;
}

}  // namespace svpf
