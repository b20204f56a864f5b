// The steps of a block's search (csrc/search_steps.cuh) played through on the host: `lanes` threads share one
// Search as the lanes of a warp do, each delayed by its own amount before every call, and print what they did.
// usage: search_lanes <lanes> <seed>
#include <pthread.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

#include <string>
#include <thread>
#include <vector>

#define __device__
#define __constant__ static const
#define __forceinline__ inline
struct int2 {
    int x, y;
};
static inline int2 make_int2(int x, int y) { return int2{x, y}; }
static pthread_barrier_t meet;
static inline void __syncwarp() { pthread_barrier_wait(&meet); }

#include "search_steps.cuh"

struct Level {
    int pel;
};
struct Params {
    int coarse_bad_sad, coarse_bad_range;
};
struct Ctx {
    const Params *P;
    const Level *L;
    int level;
};
struct Blk {
    int bnd0, bnd1, bnd2, bnd3;
};

static uint64_t mix(uint64_t v) {
    v = (v ^ (v >> 31)) * 0x9E3779B97F4A7C15ull;
    return v ^ (v >> 29);
}

struct Case {
    int stype, radius, bad_sad, bad_range, pel;
};

static void lane_main(int lane, int lanes, uint64_t seed, const Case &c, Search &q, std::string &out) {
    const Params P{c.bad_sad, c.bad_range};
    const Level L{c.pel};
    const Ctx x{&P, &L, 1};
    const Blk b{-60, -60, 61, 61};
    uint64_t r = mix(seed * 977 + (uint64_t)lane);
    auto lag = [&] {
        r = mix(r + 1);
        if (lanes > 1)
            for (volatile int k = (int)(r % 20000); k > 0; k--) {}
    };
    // a bowl with bumps: the search walks for a while, and the expansions find something now and then
    auto cost_of = [&](int2 m) {
        const long long dx = m.x - 21, dy = m.y + 13;
        return 400 + dx * dx + dy * dy + (long long)(mix(seed ^ mix((uint64_t)(m.x * 4096 + m.y))) % 90);
    };
    if (lane == 0) {
        q = Search{};
        q.stype = c.stype; q.radius = c.radius;
        q.bcost = cost_of(make_int2(0, 0)); q.bsad = (unsigned)q.bcost;
        q.own_x = 3; q.own_y = -2;
    }
    __syncwarp();
    search_begin(q, RS_ALL);
    int bad = 0;
    char line[128];
    for (int steps = 0; steps < 500; steps++) {
        Gen g{0, 0, 0, 0, 0, 0, 0};
        lag();
        if (!search_next(q, x, b, 5, bad, g)) break;
        lag();
        long long cost = q.bcost;
        unsigned sad = q.bsad;
        int w = -1;
        for (int i = 0; i < g.n; i++) {
            const int2 m = gen_mv(g, i);
            if (m.x < b.bnd0 || m.y < b.bnd1 || m.x >= b.bnd2 || m.y >= b.bnd3) continue;
            const long long k = cost_of(m);
            if (k < cost) { cost = k; sad = (unsigned)k; w = i; }
        }
        pthread_barrier_wait(&meet);  // the evaluation's votes and shuffles
        q.bcost = cost;
        q.bsad = sad;
        lag();
        search_took(q, g, w);
        snprintf(line, sizeof(line), "%d %d %d %d %d %d: %d\n", g.kind, g.cx, g.cy, g.r, g.odir, g.n, w);
        out += line;
    }
    __syncwarp();
    snprintf(line, sizeof(line), "= %d %d %u %lld %d\n", q.bmx, q.bmy, q.bsad, q.bcost, bad);
    out += line;
}

int main(int argc, char **argv) {
    const int lanes = argc > 1 ? atoi(argv[1]) : 32;
    const uint64_t seed = argc > 2 ? (uint64_t)atoll(argv[2]) : 1;
    const Case cases[] = {{2, 16, 0, 0, 1}, {3, 12, 0, 0, 1}, {4, 4, 0, 0, 1}, {2, 8, 5, -9, 2}, {4, 1, 5, 7, 1}, {0, 1, 5, -40, 1}};
    pthread_barrier_init(&meet, nullptr, (unsigned)lanes);
    for (const Case &c : cases) {
        Search q;
        std::vector<std::string> out((size_t)lanes);
        std::vector<std::thread> th;
        for (int l = 0; l < lanes; l++) th.emplace_back([&, l] { lane_main(l, lanes, seed, c, q, out[(size_t)l]); });
        for (auto &t : th) t.join();
        for (int l = 1; l < lanes; l++)
            if (out[(size_t)l] != out[0]) { printf("lane %d differs from lane 0\n", l); return 1; }
        fputs(out[0].c_str(), stdout);
    }
    return 0;
}
