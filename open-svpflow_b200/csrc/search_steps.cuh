// search_steps.cuh -- the steps of one block's search: candidate generators and the state machine that
// issues them (included by analyse_body.cuh inside its namespace; holds nothing but that, so that it also
// compiles for the host, where lanes that do not run in step can be played through).
//
// Follows crates/svpflow1/src/analyse_search.rs: exact_search_block :684-768, exact_refine_search :771-826,
// exact_expanding :849-885, exact_hex2 :942-1033, exact_umh :1036-1119, the bad-SAD expansion :611-672.

__device__ __forceinline__ int imin(int a, int b) { return a < b ? a : b; }
__device__ __forceinline__ int imax(int a, int b) { return a > b ? a : b; }
__device__ __forceinline__ int iclamp(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }
__device__ __forceinline__ int sat_i32(long long r) {
    return r > 2147483647LL ? 2147483647 : (r < -2147483648LL ? (int)0x80000000 : (int)r);
}

enum : int { BK_EXH = 1, BK_UMH, BK_HEX6, BK_HEX3, BK_RING };

// What a block's search keeps from turn to turn, identical in every lane of the warp (see search_next). One copy
// per warp in shared memory, which every lane reads and writes alike, and lanes need not run in step. So whatever
// changes a word of it has read all it needs, meets the other lanes (__syncwarp), stores, and meets them again: no
// lane sees a word that another has moved on already, or moves one on twice.
struct Search {
    int state, stage, stype, radius;
    int predx, predy;                       // predictor of the motion penalty
    int lambda, own_x, own_y, ppx, ppy;     // the block's penalty factor, its own predictor and the refinement's
    int bmx, bmy;                           // the best so far
    unsigned bsad;
    long long bcost;
    int hbx, hby, hdir, hi, hrad, hret, bad_r, bad_max;
    unsigned found;
    int sets_mv;
    int rx, ry;                             // a walk: the outcome before a bad-SAD expansion made ahead of the test
    unsigned rsad;
    long long rcost;
};

// candidate generators (the reference's loop orders)
__constant__ int2 c_hex2[8] = {{-1, -2}, {-2, 0}, {-1, 2}, {1, 2}, {2, 0}, {1, -2}, {-1, -2}, {-2, 0}};  // :889-898
__constant__ int c_mod6m1[8] = {5, 0, 1, 2, 3, 4, 5, 0};
__constant__ int2 c_hex4[16] = {{-4, 2}, {-4, 1}, {-4, 0}, {-4, -1}, {-4, -2}, {4, -2}, {4, -1}, {4, 0},
                                {4, 1},  {4, 2},  {2, 3},  {0, 4},   {-2, 3},  {-2, -3}, {0, -4}, {2, -3}};  // :1075-1092

struct Gen {
    int kind, cx, cy, r, step, odir, n;
};
__device__ __forceinline__ int ring_m(int r, int step) { return 2 * r > step ? (2 * r - 1) / step : 0; }
__device__ __forceinline__ Gen make_gen(int kind, int cx, int cy, int r, int step, int odir) {
    Gen g{kind, cx, cy, r, step, odir, 0};
    switch (kind) {
    case BK_EXH: g.n = (2 * r + 1) * (2 * r + 1); break;
    case BK_UMH: g.n = 4 * (r / 2 > 0 ? r / 2 : 0) + 16 * imax(r / 4, 1); break;
    case BK_HEX6: g.n = 6; break;
    case BK_HEX3: g.n = 3; break;
    case BK_RING: g.n = 4 * ring_m(r, step) + 4; break;
    }
    return g;
}
__device__ int2 gen_mv(const Gen &g, int i) {
    const int cx = g.cx, cy = g.cy, r = g.r;
    switch (g.kind) {
    case BK_EXH: {  // exact_refine_search type 4, :799-823 (raster over the square)
        const int w = 2 * r + 1;
        return make_int2(cx - r + i % w, cy - r + i / w);
    }
    case BK_UMH: {  // exact_umh, :1055-1114
        const int nd = r / 2;
        if (i < 2 * nd) { int dd = 1 + 2 * (i >> 1); return make_int2(cx + ((i & 1) ? dd : -dd), cy); }
        i -= 2 * nd;
        if (i < 2 * nd) { int dd = 1 + 2 * (i >> 1); return make_int2(cx, cy + ((i & 1) ? dd : -dd)); }
        i -= 2 * nd;
        const int scale = 1 + i / 16;
        const int2 h = c_hex4[i % 16];
        return make_int2(cx + h.x * scale, cy + h.y * scale);
    }
    case BK_HEX6: { int2 h = c_hex2[i + 1]; return make_int2(cx + h.x, cy + h.y); }
    case BK_HEX3: { int2 h = c_hex2[g.odir + i]; return make_int2(cx + h.x, cy + h.y); }
    case BK_RING: {  // exact_expanding, :849-885
        const int step = g.step, m = ring_m(r, step);
        if (i < 2 * m) { int off = -r + step + (i >> 1) * step; return make_int2(cx + off, (i & 1) ? cy + r : cy - r); }
        i -= 2 * m;
        if (i < 2 * m) { int off = -r + step + (i >> 1) * step; return make_int2((i & 1) ? cx + r : cx - r, cy + off); }
        i -= 2 * m;
        const int sx = (i < 2) ? -r : r, sy = (i & 1) ? r : -r;
        return make_int2(cx + sx, cy + sy);
    }
    }
    return make_int2(0, 0);
}

// The bad-SAD threshold after `count` bad blocks (:605-616).
template <class PARAMS>
__device__ __forceinline__ int bad_limit(const PARAMS &P, int count) {
    return sat_i32((long long)P.coarse_bad_sad + (long long)(sat_i32((long long)P.coarse_bad_sad * count) / 16));
}

// search states of one block (exact_search_block :684-768, exact_refine_search :771-826,
// exact_hex2 :942-1033, exact_umh :1036-1119, bad-SAD expansion :611-672)
enum { S_REFINE, S_HEX_START, S_HEX_ITER, S_HEX_EXIT, S_BAD, S_BAD_RING, S_FINAL_RING, S_STORE };

// The refinement and bad-SAD expansion of one block (exact_refine_search :771-826,
// exact_hex2 :942-1033, exact_umh :1036-1119, the expansion :611-672): a state machine
// replicated in every thread of the direction, issuing one evaluation step at a time.
// (ppx, ppy): predictor of the motion penalty; (own_x, own_y): the block's own predictor,
// which the bad-SAD expansion switches to. `stage`: RS_ALL runs the refinement and the
// expansion, RS_REFINE_ONLY stops where the expansion's test begins, RS_BAD_ONLY starts
// there (a walk runs the two apart: the test reads the bad count of the blocks before),
// RS_NONE runs nothing.
enum { RS_NONE, RS_ALL, RS_REFINE_ONLY, RS_BAD_ONLY };
// Begins it; the lanes have met since any of them read what it sets.
__device__ __forceinline__ void search_begin(Search &q, int stage) {
    q.stage = stage;
    q.predx = q.ppx; q.predy = q.ppy;
    q.state = stage == RS_NONE ? S_STORE : (stage == RS_BAD_ONLY ? S_BAD : S_REFINE);
    q.hdir = -2; q.hi = q.hrad = q.hret = 0;
    __syncwarp();
}
// The next step's candidates; false when there is none. `state` and `bad_r` (q.state, q.bad_r) are the
// words that a call reads and moves on; of the others it only sets what it does not read.
template <class CTX, class BLK>
__device__ __forceinline__ bool search_step(Search &q, const CTX &x, const BLK &b, int64_t idx, int &bad_count, Gen &g,
                                            int &state, int bad_r, bool &sets_mv) {
    const auto &P = *x.P;
    const auto &L = *x.L;
    while (state != S_STORE) {
        if (state == S_BAD && q.stage == RS_REFINE_ONLY) {
            state = S_STORE;
            break;
        }
        if (state == S_REFINE) {
            if (q.stype == 4) { state = S_BAD; g = make_gen(BK_EXH, q.bmx, q.bmy, q.radius, 0, 0); return true; }
            if (q.stype == 3) {
                state = S_HEX_START; q.hrad = q.radius; q.hret = 0;
                g = make_gen(BK_UMH, q.bmx, q.bmy, q.radius, 0, 0);
                return true;
            }
            if (q.stype == 2) { state = S_HEX_START; q.hrad = q.radius; q.hret = 0; }
            else state = S_BAD;
        } else if (state == S_HEX_START) {
            q.hbx = q.bmx; q.hby = q.bmy;
            if (q.hrad > 1) { sets_mv = false; state = S_HEX_ITER; g = make_gen(BK_HEX6, q.bmx, q.bmy, 0, 0, 0); return true; }
            state = q.hret ? S_FINAL_RING : S_BAD;
            g = make_gen(BK_RING, q.bmx, q.bmy, 1, 1, 0);
            return true;
        } else if (state == S_HEX_ITER) {
            if (q.hi < q.hrad / 2 && q.hbx >= b.bnd0 && q.hby >= b.bnd1 && q.hbx < b.bnd2 && q.hby < b.bnd3) {
                sets_mv = false;
                g = make_gen(BK_HEX3, q.hbx, q.hby, 0, 0, c_mod6m1[q.hdir + 1]);
                return true;
            }
            state = S_HEX_EXIT;
        } else if (state == S_HEX_EXIT) {
            q.bmx = q.hbx; q.bmy = q.hby;
            state = q.hret ? S_FINAL_RING : S_BAD;
            g = make_gen(BK_RING, q.hbx, q.hby, 1, 1, 0);
            return true;
        } else if (state == S_BAD) {
            q.found = q.bsad;
            if (x.level > 0 && idx > 1 && P.coarse_bad_sad > 0 && (int)q.bsad > bad_limit(P, bad_count)) {
                bad_count++;
                q.predx = q.own_x; q.predy = q.own_y;  // the block's own predictor
                if (P.coarse_bad_range < 0) {
                    const int bad_max = -P.coarse_bad_range * L.pel;
                    q.bad_max = bad_max; q.bad_r = L.pel;
                    if (L.pel < bad_max) { state = S_BAD_RING; g = make_gen(BK_RING, 0, 0, L.pel, L.pel, 0); return true; }
                    state = S_FINAL_RING;
                } else if (P.coarse_bad_range > 0) {
                    q.hrad = P.coarse_bad_range * L.pel; q.hret = 1;
                    state = S_HEX_START;
                    g = make_gen(BK_UMH, 0, 0, P.coarse_bad_range * L.pel, 0, 0);
                    return true;
                } else state = S_FINAL_RING;
            } else state = S_STORE;
        } else if (state == S_BAD_RING) {
            if (q.bsad < q.found / 4) state = S_FINAL_RING;
            else {
                q.bad_r = bad_r + L.pel;
                if (bad_r + L.pel < q.bad_max) { g = make_gen(BK_RING, 0, 0, bad_r + L.pel, L.pel, 0); return true; }
                state = S_FINAL_RING;
            }
        } else {  // S_FINAL_RING
            state = S_STORE;
            g = make_gen(BK_RING, q.bmx, q.bmy, 1, 1, 0);
            return true;
        }
    }
    return false;
}
template <class CTX, class BLK>
__device__ __forceinline__ bool search_next(Search &q, const CTX &x, const BLK &b, int64_t idx, int &bad_count, Gen &g) {
    int state = q.state;
    const int bad_r = q.bad_r;
    bool sets_mv = true;
    __syncwarp();
    const bool more = search_step(q, x, b, idx, bad_count, g, state, bad_r, sets_mv);
    q.state = state;
    q.sets_mv = sets_mv;
    __syncwarp();
    return more;
}
// The step's outcome: candidate w of g was accepted (its cost and sad are in bcost, q.bsad), or none (-1).
__device__ __forceinline__ void search_took(Search &q, const Gen &g, int w) {
    const bool hex = g.kind == BK_HEX6 || g.kind == BK_HEX3, sets_mv = q.sets_mv != 0;
    const int hbx = q.hbx, hby = q.hby, hi = q.hi;
    __syncwarp();
    if (hex) {  // exact_check_dir: a label, best.mv set at exit
        if (w >= 0) {
            const int hdir = g.kind == BK_HEX6 ? w : g.odir + w - 1;
            q.hdir = hdir;
            q.hbx = hbx + c_hex2[hdir + 1].x; q.hby = hby + c_hex2[hdir + 1].y;
            q.hi = g.kind == BK_HEX6 ? 1 : hi + 1;
            q.state = S_HEX_ITER;
        } else q.state = S_HEX_EXIT;
    } else if (w >= 0 && sets_mv) {
        const int2 m = gen_mv(g, w);
        q.bmx = m.x; q.bmy = m.y;
    }
    __syncwarp();
}
