// analyse_body.cuh -- hierarchical block search (Analyse) on sm_100a.
//
// Included by one translation unit per launch variant (analyse_nt128.cu, analyse_nt64.cu,
// analyse_nt32.cu, analyse_nt128b3.cu, analyse_nt64b6.cu): SVPF_NT = threads per search
// direction, SVPF_MINB = resident CTAs per SM the register budget is cut for (2, 4, 8: 128
// registers per thread; 3, 6: 80), SVPF_VARIANT = the variant's namespace. Each variant
// exports a plain launcher (one CTA per pair; in the look-ahead shapes, by default, the pair
// kernel only makes the ground for each level, a cooperative walk kernel with one CTA per warp
// searches it across the SMs, and a pack kernel writes the payloads) and a persistent batch
// launcher (CTAs drain a device work queue of frame pairs from many clips).
//
// Restates crates/svpflow1/src/analyse_search.rs:68-2811 for the GPU:
//   * a frame pair has a forward search (current -> reference) and a backward search
//     (reference -> current), which meet once per level: the forward search of a level
//     needs the backward field of the level above projected onto it, and vice versa (:128-191).
//   * inside a level the blocks run in the reference's serial order (serpentine at
//     level 0, score-sorted at coarser levels, :302-419): each block takes already
//     searched neighbours as candidates, so the order is a true dependency chain. walk_level
//     keeps many blocks of it in flight, one per warp, and is exact all the same; search_level
//     takes them one by one, all warps of a direction on the same block (the batch kernel, the
//     smallest levels, inputs on which the reference panics).
//   * every step of a block's search is a batch of candidate vectors whose positions are
//     known before any is evaluated (special candidates; the UMH cross + hexagons; an
//     exhaustive square; a hexagon step; an expanding ring), 32 at a time, one per lane. The
//     lanes test their candidates and set them up side by side, the whole warp evaluates
//     those that pass one after another (eval_cands), and the first of minimal cost is kept.
//     First-minimum equals the reference's sequential `if cost < best.cost` scan (:1122-1155)
//     whenever cost >= motion penalty, i.e. pnew >= -256; below that the step replays the
//     sequential scan over the costs.
//   * a candidate whose block and reference block lie inside their planes takes the fast
//     path, one whose reference block reaches out of a plane a clamped form of it
//     (clamped_cands); any other candidate takes the reference's own read path (edge-shifted,
//     clamped, masked; :1638-2351) through cand_setup, which keeps the reference's wrapping
//     index arithmetic.
//
// SATD is a contraction with the 16x16 Sylvester matrix and runs on the tensor cores, exactly (see
// the fast path); the two f64 formulas (adapt_lambda, exact_lambda) are IEEE-exact (exact_lambda is
// host-precomputed).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include "svpf_device.h"

#if !defined(SVPF_NT) || !defined(SVPF_MINB) || !defined(SVPF_VARIANT)
#error "define SVPF_NT, SVPF_MINB and SVPF_VARIANT before including analyse_body.cuh"
#endif
// SVPF_LOOKAHEAD: the shape's plain launcher walks the levels (walk_level) when the parameter block
// asks for it. Only the 128-thread shapes with 128 registers do: the plain path and the server take
// them; the others serve batches, whose queue keeps every CTA busy with pairs of its own.
#ifndef SVPF_LOOKAHEAD
#define SVPF_LOOKAHEAD 0
#endif

namespace svpf {
namespace SVPF_VARIANT {

namespace {

#ifdef SVPF_PX16
typedef uint16_t px_t;             // this project's 10-bit extension (no reference behaviour)
constexpr unsigned PX_MID = 512;   // chroma default of the clamped read paths
constexpr unsigned DC_SHIFT = 2;   // the payload's block luma byte is mean >> 2
#else
typedef uint8_t px_t;
constexpr unsigned PX_MID = 128;
constexpr unsigned DC_SHIFT = 0;
#endif
constexpr int NT = SVPF_NT;        // threads per search direction
static_assert(NT == 32 || NT == 64 || NT == 128, "threads per direction");
constexpr int NW = NT / 32;

enum : uint8_t { LM_DIRECT = 1, LM_SATD_MASK = 2, LM_SAD_BREAK = 3, LM_EDGE = 4, LM_DC = 5 };
enum : uint8_t { CM_NONE = 0, CM_DIRECT = 1, CM_SAD_BREAK = 3, CM_EDGE = 4 };

constexpr int ST_PANIC = 1;    // status bit: the reference indexes out of range here (it would panic)
constexpr int ST_TIMEOUT = 4;  // status bit: a bounded wait inside the kernel ran out (internal error)

#include "search_steps.cuh"

struct Cand {
    int64_t l_sbase, l_rbase, c_sbase, c_rbase;  // flat bases of the direct read paths
    int32_t l_sx, l_sy, l_rx, l_ry;              // origins of the clamped / masked paths
    int32_t c_sx, c_sy, c_rx, c_ry;
    int32_t l_srow, l_rrow, c_srow, c_rrow;      // first row of the source / reference sub-plane
    int32_t c_rows;                              // chroma rows covered (n x n for square SATD)
    uint8_t lmode, cmode, lsatd, csatd;
};

// Per-block constants, identical in every thread of a direction. In shared memory, one copy per warp, like
// Search: they are read once per 32 candidates, and registers are what bounds the warps in flight.
// Changed as Search is, between two meetings of the lanes.
struct BlkC {
    int px, py, bw, bh, px2, py2;
    int bnd0, bnd1, bnd2, bnd3;            // mv_bounds
    int chroma, fast_src;
    int fx0, fx1, fy0, fy1;                // vectors taking the fast path lie in this box (inclusive) ...
    int lbase, llim, cbase, clim;          // ... and have lref <= llim, cref <= clim; the offsets (from the frame's
                                           // first sample) of the reference blocks at vector 0
    int64_t lsrc, csrc;                    // offset of the source block (luma, U)
};

// Shared state of one search direction. A block is searched by a group of warps: the whole
// direction (search_level), or one warp (a walk, the refine pass: a block per warp in
// flight). Per-warp entries are indexed by the warp's place in the direction; a group's
// entries are those of its first warp (Ctx::wbase). W: the warps it holds state for (the
// direction's, or one for a CTA of a walk).
template <int W>
struct alignas(16) DirShT {
    Search q[W];                          // per warp: its block's search ...
    BlkC blk[W];                          // ... and constants
    int lmx[W][32], lmy[W][32];           // per warp: the special candidates, one per lane, ...
    unsigned lsd[W][32];                  // ... and their exact_sad
    long long K[2][W];                    // per-warp best (cost, index, sad) of a step, double-buffered
    int I[2][W];
    unsigned S[2][W];
    unsigned slot[2][32];                 // special candidates' exact_sad, shared by a group's warps
    unsigned dc[2][W], dcs[2], score[2];  // a block's luma sum (per warp; on the general path), its predictor's re-score
    long long rk[2][32];                  // exact sequential scan: the costs of 32 candidates
    unsigned rs[2][32];
    int unsafe_;                          // the level has an input the reference panics on
    int gx, gy;           // global predictor (doubled) for the next level
    int order_len;
    int abort_;
    long long r64[W][3];
    int r32[W][2];
};
// After the directions' DirShT, per warp of each: the block's staged source (512 bytes per group of
// eight tiles) and the group's offsets (128 bytes), AnalyseParams::stage_groups of each.
constexpr int kGroupBytes = 640;
using DirSh = DirShT<NW>;  // a search direction of the pair kernels
using WarpSh = DirShT<1>;  // a CTA (one warp) of a walk or the refine pass

struct Planes {
    const px_t *y, *u, *v;
};

struct Geo {  // per level
    int lw, lh, clw, clh;
    int64_t ys, cs, ylen, clen;
    int ys32, cs32;   // the strides again, for 32-bit offsets (planes are below 2^30 bytes)
};

// Named barrier of one search direction (ids 1 and 2; 0 is __syncthreads). Immediate ids,
// so the kernel reserves three barriers, not all sixteen (barriers bound CTAs per SM).
__device__ __forceinline__ void dbar(int d) {
    if (d) asm volatile("bar.sync 2, %0;" ::"n"(NT) : "memory");
    else asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
}
__device__ __forceinline__ unsigned sat_add(unsigned a, unsigned b) { unsigned r = a + b; return r < a ? 0xFFFFFFFFu : r; }
__device__ __forceinline__ unsigned sat_mul(unsigned a, unsigned b) {
    unsigned long long r = (unsigned long long)a * b;
    return r > 0xFFFFFFFFull ? 0xFFFFFFFFu : (unsigned)r;
}
__device__ __forceinline__ bool is_blk(int n) { return n == 4 || n == 8 || n == 16 || n == 32; }
// reads of a slice: an index past the end (or a wrapped, i.e. negative, one) is None
__device__ __forceinline__ unsigned rd(const px_t *p, int64_t len, int64_t i, unsigned dflt) {
    return (i >= 0 && i < len) ? (unsigned)__ldg(p + i) : dflt;
}
__device__ __forceinline__ long long pen(int pnew, unsigned x) { return (long long)x + (((long long)pnew * (long long)x) >> 8); }
// (lambda * |pred - mv|^2) >> 8; vectors are below 2^16 in magnitude, so the differences
// fit 32 bits and the squares are single widening multiplies
__device__ __forceinline__ long long motion_penalty(int lambda, int px_, int py_, int mx, int my) {
    const int dx = px_ - mx, dy = py_ - my;
    return ((long long)lambda * ((long long)dx * dx + (long long)dy * dy)) >> 8;
}

// hadamard4_satd, analyse_search.rs:2681-2702: rows, then columns; the last column
// stage and its absolute values use |a+b| + |a-b| = 2 max(|a|, |b|).
__device__ __forceinline__ unsigned hadamard4(const int d[16]) {
    int t[16];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        int s0 = d[i * 4] + d[i * 4 + 1], s1 = d[i * 4] - d[i * 4 + 1];
        int s2 = d[i * 4 + 2] + d[i * 4 + 3], s3 = d[i * 4 + 2] - d[i * 4 + 3];
        t[i * 4] = s0 + s2; t[i * 4 + 1] = s1 + s3; t[i * 4 + 2] = s0 - s2; t[i * 4 + 3] = s1 - s3;
    }
    int s = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        int s0 = t[j] + t[4 + j], s1 = t[j] - t[4 + j], s2 = t[8 + j] + t[12 + j], s3 = t[8 + j] - t[12 + j];
        s += max(abs(s0), abs(s2)) + max(abs(s1), abs(s3));
    }
    return (unsigned)(2 * s);
}

// -------------------------------------------------------------------------------------------
// Candidate set-up on the reference's read paths (any candidate; the general path).
//   edge_shift_origins :1638-1676 / block_cost_edge_lc :1996-2167
//   block_cost_luma_interior :1719-1852 / satd_luma_clamp :2353-2436
//   chroma_sad_x4 :2169-2303
__device__ void cand_setup(Cand &c, const AnalyseParams &P, const LevelInfo &L, const Geo &G, int level, int px, int py,
                           int bw, int bh, int mvx, int mvy, bool chroma, int satd, int pel_in, bool dc) {
    const int pel = imax(pel_in, 1);
    const int lw = G.lw, lh = G.lh;
    const int64_t y_off = L.y_off, c_off = L.c_off;
    if (dc) {  // block_luma_dc, :1566-1617 (a sum over the rows/columns the loop reaches)
        c.lmode = LM_DC; c.lsatd = 0; c.cmode = CM_NONE; c.csatd = 0;
        c.l_sx = px; c.l_sy = py; c.l_srow = (int32_t)y_off;
        c.c_rows = 0;
        return;
    }
    // edge_shift_origins
    const int bminx = -pel * px, bminy = -pel * py;
    const int bmaxx = pel * (lw - px - bw) + 1, bmaxy = pel * (lh - py - bh) + 1;
    const int ox = mvx < bminx ? mvx - bminx : ((bmaxx > bminx && mvx >= bmaxx) ? mvx + 1 - bmaxx : 0);
    const int oy = mvy < bminy ? mvy - bminy : ((bmaxy > bminy && mvy >= bmaxy) ? mvy + 1 - bmaxy : 0);
    const bool l0sub = level == 0 && pel >= 2;
    if (ox != 0 || oy != 0) {
        const int cx = iclamp(px - ox, 0, imax(lw - bw, 0)), cy = iclamp(py - oy, 0, imax(lh - bh, 0));
        int rx0, ry0;
        if (pel == 1) { rx0 = cx + mvx; ry0 = cy + mvy; }
        else if (pel == 4) { rx0 = (4 * cx + mvx) >> 2; ry0 = (4 * cy + mvy) >> 2; }
        else { rx0 = (2 * cx + mvx) >> 1; ry0 = (2 * cy + mvy) >> 1; }
        const int sub = l0sub ? (mvy & 1) * pel + (mvx & 1) : 0;
        c.lmode = LM_EDGE;
        c.lsatd = satd && is_blk(bw) && is_blk(bh) && bw == bh;
        c.l_sx = cx; c.l_sy = cy; c.l_rx = rx0; c.l_ry = ry0;
        c.l_srow = (int32_t)y_off; c.l_rrow = (int32_t)(y_off + (int64_t)sub * lh);
        if (chroma) {
            const int cw = bw / 2, ch = bh / 2;
            const int ccx = (px >> 1) - ((px - cx) >> 1), ccy = (py >> 1) - ((py - cy) >> 1);
            c.cmode = CM_EDGE;
            c.csatd = satd && cw == ch && (cw == 4 || cw == 8 || cw == 16);
            c.c_sx = ccx; c.c_sy = ccy;
            c.c_rx = ((mvx >> 1) + 2 * ccx) >> 1; c.c_ry = ((mvy >> 1) + 2 * ccy) >> 1;
            c.c_srow = (int32_t)c_off; c.c_rrow = (int32_t)(c_off + (int64_t)sub * G.clh);
            c.c_rows = ch;
        } else {
            c.cmode = CM_NONE; c.csatd = 0; c.c_rows = 0;
        }
        return;
    }
    // ---- luma, no edge shift
    const int px2 = px - (level > 0 && px + bw >= lw), py2 = py - (level > 0 && py + bh >= lh);
    int mx = mvx, my = mvy, sub = 0;
    if (l0sub) { sub = (mvy & 1) * pel + (mvx & 1); mx = mvx >> 1; my = mvy >> 1; }
    const uint64_t cur_row0 = (uint64_t)y_off, ref_row0 = (uint64_t)(y_off + (int64_t)sub * lh);
    const uint64_t px_u = (uint64_t)(int64_t)px2, py_u = (uint64_t)(int64_t)py2;
    c.l_srow = (int32_t)cur_row0; c.l_rrow = (int32_t)ref_row0;
    c.l_sx = px2; c.l_sy = py2; c.l_rx = px2 + mx; c.l_ry = py2 + my;
    const uint64_t ys = (uint64_t)G.ys;
    if (satd && is_blk(bw) && is_blk(bh) && bw == bh) {
        const uint64_t n = (uint64_t)bw;
        const int rx0 = px2 + mx, ry0 = py2 + my;
        auto smul = [](uint64_t a, uint64_t b) -> uint64_t { return (a != 0 && b > ~0ull / a) ? ~0ull : a * b; };
        auto sadd = [](uint64_t a, uint64_t b) -> uint64_t { uint64_t r = a + b; return r < a ? ~0ull : r; };
        const uint64_t src_end = sadd(smul(cur_row0 + py_u + n - 1, ys), px_u + n);
        const uint64_t ref_end = ry0 >= 0 ? sadd(smul(ref_row0 + (uint64_t)ry0 + n - 1, ys), (uint64_t)imax(rx0, 0) + n) : ~0ull;
        const bool interior = px_u + n <= (uint64_t)lw && py_u + n <= (uint64_t)lh && rx0 >= 0 && ry0 >= 0 &&
                              (uint64_t)rx0 + n <= (uint64_t)lw && (uint64_t)ry0 + n <= (uint64_t)lh &&
                              src_end <= (uint64_t)G.ylen && ref_end <= (uint64_t)G.ylen;
        c.lsatd = 1;
        if (interior) {
            c.lmode = LM_DIRECT;
            c.l_sbase = (int64_t)((cur_row0 + py_u) * ys + px_u);
            c.l_rbase = (int64_t)((ref_row0 + (uint64_t)ry0) * ys + (uint64_t)rx0);
        } else {
            c.lmode = LM_SATD_MASK;
        }
    } else {
        const int rx0 = px2 + mx, ry0 = py2 + my;
        const bool interior = px2 >= 0 && py2 >= 0 && rx0 >= 0 && ry0 >= 0 && px2 + bw <= lw && py2 + bh <= lh &&
                              rx0 + bw <= lw && ry0 + bh <= lh;
        c.lsatd = 0;
        if (interior && is_blk(bw)) {
            c.lmode = LM_DIRECT;
            c.l_sbase = (int64_t)((cur_row0 + py_u) * ys + px_u);
            c.l_rbase = (int64_t)((ref_row0 + (uint64_t)ry0) * ys + (uint64_t)rx0);
        } else {
            c.lmode = LM_SAD_BREAK;
        }
    }
    // ---- chroma_sad_x4
    c.cmode = CM_NONE; c.csatd = 0; c.c_rows = 0;
    if (!chroma) return;
    const int cw = bw / 2, ch = bh / 2;
    if (cw < 4 || ch < 4) return;
    const uint64_t cpx = (uint64_t)(int64_t)px / 2, cpy = (uint64_t)(int64_t)py / 2;
    const int clw = G.clw, clh = G.clh;
    int csub = 0, mcx, mcy;
    if (l0sub) { csub = (mvy & 1) * pel + (mvx & 1); mcx = mvx >> 2; mcy = mvy >> 2; }
    else { mcx = mvx >> 1; mcy = mvy >> 1; }
    const uint64_t c_cur = (uint64_t)c_off, c_ref = (uint64_t)(c_off + ((level == 0 && pel > 1) ? (int64_t)csub * clh : 0));
    const uint64_t cs = (uint64_t)G.cs;
    c.c_srow = (int32_t)c_cur; c.c_rrow = (int32_t)c_ref;
    if (cw == 4 || cw == 8 || cw == 16) {
        const int rx0 = (int)(uint32_t)cpx + mcx, ry0 = (int)(uint32_t)cpy + mcy;
        if (cpx + cw <= (uint64_t)clw && cpy + ch <= (uint64_t)clh && rx0 >= 0 && ry0 >= 0 && rx0 + cw <= clw &&
            ry0 + ch <= clh) {
            const uint64_t su = (c_cur + cpy) * cs + cpx, ru = (c_ref + (uint64_t)ry0) * cs + (uint64_t)rx0;
            if (su + (uint64_t)(ch - 1) * cs + cw <= (uint64_t)G.clen && ru + (uint64_t)(ch - 1) * cs + cw <= (uint64_t)G.clen) {
                c.cmode = CM_DIRECT;
                c.csatd = satd ? 1 : 0;
                c.c_rows = satd ? cw : ch;  // satd_interior(.., cw) reads a cw x cw square
                c.c_sbase = (int64_t)su;
                c.c_rbase = (int64_t)ru;
                return;
            }
        }
    }
    c.cmode = CM_SAD_BREAK;
    c.csatd = 0;
    c.c_rows = ch;
    c.c_sx = cpx > 0x7FFFFFFFull ? 0x7FFFFFFF : (int)cpx;
    c.c_sy = cpy > 0x7FFFFFFFull ? 0x7FFFFFFF : (int)cpy;
    c.c_rx = (int)(uint32_t)cpx + mcx;
    c.c_ry = (int)(uint32_t)cpy + mcy;
}

// One 4x4 luma tile of a candidate: its SATD, or its SAD over the part inside the block,
// or (LM_DC) the sum of its source pixels.
__device__ unsigned luma_tile(const Cand &c, const Planes &S, const Planes &R, const Geo &G, int bw, int bh, int tile) {
    const int txn = (bw + 3) >> 2;
    const int ty = tile / txn, tx = tile - ty * txn;
    const int r0 = ty * 4, c0 = tx * 4;
    const int hh = imin(4, bh - r0), ww = imin(4, bw - c0);
    const int64_t ys = G.ys, ylen = G.ylen;
    const int lw = G.lw, lh = G.lh;
    int d[16];
#pragma unroll
    for (int i = 0; i < 16; i++) d[i] = 0;
    unsigned dcsum = 0;
    switch (c.lmode) {
    case LM_DIRECT:
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (r < hh && q < ww)
                    d[r * 4 + q] = (int)rd(S.y, ylen, c.l_sbase + (int64_t)(r0 + r) * ys + c0 + q, 0) -
                                   (int)rd(R.y, ylen, c.l_rbase + (int64_t)(r0 + r) * ys + c0 + q, 0);
        break;
    case LM_SATD_MASK:
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int sy = c.l_sy + r0 + r;
            const int ry = iclamp(c.l_ry + r0 + r, 0, lh - 1);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int sx = c.l_sx + c0 + q;
                const int rx = iclamp(c.l_rx + c0 + q, 0, lw - 1);
                int a = (sy >= 0 && sy < lh && sx >= 0 && sx < lw) ? (int)rd(S.y, ylen, ((int64_t)c.l_srow + sy) * ys + sx, 0) : 0;
                int b = (int)rd(R.y, ylen, ((int64_t)c.l_rrow + ry) * ys + rx, 0);
                d[r * 4 + q] = a - b;
            }
        }
        break;
    case LM_SAD_BREAK:
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int sy = c.l_sy + r0 + r;
            const int ry = iclamp(c.l_ry + r0 + r, 0, lh - 1);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int sx = c.l_sx + c0 + q;
                if (r < hh && q < ww && c.l_sy >= 0 && sy < lh && c.l_sx >= 0 && sx < lw) {
                    const int rx = iclamp(c.l_rx + c0 + q, 0, lw - 1);
                    d[r * 4 + q] = (int)rd(S.y, ylen, ((int64_t)c.l_srow + sy) * ys + sx, 0) -
                                   (int)rd(R.y, ylen, ((int64_t)c.l_rrow + ry) * ys + rx, 0);
                }
            }
        }
        break;
    case LM_EDGE: {
        const int mh = imax(lh - 1, 0), mw = imax(lw - 1, 0);
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int sy = iclamp(c.l_sy + r0 + r, 0, mh), ry = iclamp(c.l_ry + r0 + r, 0, mh);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (r < hh && q < ww) {
                    const int sx = iclamp(c.l_sx + c0 + q, 0, mw), rx = iclamp(c.l_rx + c0 + q, 0, mw);
                    d[r * 4 + q] = (int)rd(S.y, ylen, ((int64_t)c.l_srow + sy) * ys + sx, 0) -
                                   (int)rd(R.y, ylen, ((int64_t)c.l_rrow + ry) * ys + rx, 0);
                }
            }
        }
        break;
    }
    case LM_DC:
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int sy = c.l_sy + r0 + r, sx = c.l_sx + c0 + q;
                if (r < hh && q < ww && c.l_sy >= 0 && sy < lh && c.l_sx >= 0 && sx < lw)
                    dcsum += rd(S.y, ylen, ((int64_t)c.l_srow + sy) * ys + sx, 0);
            }
        return dcsum;
    default: return 0;
    }
    if (c.lsatd) return hadamard4(d);
    unsigned s = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) s += (unsigned)abs(d[i]);
    return s;
}

// One 4x4 tile of one chroma plane of a candidate on the general path.
__device__ unsigned chroma_tile1(const Cand &c, const px_t *sp, const px_t *rp, const Geo &G, int cw, int tile) {
    if (c.cmode == CM_NONE) return 0;
    const int txn = (cw + 3) >> 2;
    const int ty = tile / txn, tx = tile - ty * txn;
    const int r0 = ty * 4, c0 = tx * 4;
    if (r0 >= c.c_rows || c0 >= cw) return 0;
    const int hh = imin(4, c.c_rows - r0), ww = imin(4, cw - c0);
    const int64_t cs = G.cs, clen = G.clen;
    const int clw = G.clw, clh = G.clh;
    int d[16];
#pragma unroll
    for (int i = 0; i < 16; i++) d[i] = 0;
    if (c.cmode == CM_DIRECT) {
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (r < hh && q < ww)
                    d[r * 4 + q] = (int)rd(sp, clen, c.c_sbase + (int64_t)(r0 + r) * cs + c0 + q, 0) -
                                   (int)rd(rp, clen, c.c_rbase + (int64_t)(r0 + r) * cs + c0 + q, 0);
    } else if (c.cmode == CM_SAD_BREAK) {
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const long long sy = (long long)c.c_sy + r0 + r;
            const int ry = iclamp(c.c_ry + r0 + r, 0, clh - 1);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const long long sx = (long long)c.c_sx + c0 + q;
                if (r < hh && q < ww && sy < clh && sx < clw) {
                    const int rx = iclamp(c.c_rx + c0 + q, 0, clw - 1);
                    d[r * 4 + q] = (int)rd(sp, clen, ((int64_t)c.c_srow + sy) * cs + sx, PX_MID) -
                                   (int)rd(rp, clen, ((int64_t)c.c_rrow + ry) * cs + rx, PX_MID);
                }
            }
        }
    } else {  // CM_EDGE
        const int mh = imax(clh - 1, 0), mw = imax(clw - 1, 0);
        const unsigned dflt = c.csatd ? 0u : PX_MID;
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int sy = iclamp(c.c_sy + r0 + r, 0, mh), ry = iclamp(c.c_ry + r0 + r, 0, mh);
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (r < hh && q < ww) {
                    const int sx = iclamp(c.c_sx + c0 + q, 0, mw), rx = iclamp(c.c_rx + c0 + q, 0, mw);
                    d[r * 4 + q] = (int)rd(sp, clen, ((int64_t)c.c_srow + sy) * cs + sx, dflt) -
                                   (int)rd(rp, clen, ((int64_t)c.c_rrow + ry) * cs + rx, dflt);
                }
        }
    }
    if (c.csatd) return hadamard4(d);
    unsigned s = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) s += (unsigned)abs(d[i]);
    return s;
}

// -------------------------------------------------------------------------------------------
// Fast path: candidates whose source and reference blocks lie inside their planes.
//
// One warp evaluates one candidate at a time. Its 4x4 tiles (luma, then U, then V) are taken in
// groups of eight: lane 4 n + r loads the four samples of row r of the group's tile n as 32-bit
// words from 4-byte aligned addresses, funnel-shifted (the caller guarantees 8 readable samples
// after the first sample of every row, see fast_setup), so a load touches the eight rows of a
// group once instead of one row of each of up to 32 candidates.
//
// SATD of a group is one tensor-core instruction: the 4x4 Hadamard transform of a tile is the
// 16x16 Sylvester matrix times its 16 samples, so mma.m16n8k16 gives H ref for eight tiles, with
// -H src (made once per block, stage_source) as its accumulator, and the warp sums the absolute
// values of the 128 results. Exact: a sample s goes in as the half 1024 + s (one byte permute; the
// bias is the same in src and ref and cancels), H holds +-1, products and sums are integers below
// 2^15 and accumulate in f32. The coefficients' order and signs do not matter to the sum. SAD of a
// group is a packed byte difference per lane.
//
// What it measured: see eval_cands.
constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr float kIntBias = 8388608.f;  // 2^23: the low bits of such a float are the integer added to it

struct Smp {  // four samples: 8-bit, the word in a; 16-bit, two halfword pairs
    uint32_t a, b;
};
// A frame as the fast path reads it: its first sample's address rounded down to a word, and the bytes
// that took off. Offsets are bytes from there, below 2^32 (planes are below 2^30 samples).
struct Frame {
    const char *p;
    unsigned mis;
};
__device__ __forceinline__ Frame frame_of(const px_t *p) {
    const uintptr_t a = (uintptr_t)p;
    return Frame{(const char *)(a & ~(uintptr_t)3), (unsigned)(a & 3)};
}
__device__ __forceinline__ const uint32_t *word_at(const Frame &f, unsigned o) {
    return reinterpret_cast<const uint32_t *>(f.p + (size_t)(o & ~3u));
}
#ifndef SVPF_PX16
__device__ __forceinline__ Smp ld4(const Frame &f, unsigned o) {
    const uint32_t *q = word_at(f, o);
    return Smp{__funnelshift_r(__ldg(q), __ldg(q + 1), o * 8u), 0u};  // the shift counts modulo 32
}
// the samples as biased halves (samples 0,1 and 2,3)
__device__ __forceinline__ void halves(const Smp &w, uint32_t &lo, uint32_t &hi) {
    lo = __byte_perm(w.a, 0x64646464u, 0x4140);
    hi = __byte_perm(w.a, 0x64646464u, 0x4342);
}
// acc + |s - r| summed where m is all ones (0: acc)
__device__ __forceinline__ unsigned sad4(const Smp &s, const Smp &r, unsigned m, unsigned acc) {
    return __dp4a(__vabsdiffu4(s.a, r.a), m & 0x01010101u, acc);
}
__device__ __forceinline__ unsigned sum4(const Smp &s) { return __dp4a(s.a, 0x01010101u, 0u); }
constexpr unsigned kHighBits = 0u;
#else
// four 16-bit samples (2-byte aligned): three aligned words funnel-shifted into two pairs
__device__ __forceinline__ Smp ld4(const Frame &f, unsigned o) {
    const uint32_t *q = word_at(f, o);
    const uint32_t w0 = __ldg(q), w1 = __ldg(q + 1), w2 = __ldg(q + 2);
    return Smp{__funnelshift_r(w0, w1, o * 8u), __funnelshift_r(w1, w2, o * 8u)};
}
// Samples 0..1023 fit the mantissa of 1024 + s too. Larger ones are outside the extension's range but not refused: the
// callers gather the bits of what they turn into halves, and take the general path, which is right for every
// uint16, where any of kHighBits is set.
constexpr unsigned kHighBits = 0xFC00FC00u;
__device__ __forceinline__ void halves(const Smp &w, uint32_t &lo, uint32_t &hi) {
    lo = w.a | 0x64006400u;
    hi = w.b | 0x64006400u;
}
__device__ __forceinline__ unsigned sad4(const Smp &s, const Smp &r, unsigned m, unsigned acc) {
    return acc + ((__vsadu2(s.a, r.a) + __vsadu2(s.b, r.b)) & m);
}
__device__ __forceinline__ unsigned sum4(const Smp &s) { return (s.a & 0xFFFFu) + (s.a >> 16) + (s.b & 0xFFFFu) + (s.b >> 16); }
#endif

// This lane's part of the Sylvester matrix as the A operand of mma.m16n8k16: row m is coefficient
// (m / 4, m % 4), column k < 8 is sample (k / 2, k % 2) of a tile and k >= 8 sample ((k - 8) / 2,
// 2 + k % 2), the order in which a lane's two B registers hold its row.
__device__ __forceinline__ uint32_t hadamard_pair(int m, int k) {  // columns k, k + 1 (k even)
    const int r = (k & 7) >> 1, q = k >= 8 ? 2 : 0, mr = m >> 2, mq = m & 3;
    const int s0 = __popc(mr & r) + __popc(mq & q), s1 = __popc(mr & r) + __popc(mq & (q + 1));
    return ((s0 & 1) ? 0xBC00u : 0x3C00u) | (((s1 & 1) ? 0xBC00u : 0x3C00u) << 16);
}
__device__ __forceinline__ float4 mma_hadamard(const uint4 &h, uint32_t lo, uint32_t hi, const float4 &c) {
    float4 d;
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=f"(d.x), "=f"(d.y), "=f"(d.z), "=f"(d.w)
        : "r"(h.x), "r"(h.y), "r"(h.z), "r"(h.w), "r"(lo), "r"(hi), "f"(c.x), "f"(c.y), "f"(c.z), "f"(c.w));
    return d;
}

// -------------------------------------------------------------------------------------------
struct Ctx {
    const AnalyseParams *P;
    const LevelInfo *L;
    Geo G;
    Planes S, R;
    int level, d, tid, satd, pel;
    int nw, wbase;   // warps of the group searching the block, and its first warp in the direction;
                     // tid is the thread's index in that group
    int pnew;        // new-candidate penalty of the current search (opts.pnew; pnew / factor in the refine pass)
    // the fast path's groups of eight tiles (set_groups): per-lane masks, one bit per group
    int ng;          // groups
    unsigned lmask, cmask;  // the lane's tile is a luma one, a chroma one (neither: the place is empty)
    unsigned dlmask, dcmask;  // the same of the tile pair whose SATD sums the lane holds
    unsigned smask;  // the group is searched with SATD (the same in every lane)
    unsigned lshift; // halvings of the luma sum
    Frame fs, fr;
    uint4 h;         // hadamard_pair's registers
    unsigned *off;   // [ng][32] shared: byte offset of the lane's row from the candidate's luma / U block
    float4 *src;     // [ng][32] shared: the block's staged source (-H src, or the samples)
};

// Barrier of the group searching a block: the direction's named barrier, or the warp.
__device__ __forceinline__ void gsync(const Ctx &x) {
    if (x.nw == 1) __syncwarp();
    else dbar(x.d);
}

// Whether chroma takes part in a level's costs.
__device__ __forceinline__ bool has_chroma(const LevelInfo &L) { return !L.smallest && (L.bw >> 1) >= 4 && (L.bh >> 1) >= 4; }

// The groups of eight 4x4 tiles of a candidate of x.L. Luma and chroma share groups when both are
// searched the same way; square blocks searched with SATD are, others (luma SAD, chroma SATD) start
// chroma at a group of its own. x.off is written by every warp with the same values.
__device__ __forceinline__ void set_groups(Ctx &x) {
    const LevelInfo &L = *x.L;
    const int lane = x.tid & 31;
    const int bw = L.bw, bh = L.bh, cw = bw >> 1, ch = bh >> 1;
    const bool lsatd = x.satd && is_blk(bw) && is_blk(bh) && bw == bh, chroma = has_chroma(L);
    const int tx = imax(bw >> 2, 1), tl = tx * imax(bh >> 2, 1), lgtx = 31 - __clz(tx);
    const int crows = x.satd ? cw : ch, ctx = imax(cw >> 2, 1), lgctx = 31 - __clz(ctx), tc = chroma ? ctx * (crows >> 2) : 0;
    const int c0 = lsatd == (x.satd != 0) && tl > 1 ? tl : (tl + 7) & ~7;  // chroma's first tile place
    x.ng = chroma ? (c0 + 2 * tc + 7) >> 3 : (tl + 7) >> 3;
    x.lmask = x.cmask = x.dlmask = x.dcmask = x.smask = 0;
    // a single tile (4x4 blocks) fills both places of its pair and counts twice
    const int tl2 = tl == 1 && lsatd ? 2 : tl;
    x.lshift = (lsatd ? 1 : 0) + (tl2 - tl);
    const int row = lane & 3;
    for (int g = 0; g < x.ng; g++) {
        const int t = g * 8 + (lane >> 2), dt = g * 8 + (lane & 3) * 2;
        unsigned o = 0;  // an empty place reads the block's first row
        if (t < tl2) {
            x.lmask |= 1u << g;
            if (t < tl) o = (unsigned)(((t >> lgtx) * 4 + row) * x.G.ys32 + (t & (tx - 1)) * 4);
            else o = (unsigned)(row * x.G.ys32);
        } else if (t >= c0 && t < c0 + 2 * tc) {
            const int pl = t - c0 >= tc, ct = t - c0 - pl * tc;
            x.cmask |= 1u << g;
            o = (unsigned)(pl ? (unsigned)x.G.clen : 0u) + (unsigned)(((ct >> lgctx) * 4 + row) * x.G.cs32 + (ct & (ctx - 1)) * 4);
        }
        x.off[g * 32 + lane] = o * (unsigned)sizeof(px_t);
        if (dt < tl2) x.dlmask |= 1u << g;
        else if (dt >= c0 && dt < c0 + 2 * tc) x.dcmask |= 1u << g;
        if (g * 8 < c0 ? lsatd : x.satd != 0) x.smask |= 1u << g;
    }
    const int m = lane >> 2, k = (lane & 3) * 2;
    x.h = make_uint4(hadamard_pair(m, k), hadamard_pair(m + 8, k), hadamard_pair(m, k + 8), hadamard_pair(m + 8, k + 8));
    __syncwarp();
}

// The staging area of a warp (see kGroupBytes): x.src that of the group's first warp, x.off its own.
__device__ __forceinline__ void set_stage(Ctx &x, unsigned char *area, int groups, int first, int warp) {
    x.src = reinterpret_cast<float4 *>(area + (size_t)first * groups * kGroupBytes);
    x.off = reinterpret_cast<unsigned *>(area + (size_t)warp * groups * kGroupBytes + (size_t)groups * 512);
}

// Every lane has done with the block before; on return all may read this one's.
__device__ __forceinline__ void make_blk(const Ctx &x, int px, int py, bool chroma, BlkC &out) {
    BlkC b;
    const LevelInfo &L = *x.L;
    const Geo &G = x.G;
    const int bw = L.bw, bh = L.bh, pel = imax(x.pel, 1);
    b.px = px; b.py = py; b.bw = bw; b.bh = bh;
    b.px2 = px - (x.level > 0 && px + bw >= G.lw);
    b.py2 = py - (x.level > 0 && py + bh >= G.lh);
    b.bnd0 = -pel * px; b.bnd1 = -pel * py;
    b.bnd2 = pel * (G.lw - px - bw) + 1; b.bnd3 = pel * (G.lh - py - bh) + 1;
    // bounds above which the edge shift starts
    const int ubx = b.bnd2 > b.bnd0 ? b.bnd2 : 0x7FFFFFFF, uby = b.bnd3 > b.bnd1 ? b.bnd3 : 0x7FFFFFFF;
    b.chroma = chroma;
    const bool fastable = bw > 0 && bh > 0 && (bw & 3) == 0 && (bh & 3) == 0;
    b.lsrc = ((int64_t)L.y_off + b.py2) * G.ys + b.px2;
    b.fast_src = fastable && b.px2 >= 0 && b.py2 >= 0 && b.px2 + bw <= G.lw && b.py2 + bh <= G.lh &&
                 b.lsrc + (int64_t)(bh - 1) * G.ys + bw + 8 <= G.ylen;
    const int cw = bw / 2, ch = bh / 2, crows = x.satd ? cw : ch, cpx = px / 2, cpy = py / 2;
    const int64_t csrc = ((int64_t)L.c_off + cpy) * G.cs + cpx;
    b.csrc = G.ylen + csrc;
    // the fast-path box: no edge shift, reference block inside the level (luma, and chroma when
    // it is evaluated); with l0sub the luma offset is mv >> 1 and the chroma one mv >> 2
    const bool l0sub = x.level == 0 && pel >= 2;
    const int ls = l0sub ? 1 : 0, cshift = l0sub ? 2 : 1;
    b.fx0 = imax(b.bnd0, (-b.px2) * (1 << ls));
    b.fx1 = imin(ubx - 1, (G.lw - bw - b.px2) * (1 << ls) + (1 << ls) - 1);
    b.fy0 = imax(b.bnd1, (-b.py2) * (1 << ls));
    b.fy1 = imin(uby - 1, (G.lh - bh - b.py2) * (1 << ls) + (1 << ls) - 1);
    if (chroma && cw >= 4 && ch >= 4) {
        const bool cfast_src = (cw == 4 || cw == 8 || cw == 16) && (ch & 3) == 0 && px >= 0 && py >= 0 &&
                               cpx + cw <= G.clw && cpy + ch <= G.clh &&
                               csrc + (int64_t)(crows - 1) * G.cs + cw + 8 <= G.clen;
        b.fx0 = imax(b.fx0, (-cpx) * (1 << cshift));
        b.fx1 = imin(b.fx1, (G.clw - cw - cpx) * (1 << cshift) + (1 << cshift) - 1);
        b.fy0 = imax(b.fy0, (-cpy) * (1 << cshift));
        b.fy1 = imin(b.fy1, (G.clh - ch - cpy) * (1 << cshift) + (1 << cshift) - 1);
        if (!cfast_src) b.fast_src = 0;
    }
    if (!b.fast_src) b.fx1 = b.fx0 - 1;  // empty box
    b.lbase = ((int)L.y_off + b.py2) * G.ys32 + b.px2;
    b.llim = (int)G.ylen - (bh - 1) * G.ys32 - bw - 8;
    b.cbase = (int)G.ylen + ((int)L.c_off + cpy) * G.cs32 + cpx;
    b.clim = (int)(G.ylen + G.clen) - (crows - 1) * G.cs32 - cw - 8;
    out = b;
    __syncwarp();
}

// Does (block, mv) take the fast path? If so, the byte offsets of its reference blocks (see Frame).
// It does when the reference takes its direct reads for both luma and chroma: no edge
// shift, the luma block and the reference block inside the level, the chroma blocks too.
__device__ __forceinline__ bool fast_setup(const Ctx &x, const BlkC &b, int mvx, int mvy, unsigned &lref, unsigned &cref) {
    if (mvx < b.fx0 || mvx > b.fx1 || mvy < b.fy0 || mvy > b.fy1) return false;
    const int pel = imax(x.pel, 1);
    const bool l0sub = x.level == 0 && pel >= 2;
    const int sub = l0sub ? (mvy & 1) * pel + (mvx & 1) : 0;
    const int mx = l0sub ? mvx >> 1 : mvx, my = l0sub ? mvy >> 1 : mvy;
    const int lr = b.lbase + (sub * x.G.lh + my) * x.G.ys32 + mx;
    if (lr > b.llim) return false;
    lref = (unsigned)lr * (unsigned)sizeof(px_t) + x.fr.mis;
    cref = 0;
    if (b.chroma && b.bw >= 8 && b.bh >= 8) {
        const int mcx = l0sub ? mvx >> 2 : mvx >> 1, mcy = l0sub ? mvy >> 2 : mvy >> 1;
        const int cr = b.cbase + ((l0sub ? sub * x.G.clh : 0) + mcy) * x.G.cs32 + mcx;
        if (cr > b.clim) return false;
        cref = (unsigned)cr * (unsigned)sizeof(px_t) + x.fr.mis;
    }
    return true;
}

__device__ __forceinline__ void set_geo(Geo &G, const AnalyseParams &P, const LevelInfo &L) {
    G.lw = L.lw; G.lh = L.lh; G.clw = L.lw / 2; G.clh = L.lh / 2;
    G.ys = P.y_stride; G.cs = P.c_stride; G.ylen = P.y_len; G.clen = P.c_len;
    G.ys32 = (int)P.y_stride; G.cs32 = (int)P.c_stride;
}
__device__ __forceinline__ Planes planes_of(const px_t *frame, const AnalyseParams &P) {
    return Planes{frame, frame + P.y_len, frame + P.y_len + P.c_len};
}

__device__ __forceinline__ void set_frames(Ctx &x, const AnalyseParams &P, const px_t *src, const px_t *ref) {
    x.S = planes_of(src, P);
    x.R = planes_of(ref, P);
    x.fs = frame_of(src);
    x.fr = frame_of(ref);
}

// One candidate on the general path, the reference's own read path through cand_setup, by the whole
// warp: exact_sad's luma (x) and chroma (y) parts. SLOW_DC: the sum of the block's luma samples
// (block_luma_dc). Out of line, with few arguments, so that the callers keep their registers.
enum { SLOW_CHROMA = 1, SLOW_DC = 2, SLOW_STAGED = 4 };
__device__ __noinline__ uint2 slow_warp(const AnalyseParams *Pp, const LevelInfo *Lp, const px_t *src, const px_t *ref,
                                        int level, int px, int py, int mvx, int mvy, int what) {
    const AnalyseParams &P = *Pp;
    const LevelInfo &L = *Lp;
    Geo G;
    set_geo(G, P, L);
    const Planes S = planes_of(src, P), R = planes_of(ref, P);
    const bool chroma = (what & SLOW_CHROMA) != 0;
    Cand c;
    cand_setup(c, P, L, G, level, px, py, L.bw, L.bh, mvx, mvy, chroma, L.satd, L.pel, (what & SLOW_DC) != 0);
    unsigned rl = 0, ru = 0, rv = 0;
    const int T = L.tl + (chroma ? 2 * L.tc : 0);
    for (int t = (int)(threadIdx.x & 31); t < T; t += 32) {
        if (t < L.tl) rl += luma_tile(c, S, R, G, L.bw, L.bh, t);
        else if (c.cmode != CM_NONE) {
            int ct = t - L.tl;
            const int pl = ct >= L.tc;
            ct -= pl * L.tc;
            const unsigned v = chroma_tile1(c, pl ? S.v : S.u, pl ? R.v : R.u, G, L.bw / 2, ct);
            if (pl) rv += v; else ru += v;
        }
    }
    rl = __reduce_add_sync(kFull, rl);
    ru = __reduce_add_sync(kFull, ru);
    rv = __reduce_add_sync(kFull, rv);
    unsigned C = 0;
    if (c.cmode != CM_NONE && chroma) C = c.csatd ? sat_mul(sat_add(ru >> 1, rv >> 1), 4) : sat_mul(ru + rv, 4);
    return make_uint2(c.lsatd ? (rl >> 1) : rl, C);
}
__device__ __forceinline__ uint2 eval_slow(const Ctx &x, int px, int py, int mvx, int mvy, int what) {
    return slow_warp(x.P, x.L, x.S.y, x.R.y, x.level, px, py, mvx, mvy, what);
}
__device__ __forceinline__ unsigned sad_of(uint2 lc) { return sat_add(lc.x, lc.y); }

// U groups of NB candidates: every load is in flight before the first is used, and a group's staged
// source, offset and masks are read once for all of them.
template <int U, int NB, bool SATD>
__device__ __forceinline__ void eval_groups(const Ctx &x, int g0, const unsigned (&lr)[NB], const unsigned (&cr)[NB],
                                            float (&fl)[NB], float (&fc)[NB], unsigned (&il)[NB], unsigned (&ic)[NB],
                                            unsigned &high) {
    const int lane = x.tid & 31;
    Smp w[U][NB];
    float4 c[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int g = g0 + u;
        const unsigned o = x.off[g * 32 + lane];
        const bool chroma = (x.cmask >> g) & 1u;
        c[u] = x.src[g * 32 + lane];
#pragma unroll
        for (int q = 0; q < NB; q++) w[u][q] = ld4(x.fr, (chroma ? cr[q] : lr[q]) + o);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int g = g0 + u;
        if (SATD) {
            const float wl = (x.dlmask >> g) & 1u ? 1.f : 0.f, wc = (x.dcmask >> g) & 1u ? 1.f : 0.f;
#pragma unroll
            for (int q = 0; q < NB; q++) {
                uint32_t lo, hi;
                halves(w[u][q], lo, hi);
                if (kHighBits) high |= w[u][q].a | w[u][q].b;
                const float4 d = mma_hadamard(x.h, lo, hi, c[u]);
                const float v = (fabsf(d.x) + fabsf(d.y)) + (fabsf(d.z) + fabsf(d.w));
                fl[q] = fmaf(v, wl, fl[q]);
                fc[q] = fmaf(v, wc, fc[q]);
            }
        } else {
            const unsigned ml = 0u - ((x.lmask >> g) & 1u), mc = 0u - ((x.cmask >> g) & 1u);
            const Smp sm{__float_as_uint(c[u].x), __float_as_uint(c[u].y)};
#pragma unroll
            for (int q = 0; q < NB; q++) {
                il[q] = sad4(sm, w[u][q], ml, il[q]);
                ic[q] = sad4(sm, w[u][q], mc, ic[q]);
            }
        }
    }
}

// NB candidates on the fast path by the whole warp. lref, cref: the lanes' set-ups; m: the lanes
// still to take, of which the lowest NB go (fewer left: the last one again, unused). Three groups,
// all SATD (16x16 blocks with chroma, TRI): in one go; else group by group. A 4x4 tile's SATD is even
// (its coefficients share their parity), so halving the sum of tiles is halving each plane's. `high` gathers the bits of
// the samples turned into halves.
template <int NB, bool TRI>
__device__ __forceinline__ void eval_fast(const Ctx &x, unsigned lref, unsigned cref, unsigned &m, unsigned &L, unsigned &C,
                                          unsigned &high) {
    const int lane = x.tid & 31;
    unsigned lr[NB], cr[NB], il[NB], ic[NB];
    float fl[NB], fc[NB];
    int who[NB];
#pragma unroll
    for (int q = 0; q < NB; q++) {
        who[q] = m ? __ffs(m) - 1 : who[q > 0 ? q - 1 : 0];
        m &= m - 1;
        lr[q] = __shfl_sync(kFull, lref, who[q]);
        cr[q] = __shfl_sync(kFull, cref, who[q]);
        fl[q] = fc[q] = kIntBias;
        il[q] = ic[q] = 0;
    }
    if (TRI) {
        eval_groups<3, NB, true>(x, 0, lr, cr, fl, fc, il, ic, high);
    } else {
#pragma unroll 1
        for (int g = 0; g < x.ng; g++) {
            if ((x.smask >> g) & 1u) eval_groups<1, NB, true>(x, g, lr, cr, fl, fc, il, ic, high);
            else eval_groups<1, NB, false>(x, g, lr, cr, fl, fc, il, ic, high);
        }
    }
#pragma unroll
    for (int q = 0; q < NB; q++) {
        const unsigned sl = __reduce_add_sync(kFull, il[q] + (__float_as_uint(fl[q]) - __float_as_uint(kIntBias)));
        const unsigned sc = __reduce_add_sync(kFull, ic[q] + (__float_as_uint(fc[q]) - __float_as_uint(kIntBias)));
        if (lane == who[q]) {
            L = sl >> x.lshift;
            C = x.satd ? (sc >> 1) * 4u : sc * 4u;
        }
    }
}

// The block's source for the fast path (Ctx::src) and the sum of its luma samples, each warp of
// the group taking every nw-th group of tiles: the sum is the warp's part. A block whose source holds samples too
// large for it leaves the fast path (every warp looks at all of it).
__device__ __forceinline__ unsigned stage_source(const Ctx &x, BlkC &b) {
    unsigned s = 0, high = 0;
    const int lane = x.tid & 31;
    const unsigned lo_ = (unsigned)b.lsrc * (unsigned)sizeof(px_t) + x.fs.mis, co = (unsigned)b.csrc * (unsigned)sizeof(px_t) + x.fs.mis;
#pragma unroll 1
    for (int g = kHighBits ? 0 : x.tid >> 5; g < x.ng; g += kHighBits ? 1 : x.nw) {
        const bool chroma = (x.cmask >> g) & 1u;
        const Smp w = ld4(x.fs, (chroma ? co : lo_) + x.off[g * 32 + lane]);
        if (kHighBits && ((x.smask >> g) & 1u)) high |= w.a | w.b;
        if (kHighBits && x.nw > 1 && g % x.nw != (x.tid >> 5)) continue;
        if (((x.lmask >> g) & 1u) && !(x.lshift == 2 && lane >= 4)) s += sum4(w);
        float4 c = make_float4(__uint_as_float(w.a), __uint_as_float(w.b), 0.f, 0.f);
        if ((x.smask >> g) & 1u) {
            uint32_t lo, hi;
            halves(w, lo, hi);
            c = mma_hadamard(x.h, lo, hi, make_float4(0.f, 0.f, 0.f, 0.f));
            c = make_float4(-c.x, -c.y, -c.z, -c.w);
        }
        x.src[g * 32 + lane] = c;
    }
    if (kHighBits && __any_sync(kFull, (high & kHighBits) != 0)) {
        __syncwarp();
        b.fast_src = 0;
        b.fx1 = b.fx0 - 1;  // an empty box
        __syncwarp();
    }
    return __reduce_add_sync(kFull, s);
}

// Four samples whose first would be at x of a row of n >= 4 samples, places outside the row taking
// the row's end sample (w: the samples loaded at x clamped to 0 .. n - 4): e = x - that place.
__device__ __forceinline__ Smp spread_ends(const Smp &w, int e) {
    e = iclamp(e, -3, 3);
    const unsigned sel = __funnelshift_r(0x33210000u, 0x33u, (unsigned)(12 + 4 * e)) & 0xFFFFu;  // sample i + e, clamped
#ifndef SVPF_PX16
    return Smp{__byte_perm(w.a, 0u, sel), 0u};
#else
    const unsigned j0 = sel & 3u, j1 = (sel >> 4) & 3u, j2 = (sel >> 8) & 3u, j3 = (sel >> 12) & 3u;
    const unsigned s01 = (j0 * 0x22u + 0x10u) | (j1 * 0x2200u + 0x1000u), s23 = (j2 * 0x22u + 0x10u) | (j3 * 0x2200u + 0x1000u);
    return Smp{__byte_perm(w.a, w.b, s01), __byte_perm(w.a, w.b, s23)};
#endif
}

// The candidates that do not take the fast path, lanes `mask`, for a block at (px, py). Most of them
// (a quarter-pel field, whose vectors the reference reads as half-pel ones, has them everywhere) lie
// inside mv_bounds with the block's source inside its planes and only the reference block reaching
// out: then every read is the staged source against samples clamped to the plane (:1719-1852,
// :2353-2436), and chroma is compared by SATD where its block lies inside and by SAD where it does
// not (:2169-2303). They go through the groups of eight tiles as on the fast path, NB at a time; the
// others one by one through slow_warp. Out of line: called once for all of a step's such candidates.
__device__ __noinline__ uint2 clamped_cands(const AnalyseParams *Pp, const LevelInfo *Lp, const px_t *src, const px_t *ref,
                                            const float4 *stage, int level, int px, int py, unsigned mask, int mvx, int mvy,
                                            int what) {
    constexpr int NB = 4;
    const AnalyseParams &P = *Pp;
    const LevelInfo &L = *Lp;
    Ctx x;  // the fields the group tables need
    x.L = Lp;
    x.satd = L.satd;
    x.tid = (int)(threadIdx.x & 31);
    set_geo(x.G, P, L);
    const int lane = x.tid;
    const Geo &G = x.G;
    const int bw = L.bw, bh = L.bh, cw = bw >> 1, ch = bh >> 1, pel = imax(L.pel, 1);
    const bool chroma = (what & SLOW_CHROMA) != 0 && cw >= 4 && ch >= 4;
    const int px2 = px - (level > 0 && px + bw >= G.lw), py2 = py - (level > 0 && py + bh >= G.lh);
    const int cpx = px / 2, cpy = py / 2;
    const bool l0sub = level == 0 && pel >= 2;
    const Frame fs = frame_of(src), fr = frame_of(ref);
    // this lane's candidate: may it go through the groups?
    const int sub = l0sub ? (mvy & 1) * pel + (mvx & 1) : 0;
    const int lrow0 = (int)L.y_off + sub * G.lh, crow0 = (int)L.c_off + sub * G.clh;
    const int rx = px2 + (l0sub ? mvx >> 1 : mvx), ry = py2 + (l0sub ? mvy >> 1 : mvy);
    const int crx = cpx + (l0sub ? mvx >> 2 : mvx >> 1), cry = cpy + (l0sub ? mvy >> 2 : mvy >> 1);
    const int b0 = -pel * px, b1 = -pel * py, b2 = pel * (G.lw - px - bw) + 1, b3 = pel * (G.lh - py - bh) + 1;
    bool ok = (what & SLOW_STAGED) != 0 && (bw == bh || !L.satd) && mvx >= b0 && mvy >= b1 && !(b2 > b0 && mvx >= b2) &&
              !(b3 > b1 && mvy >= b3);
    ok = ok && (int64_t)(lrow0 + iclamp(ry + bh - 1, 0, G.lh - 1)) * G.ys + iclamp(rx + bw - 4, 0, G.lw - 4) + 8 <= G.ylen;
    if (chroma)
        ok = ok && (int64_t)(crow0 + iclamp(cry + ch - 1, 0, G.clh - 1)) * G.cs + iclamp(crx + cw - 4, 0, G.clw - 4) + 8 <= G.clen;
    const bool cdirect = crx >= 0 && cry >= 0 && crx + cw <= G.clw && cry + ch <= G.clh;
    unsigned mm = __ballot_sync(kFull, ok) & mask, ms = mask & ~mm;
    const unsigned cdm = __ballot_sync(kFull, cdirect);
    uint2 out = make_uint2(0u, 0u);
    if (mm) {
        // the group tables (as set_groups), without offsets
        const bool lsatd = L.satd && bw == bh;  // ok implies the same kind for both
        const int tx = imax(bw >> 2, 1), tl = tx * imax(bh >> 2, 1), lgtx = 31 - __clz(tx);
        const int ctx = imax(cw >> 2, 1), lgctx = 31 - __clz(ctx), tc = chroma ? ctx * (ch >> 2) : 0;
        const int c0 = lsatd == (L.satd != 0) && tl > 1 ? tl : (tl + 7) & ~7;
        const int tl2 = tl == 1 && lsatd ? 2 : tl, ng = chroma ? (c0 + 2 * tc + 7) >> 3 : (tl + 7) >> 3;
        const int lshift = (lsatd ? 1 : 0) + (tl2 - tl);
        const int m = lane >> 2, k = (lane & 3) * 2;
        const uint4 h = make_uint4(hadamard_pair(m, k), hadamard_pair(m + 8, k), hadamard_pair(m, k + 8), hadamard_pair(m + 8, k + 8));
#pragma unroll 1
        while (mm) {
            int who[NB], qx[NB], qy[NB], ql[NB], cx[NB], cy[NB], ql2[NB];
            float fl[NB], fc[NB];
            unsigned il[NB], ic[NB], high = 0;
#pragma unroll
            for (int q = 0; q < NB; q++) {
                who[q] = mm ? __ffs(mm) - 1 : who[q > 0 ? q - 1 : 0];
                mm &= mm - 1;
                qx[q] = __shfl_sync(kFull, rx, who[q]);
                qy[q] = __shfl_sync(kFull, ry, who[q]);
                ql[q] = __shfl_sync(kFull, lrow0, who[q]);
                cx[q] = __shfl_sync(kFull, crx, who[q]);
                cy[q] = __shfl_sync(kFull, cry, who[q]);
                ql2[q] = __shfl_sync(kFull, crow0, who[q]);
                fl[q] = fc[q] = kIntBias;
                il[q] = ic[q] = 0;
            }
#pragma unroll 1
            for (int g = 0; g < ng; g++) {
                const int t = g * 8 + (lane >> 2), dt = g * 8 + (lane & 3) * 2;
                const bool isl = t < tl2, isc = t >= c0 && t < c0 + 2 * tc;
                const int pl = t - c0 >= tc, ct = t - c0 - pl * tc, tt = t < tl ? t : 0;
                const int ox = isc ? (ct & (ctx - 1)) * 4 : (tt & (tx - 1)) * 4;
                const int oy = (isc ? (ct >> lgctx) * 4 : (tt >> lgtx) * 4) + (lane & 3);
                const int w_ = isc ? G.clw : G.lw, h_ = isc ? G.clh : G.lh, st = isc ? G.cs32 : G.ys32;
                const unsigned plane = isc ? (unsigned)G.ylen + (pl ? (unsigned)G.clen : 0u) : 0u;
                const float4 c = stage[g * 32 + lane];
                Smp w[NB];
#pragma unroll
                for (int q = 0; q < NB; q++) {
                    const int xx = (isc ? cx[q] : qx[q]) + ox, yy = iclamp((isc ? cy[q] : qy[q]) + oy, 0, h_ - 1);
                    const int xa = iclamp(xx, 0, w_ - 4);
                    const unsigned o = plane + (unsigned)(((isc ? ql2[q] : ql[q]) + yy) * st + xa);
                    w[q] = spread_ends(ld4(fr, o * (unsigned)sizeof(px_t) + fr.mis), xx - xa);
                }
                const bool satd = g * 8 < c0 ? lsatd : L.satd != 0;
                const unsigned ml = 0u - (unsigned)isl, mc = 0u - (unsigned)isc;
                if (satd) {
                    const float wl = dt < tl2 ? 1.f : 0.f, wc = dt >= c0 && dt < c0 + 2 * tc ? 1.f : 0.f;
                    Smp s0{0u, 0u};
                    if (isc)
                        s0 = ld4(fs, (plane + (unsigned)(((int)L.c_off + cpy + oy) * st + cpx + ox)) * (unsigned)sizeof(px_t) + fs.mis);
#pragma unroll
                    for (int q = 0; q < NB; q++) {
                        uint32_t lo, hi;
                        halves(w[q], lo, hi);
                        if (kHighBits) high |= w[q].a | w[q].b;
                        const float4 d = mma_hadamard(h, lo, hi, c);
                        const float v = (fabsf(d.x) + fabsf(d.y)) + (fabsf(d.z) + fabsf(d.w));
                        fl[q] = fmaf(v, wl, fl[q]);
                        fc[q] = fmaf(v, wc, fc[q]);
                        ic[q] = sad4(s0, w[q], mc, ic[q]);
                    }
                } else {
                    const Smp sm{__float_as_uint(c.x), __float_as_uint(c.y)};
#pragma unroll
                    for (int q = 0; q < NB; q++) {
                        il[q] = sad4(sm, w[q], ml, il[q]);
                        ic[q] = sad4(sm, w[q], mc, ic[q]);
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < NB; q++) {
                const unsigned sl = __reduce_add_sync(kFull, il[q] + (__float_as_uint(fl[q]) - __float_as_uint(kIntBias)));
                const unsigned st_ = __reduce_add_sync(kFull, __float_as_uint(fc[q]) - __float_as_uint(kIntBias));
                const unsigned sa = __reduce_add_sync(kFull, ic[q]);
                if (lane == who[q])
                    out = make_uint2(sl >> lshift, L.satd && ((cdm >> who[q]) & 1u) ? (st_ >> 1) * 4u : sa * 4u);
            }
            if (kHighBits && __any_sync(kFull, (high & kHighBits) != 0)) {
#pragma unroll
                for (int q = 0; q < NB; q++) ms |= 1u << who[q];
            }
        }
    }
#pragma unroll 1
    while (ms) {
        const int j = __ffs(ms) - 1;
        ms &= ms - 1;
        const uint2 r = slow_warp(Pp, Lp, src, ref, level, px, py, __shfl_sync(kFull, mvx, j), __shfl_sync(kFull, mvy, j), what);
        if (lane == j) out = r;
    }
    return out;
}

// Evaluates every lane's candidate (lanes with `ok`): L and C of exact_sad in the lane that holds
// it. The lanes set their candidates up side by side, then the warp evaluates one after another.
// Bound: the latency of the loads, which the candidates evaluated together overlap, then instruction
// issue. Per 16x16 candidate with chroma this is about 120 warp instructions with all that surrounds
// it, against 167 when groups of lanes each transformed whole tiles in f16x2 (14.2 k against 19.2 k
// per level-0 block of the 1080p configuration, its repeats included).
__device__ __forceinline__ void eval_cands(const Ctx &x, const BlkC &b, bool ok, int mvx, int mvy, unsigned &L, unsigned &C) {
    const int lane = x.tid & 31;
    unsigned lref = 0, cref = 0;
    const bool fast = ok && fast_setup(x, b, mvx, mvy, lref, cref);
    unsigned mf = __ballot_sync(kFull, fast), ms = __ballot_sync(kFull, ok && !fast);
    L = C = 0;
    unsigned high = 0;
    const unsigned all = mf;
#pragma unroll 1
    while (mf) {
        if (x.ng == 3 && x.smask == 7u) eval_fast<4, true>(x, lref, cref, mf, L, C, high);
        else if (__popc(mf) > 4) eval_fast<8, false>(x, lref, cref, mf, L, C, high);
        else eval_fast<4, false>(x, lref, cref, mf, L, C, high);
    }
    if (kHighBits && __any_sync(kFull, (high & kHighBits) != 0)) ms |= all;  // samples too large for the fast path
    if (ms) {
        const uint2 r = clamped_cands(x.P, x.L, x.S.y, x.R.y, x.src, x.level, b.px, b.py, ms, mvx, mvy,
                                      (b.chroma ? SLOW_CHROMA : 0) | (b.fast_src ? SLOW_STAGED : 0));
        if ((ms >> lane) & 1u) { L = r.x; C = r.y; }
    }
    if (!b.chroma) C = 0;
}

// The lane holding the least (cost, place) among those with `act`, or -1. Costs of a word or less
// take two redux; the others a shuffle tree.
__device__ __forceinline__ int first_min(bool act, long long cost, int place) {
    if (!__any_sync(kFull, act)) return -1;
    bool e;
    if (!__any_sync(kFull, act && (unsigned long long)cost >= 0xFFFFFFFFull)) {
        const unsigned u = act ? (unsigned)cost : 0xFFFFFFFFu;
        const unsigned least = __reduce_min_sync(kFull, u);
        e = act && u == least;
    } else {
        long long m = act ? cost : 0x7FFFFFFFFFFFFFFFLL;
#pragma unroll 1
        for (int o = 16; o > 0; o >>= 1) {
            const long long v = __shfl_xor_sync(kFull, m, o);
            m = v < m ? v : m;
        }
        e = act && cost == m;
    }
    const int pm = __reduce_min_sync(kFull, e ? place : 0x7FFFFFFF);
    return __ffs(__ballot_sync(kFull, e && place == pm)) - 1;
}

// One search step: candidates g over the block against the running best `best_cost`, 32 at a time,
// one per lane. The group's warps share the candidates that pass exact_ok and the motion-penalty
// cut, every nw-th of them, and combine their winners. A candidate whose motion penalty reaches the
// best cost cannot win (cost >= penalty for pnew >= -256), so the reference's skip and a skip
// against an earlier, larger best decide alike. On return, identically in every thread: win =
// accepted candidate or -1, and the new best cost / sad when accepted.
template <class SH>
__device__ __forceinline__ void eval_step(const Ctx &x, const BlkC &b, SH &s, int &ph, const Gen &g, int lambda,
                                          int predx, int predy, long long &best_cost, unsigned &best_sad, int &win) {
    const int lane = x.tid & 31, warp = x.tid >> 5, wi = x.wbase + warp;  // wi: the warp's place in the direction
    const bool serial = x.pnew < -256;
    const int pnew = x.pnew;
    long long bk = best_cost;  // the warp's own best
    int bi = -1;
    unsigned bs = 0;
    win = -1;
#pragma unroll 1
    for (int base = 0; base < g.n; base += 32) {
        const int i = base + lane;
        bool ok = i < g.n;
        int2 mv = make_int2(0, 0);
        long long motion = 0;
        if (ok) {
            mv = gen_mv(g, i);
            ok = mv.x >= b.bnd0 && mv.y >= b.bnd1 && mv.x < b.bnd2 && mv.y < b.bnd3;  // exact_ok
            motion = motion_penalty(lambda, predx, predy, mv.x, mv.y);
            if (ok) ok = motion < best_cost;  // a later candidate faces a lower best
        }
        bool mine = ok;
        const int rank = __popc(__ballot_sync(kFull, ok) & ((1u << lane) - 1u));
        if (x.nw > 1) mine = ok && rank % x.nw == warp;
        if (!serial) mine = mine && motion < bk;
        unsigned L, C;
        eval_cands(x, b, mine, mv.x, mv.y, L, C);
        const long long K = motion + pen(pnew, L) + (b.chroma ? pen(pnew, C) : 0LL);  // :1158-1221
        const unsigned sad = sat_add(L, C);
        if (serial) {  // exact sequential semantics for penalties that can be negative
            long long kk = K;
            unsigned ss = sad;
            if (x.nw > 1) {  // every warp sees every cost
                if (mine) { s.rk[ph][lane] = K; s.rs[ph][lane] = sad; }
                gsync(x);
                kk = s.rk[ph][lane];
                ss = s.rs[ph][lane];
                ph ^= 1;
            }
            for (unsigned m = __ballot_sync(kFull, ok); m; m &= m - 1) {
                const int j = __ffs(m) - 1;
                const long long mj = __shfl_sync(kFull, motion, j), kj = __shfl_sync(kFull, kk, j);
                const unsigned sj = __shfl_sync(kFull, ss, j);
                if (mj < best_cost && kj < best_cost) { best_cost = kj; best_sad = sj; win = base + j; }
            }
        } else {
            const int j = first_min(mine && K < bk, K, lane);
            if (j >= 0) {
                bk = __shfl_sync(kFull, K, j);
                bs = __shfl_sync(kFull, sad, j);
                bi = base + j;
                if (x.nw == 1) { best_cost = bk; best_sad = bs; win = bi; }
            }
        }
    }
    if (serial || x.nw == 1) return;
    // combine the group's warps
    if (lane == 0) { s.K[ph][wi] = bk; s.I[ph][wi] = bi; s.S[ph][wi] = bs; }
    gsync(x);
    for (int w = x.wbase; w < x.wbase + x.nw; w++) {
        const int ii = s.I[ph][w];
        if (ii < 0) continue;
        const long long k = s.K[ph][w];
        if (k < best_cost || (k == best_cost && win >= 0 && ii < win)) { best_cost = k; best_sad = s.S[ph][w]; win = ii; }
    }
    ph ^= 1;
}

// adapt_lambda, :1555-1564 (f64, IEEE-exact: one add, one division, two products)
__device__ __forceinline__ int adapt_lambda(int nlambda, int lsad, unsigned pred_score) {
    const double l = (double)imax(lsad, 1);
    const double half = pred_score == 0xFFFFFFFFu ? -1.0 : (double)(pred_score >> 1);
    const double t = __ddiv_rn(l, __dadd_rn(l, half));
    double v = __dmul_rn(__dmul_rn((double)nlambda, t), t);
    v = fmin(v, 21474836.47);
    if (v != v) return 0;
    if (v >= 2147483647.0) return 2147483647;
    if (v <= -2147483648.0) return (int)0x80000000;
    return (int)v;
}

// block_activity / plane_activity (:1486-1553): used only when search.coarse.distance < 0.
__device__ __noinline__ unsigned plane_activity(const px_t *data, int64_t len, int64_t stride, int64_t row, int64_t x,
                                                int w, int h, bool satd) {
    const unsigned area = (unsigned)(w * h);
    unsigned sum = 0;
    for (int y = 0; y < h; y++)
        for (int c = 0; c < w; c++) sum += rd(data, len, (row + y) * stride + x + c, 0);
    const unsigned mean = area ? sum / area : 0;
    if (!satd) {
        unsigned s = 0;
        for (int y = 0; y < h; y++)
            for (int c = 0; c < w; c++) {
                unsigned v = rd(data, len, (row + y) * stride + x + c, 0);
                s += v > mean ? v - mean : mean - v;
            }
        return area ? s / area : 0;
    }
    unsigned total = 0;
    for (int y = 0; y < h; y += 4)
        for (int x0 = 0; x0 < w; x0 += 4) {
            int dd[16];
            for (int r = 0; r < 4; r++)
                for (int q = 0; q < 4; q++) dd[r * 4 + q] = (int)rd(data, len, (row + y + r) * stride + x + x0 + q, 0) - (int)mean;
            total += hadamard4(dd);
        }
    return area ? (total >> 1) / area : 0;
}

// The three planes' activity of a block (its luma at (lx, ly), which the level's last column and row shift).
__device__ __noinline__ unsigned block_activity(const AnalyseParams *Pp, const LevelInfo *Lp, const px_t *src, int lx, int ly,
                                                int px, int py) {
    const AnalyseParams &P = *Pp;
    const LevelInfo &L = *Lp;
    const Planes S = planes_of(src, P);
    const bool satd = L.satd != 0;
    return plane_activity(S.y, P.y_len, P.y_stride, L.y_off + ly, lx, L.bw, L.bh, satd) +
           plane_activity(S.u, P.c_len, P.c_stride, L.c_off + py / 2, px / 2, L.bw / 2, L.bh / 2, satd) +
           plane_activity(S.v, P.c_len, P.c_stride, L.c_off + py / 2, px / 2, L.bw / 2, L.bh / 2, satd);
}

__device__ __forceinline__ int adaptive_radius(int radius, unsigned act) {
    if (act < 2) return 0;
    unsigned a = 255u * act / 150u;
    return ((radius * (int)(a < 255 ? a : 255)) >> 8) + 1;
}
// search orders (:302-419)
__device__ __forceinline__ int64_t initial_order_len(int gw, int gh) {
    const int64_t ni = (int64_t)imax(gh - 2, 0) * imax(gw - 2, 0);
    return ni + (int64_t)gw * (gh > 1 ? 2 : 1) + (int64_t)imax(gh - 2, 0) * (gw > 1 ? 2 : 1);
}
__device__ __forceinline__ int2 initial_order_at(int gw, int gh, int64_t k) {
    const int iw = imax(gw - 2, 0);
    const int64_t ni = (int64_t)imax(gh - 2, 0) * iw;
    if (k < ni) {
        const int y = (int)(k / iw) + 1, j = (int)(k % iw);
        return make_int2((y & 1) == 0 ? 1 + j : gw - 2 - j, y);
    }
    k -= ni;
    const int64_t nb = (int64_t)gw * (gh > 1 ? 2 : 1);
    if (k < nb) {
        if (gh > 1) return make_int2((int)(k >> 1), (k & 1) ? gh - 1 : 0);
        return make_int2((int)k, 0);
    }
    k -= nb;
    if (gw > 1) return make_int2((k & 1) ? gw - 1 : 0, 1 + (int)(k >> 1));
    return make_int2(0, 1 + (int)k);
}
__device__ __forceinline__ int64_t initial_order_pos(int gw, int gh, int x, int y) {
    const int iw = imax(gw - 2, 0);
    const int64_t ni = (int64_t)imax(gh - 2, 0) * iw;
    if (y >= 1 && y <= gh - 2 && x >= 1 && x <= gw - 2)
        return (int64_t)(y - 1) * iw + ((y & 1) == 0 ? x - 1 : gw - 2 - x);
    if (y == 0) return ni + (gh > 1 ? 2 * x : x);
    if (y == gh - 1) return ni + 2 * x + 1;
    const int64_t nb = (int64_t)gw * (gh > 1 ? 2 : 1);
    if (gw > 1) return ni + nb + 2 * (int64_t)(y - 1) + (x == gw - 1 ? 1 : 0);
    return ni + nb + (y - 1);
}
// level_search_order(gw, gh, level > 0), :326-336
__device__ __forceinline__ int2 level_order_at(int gw, int gh, int64_t k) {
    const int bw = gw - 1, bh = gh - 1;
    const int64_t n0 = initial_order_len(bw, bh);
    if (k < n0) return initial_order_at(bw, bh, k);
    k -= n0;
    if (k <= bw) return make_int2((int)k, bh);
    k -= bw + 1;
    return make_int2(bw, (int)k);
}
__device__ __forceinline__ uint32_t pack_xy(int x, int y) { return (uint32_t)(x & 0xFFFF) | ((uint32_t)y << 16); }
__device__ __forceinline__ int2 unpack_xy(uint32_t v) { return make_int2((int)(v & 0xFFFF), (int)(v >> 16)); }

// -------------------------------------------------------------------------------------------
struct DirScratch {
    uint2 *vec[2];       // field per level parity: x = (u16)dx | dy << 16, y = score
    uint8_t *luma[2];
    uint2 *proj[2];
    uint32_t *order, *order2;
    int *pos;
    unsigned long long *keys;
    unsigned *hist;
};
__device__ __forceinline__ int2 vmv(uint2 v) { return make_int2((int)(short)(v.x & 0xFFFF), (int)(short)(v.x >> 16)); }
__device__ __forceinline__ uint2 mkvec(int dx, int dy, unsigned score) {
    return make_uint2((uint32_t)(uint16_t)(short)dx | ((uint32_t)(uint16_t)(short)dy << 16), score);
}

// A direction's words in the pair's scratch (AnalyseParams::off_ctl, 64 bytes) from one launch to the
// next, and of a walked level. GO: the next walk has this direction's level to do; LATE: a bounded
// wait gave up; BAD: bad-SAD blocks of the level so far; GX, GY, ORDER: global predictor and length of
// the order; PREV: the other direction's projection exists; ABORT: the direction stopped (the status
// word says why), its payload stays unwritten.
enum { CTL_GO, CTL_LATE, CTL_BAD, CTL_GX, CTL_GY, CTL_ORDER, CTL_PREV, CTL_ABORT };

// Runs q (begun) to its end, one step after another.
template <class SH>
__device__ __forceinline__ void run_search(const Ctx &x, const BlkC &b, SH &s, int &ph, Search &q, int64_t idx, int &bad_count) {
    Gen g{0, 0, 0, 0, 0, 0, 0};
    while (search_next(q, x, b, idx, bad_count, g)) {
        int w;
        long long cost = q.bcost;
        unsigned sad = q.bsad;
        eval_step(x, b, s, ph, g, q.lambda, q.predx, q.predy, cost, sad, w);
        __syncwarp();
        q.bcost = cost;
        q.bsad = sad;
        search_took(q, g, w);
    }
}

// The payload's luma byte: the mean of the block's samples inside the level (:673-679).
__device__ __forceinline__ uint8_t block_mean(const BlkC &b, const LevelInfo &L, unsigned sum) {
    const int rows = b.py >= 0 ? imax(0, imin(b.bh, L.lh - b.py)) : 0;
    const int cols = b.px >= 0 ? imax(0, imin(b.bw, L.lw - b.px)) : 0;
    const unsigned cnt = (unsigned)(rows * cols);
    const unsigned dc = (cnt ? sum / cnt : 0) >> DC_SHIFT;
    return (uint8_t)(dc > 255 ? 255 : dc);
}

// The special candidates of a block (exact_search_block, :708-746), one per lane: lanes 0..8 the
// 3x3 neighbours in the reference's order, then the field's vector, the previous one, the global
// predictor and zero. The reference scans field, previous, global, zero, then the neighbours that
// are already processed, keeping the first of minimal cost, i.e. the least (cost, place).
constexpr int kField = 9, kPrev = 10, kGlobal = 11, kZero = 12;

// exact_sad of the lanes' candidates (lanes with `act`); equal vectors are evaluated once. With
// several warps in the group they share the candidates and meet at a barrier.
template <class SH>
__device__ __forceinline__ unsigned special_sads(const Ctx &x, const BlkC &b, SH &s, int &ph, bool act, int mx, int my) {
    const int lane = x.tid & 31;
    const unsigned long long key = ((unsigned long long)(unsigned)mx << 32) | (unsigned)my;
    const unsigned peers = __match_any_sync(kFull, key) & __ballot_sync(kFull, act);
    const int leader = act ? __ffs(peers) - 1 : lane;
    bool eval = act && leader == lane;
    const int rank = __popc(__ballot_sync(kFull, eval) & ((1u << lane) - 1u));
    if (x.nw > 1) eval = eval && rank % x.nw == (x.tid >> 5);
    unsigned L, C;
    eval_cands(x, b, eval, mx, my, L, C);
    unsigned sad = sat_add(L, C);
    if (x.nw > 1) {
        if (eval) s.slot[ph][lane] = sad;
        gsync(x);
        sad = s.slot[ph][lane];  // of the leaders; the others' entries are not used
        ph ^= 1;
    }
    return __shfl_sync(kFull, sad, leader);
}

// The per-direction search of one level (exact_search_level, :480-681). Every thread
// of the direction runs this with identical values; only the evaluation work is split.
__device__ __forceinline__ void search_level(const Ctx &x, DirSh &s, DirScratch &ds, const uint2 *prevp, int *status) {
    const AnalyseParams &P = *x.P;
    const LevelInfo &L = *x.L;
    const int level = x.level, gw = L.gw, gh = L.gh;
    const int64_t ncell = (int64_t)gw * gh;
    uint2 *field = ds.vec[level & 1];
    uint8_t *lumaf = ds.luma[level & 1];
    const int64_t order_len = s.order_len;
    const bool smallest = L.smallest != 0;
    const int lane = x.tid & 31, warp = x.tid >> 5;
    int bad_count = 0;
    int ph = 0;
    // The previous block's result: stored by thread 0 after the block's last barrier, so
    // the other warps take it from here until the next block's barrier publishes it.
    int64_t last_idx = -1;
    uint2 last_val = make_uint2(0, 0);
    for (int64_t k = 0; k < order_len; k++) {
        const int2 bxy = level == 0 ? initial_order_at(gw, gh, k) : unpack_xy(ds.order[k]);
        const int bx = bxy.x, by = bxy.y;
        const int64_t idx = (int64_t)by * gw + bx;
        int px = (level > 0 && bx == gw - 1) ? L.lw - P.block_w : bx * P.step_x;
        int py = (level > 0 && by == gh - 1) ? L.lh - P.block_h : by * P.step_y;
        px += L.pxoff;
        py += L.pyoff;
        const bool edge = level > 0 && (bx == gw - 1 || by == gh - 1);
        const int sxi = imin(bx, gw - 2), syi = imin(by, gh - 2);
        const int64_t sidx = (int64_t)syi * gw + sxi;
        if (sidx < 0 || sidx >= ncell || idx < 0 || idx >= ncell) {  // field[-1]: the reference panics
            if (x.tid == 0) { atomicOr(status, ST_PANIC); s.abort_ = 1; }
            break;
        }
        const int64_t fi = edge ? sidx : idx;
        const uint2 interp = fi == last_idx ? last_val : field[fi];
        const int2 imv = vmv(interp);
        BlkC &b = s.blk[warp];
        Search &q = s.q[warp];
        __syncwarp();  // the block before is stored
        make_blk(x, px, py, !smallest, b);
        const int phb = ph;  // this block's entries of dc and score; the specials' barrier below publishes them
        {
            unsigned part = 0;
            if (b.fast_src) part = stage_source(x, b);  // read by the evaluation, after the barrier below
            if (lane == 0) s.dc[phb][warp] = part;
        }
        const bool dc_fast = b.fast_src && b.px2 == px && b.py2 == py;
        if (!dc_fast && warp == x.nw - 1) {  // block_luma_dc on the reference's read path
            const uint2 r = eval_slow(x, px, py, 0, 0, SLOW_DC);
            if (lane == 0) s.dcs[phb] = r.x;
        }
        if (edge && !smallest && warp == 0) {  // re-score the predictor at its source block (:536-549)
            const uint2 r = eval_slow(x, sxi * P.step_x, syi * P.step_y, imv.x, imv.y, SLOW_CHROMA);
            if (lane == 0) s.score[phb] = sad_of(r);
        }
        gsync(x);
        const unsigned pred_score = edge && !smallest ? s.score[phb] : interp.y;
        const bool field_valid = pred_score != 0xFFFFFFFFu;
        // ---- the special candidates, one per lane
        bool act = false;
        int mx = 0, my = 0;
        if (lane < 9) {
            const int ny = by - 1 + lane / 3, nx = bx - 1 + lane % 3;
            if (ny >= 0 && ny < gh && nx >= 0 && nx < gw) {
                const int64_t ci = (int64_t)ny * gw + nx;
                const int64_t p = level == 0 ? initial_order_pos(gw, gh, nx, ny) : (int64_t)ds.pos[ci];
                act = p < k;
                if (act) { const int2 m = vmv(ci == last_idx ? last_val : field[ci]); mx = m.x; my = m.y; }
            }
        } else if (lane == kField) {
            act = field_valid; mx = imv.x; my = imv.y;
        } else if (lane == kPrev) {
            if (prevp) {
                const uint2 pv = prevp[idx];
                act = pv.y != 0xFFFFFFFFu && pv.y > 0;
                const int2 m = vmv(pv);
                mx = m.x; my = m.y;
            }
        } else if (lane == kGlobal) {
            act = true; mx = s.gx; my = s.gy;
        } else if (lane == kZero) {
            act = true;
        }
        const unsigned seeds = __ballot_sync(kFull, act) & 0x1FFu;
        if (__popc(seeds) > 8) {  // seeds[8] overflows: the reference panics
            if (x.tid == 0) { atomicOr(status, ST_PANIC); s.abort_ = 1; }
            break;
        }
        const bool search = !(level == 0 && P.distance == 0);
        if (!search) act = lane == (field_valid ? kField : kZero);
        const unsigned sd = special_sads(x, b, s, ph, act, mx, my);
        // the penalty of the lane's special candidate; read here, since a meeting of the lanes makes the loop read it anew
    const int pp = lane < 9 ? P.pnbour : lane == kPrev ? P.prev : lane == kGlobal ? P.pglobal : lane == kZero ? P.pzero : 0;
        const int place = lane < 9 ? 4 + __popc(seeds & ((1u << lane) - 1u)) : lane - kField;
        const long long cost = (long long)sd + (((long long)pp * sd) >> 8);
        const int wl = first_min(act, cost, place);
        const unsigned wsad = __shfl_sync(kFull, sd, wl);
        q.bmx = __shfl_sync(kFull, mx, wl); q.bmy = __shfl_sync(kFull, my, wl);
        q.bsad = wsad;
        q.bcost = (long long)wsad;
        int lambda = 0, radius = 0, stype = 0, ppx = imv.x, ppy = imv.y;
        if (search) {
            const long long cf = __shfl_sync(kFull, cost, kField), cp = __shfl_sync(kFull, cost, kPrev);
            const bool prev = __shfl_sync(kFull, act, kPrev);
            const int pmx = __shfl_sync(kFull, mx, kPrev), pmy = __shfl_sync(kFull, my, kPrev);
            if (prev && (!field_valid || cp < cf)) { ppx = pmx; ppy = pmy; }
            lambda = adapt_lambda(L.lambda_base, L.lsad, pred_score);
            radius = L.base_radius;
            if (level > 0 && P.coarse_distance < 0) {
                radius = adaptive_radius(radius, block_activity(x.P, x.L, x.S.y, b.px2, b.py2, px, py));
            }
            stype = (edge && level == 1) ? 0 : L.search_type;
        }
        unsigned dcsum = 0;
        if (dc_fast)
            for (int w = 0; w < x.nw; w++) dcsum += s.dc[phb][w];
        else dcsum = s.dcs[phb];
        q.stype = stype; q.radius = radius; q.lambda = lambda;
        q.ppx = ppx; q.ppy = ppy; q.own_x = imv.x; q.own_y = imv.y;
        search_begin(q, search ? RS_ALL : RS_NONE);
        run_search(x, b, s, ph, q, idx, bad_count);
        // ---- store (:673-679)
        const uint2 v = mkvec(q.bmx, q.bmy, smallest ? sat_mul(q.bsad, 3) : q.bsad);
        if (x.tid == 0) {
            field[idx] = v;
            lumaf[idx] = block_mean(b, L, dcsum);
        }
        last_idx = idx;
        last_val = v;
        if (ph == phb) ph ^= 1;  // the next block writes other entries of dc and score
    }
}

// ---- a level walked by several warps (look-ahead: speculative and exact) -------------------
// exact_search_level (:480-681) with D blocks of a direction in flight, one per warp. Warp g
// searches blocks g, g + D, g + 2D, ... of the level's order. Of what a block reads, only these come
// from blocks searched before it: the vectors of its processed neighbours, taken as seeds
// (:570-585); at level > 0 an edge block's predictor, the vector of an inner cell (:520-549); the
// bad-SAD count (:605-616). Everything else (the interpolated predictor, lambda, radius, search
// type, the previous-frame, zero and global candidates) comes from the coarser level, the other
// direction and the block itself.
//
// A block publishes its vector in one 64-bit word per cell (AnalyseParams::off_keys, cleared before
// the level): the vector and a tag, stored and read in one piece, so the word itself says what it is
// and no fence or count is needed. The tag says whether the vector is the final one or a tentative
// one: a block searches with the vectors that its processed neighbours have published when it starts,
// tentative ones included (one that has published nothing is left out), publishes the result as
// tentative, and then watches the words of the neighbours that were not final. When one changes, the
// selection among the special candidates is made anew (:740-746 keep the first candidate of minimal
// cost, i.e. the least (cost, place)), and if that selects another vector the refinement runs again
// from it and the result is published anew; with the same vector (hence the same SAD) the refinement
// already run is the reference's. Once all of them are final and were the ones used, the block's own
// vector is final. So every stored vector is the reference's, whatever D and however the warps run,
// a block depends on its neighbours alone, not on the whole order before it, and a repeated refinement
// holds up the blocks after it only if its outcome differs from what they used: where a fifth of the
// blocks repeat it (noisy fields), waiting for each in turn was the larger part of the walk.
//
// The bad-SAD test needs the number of bad blocks before this one. Its threshold only grows with
// that number, so a block that is not bad by the number known so far is not bad; any other
// waits until every earlier block has passed its test (each warp publishes the next block it has not
// tested, in the histogram's words, which are free while a level is searched) and then reads the
// number. The expansion of a block that looks bad runs before that, while its seeds may still change
// (it is what such a block mostly does: at 640x360 the coarser levels took 2.5 to 3 times as long with
// the expansions one after another). The lowest block that is not finished waits for nothing, and every
// warp takes its blocks in order, so the warps, all resident, always make progress; the waits are
// bounded all the same (walk_wait.h).
// Bound: at few pairs the chain (a link is the wait's L2 round trip where nothing changed, a refinement where
// something did), at many the latency of the candidates' loads (issue 33 %). With four warps per direction
// that handed over in order, and the coarser levels in the pair's CTA: one 1080p pair 287 ms, 23 ms now; 32
// frames of 640x360 12.6 and 3.5 ms; 240 frames of 1080p 1087 and 730 ms.
// A level with an input on which the reference would panic takes search_level instead.
// stats (nullable): [0] blocks, [1] blocks that started before all their processed neighbours were
// final, [2] seeds evaluated after the start (the others had the vector of a candidate already
// evaluated), [3] blocks that ran their refinement again.
__device__ __forceinline__ unsigned long long ld_tag(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_tag(unsigned long long *p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ int ld_word(const int *p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(int *p, int v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// A word that other warps change, as one value for the whole warp: what the lanes decide by it has to be the
// same in all of them, and each lane's own load may find another.
__device__ __forceinline__ int ld_warp_word(const int *p) { return __shfl_sync(kFull, ld_word(p), 0); }

// The warp waits until done() holds in every lane. Bounded: false once `cycles` have passed (LevelInfo::wait_cycles)
// or another warp of the direction has given up (the caller flags ST_TIMEOUT and carries on). After one wait of a
// direction has given up its others return at once, so a failure costs one bound, not one per block.
template <class F>
__device__ __forceinline__ bool spin(F done, int *late, int64_t cycles) {
    const long long t0 = clock64();
    for (int it = 1;; it++) {
        if (__all_sync(kFull, done())) return true;
        if ((it & 127) == 0) {
            const int give_up = ld_word(late) || clock64() - t0 > cycles;
            if (__shfl_sync(kFull, give_up, 0)) {
                if ((threadIdx.x & 31) == 0) st_word(late, 1);
                return false;
            }
        }
    }
}

enum { TAG_NONE, TAG_TENTATIVE, TAG_FINAL };
__device__ __forceinline__ unsigned long long tag_word(int tag, int mx, int my) {
    return ((unsigned long long)tag << 32) | mkvec(mx, my, 0).x;
}

template <class SH>
__device__ __forceinline__ void walk_level(const Ctx &x, SH &s, const DirScratch &ds, const uint2 *prevp, int g, int D,
                                           int order_len, int gxv, int gyv, int *ctl, int *status, unsigned long long *stats) {
    const AnalyseParams &P = *x.P;
    const LevelInfo &L = *x.L;
    const int level = x.level, gw = L.gw, gh = L.gh;
    uint2 *field = ds.vec[level & 1];
    uint8_t *lumaf = ds.luma[level & 1];
    const bool smallest = L.smallest != 0;
    int *progress = (int *)ds.hist;
    const int lane = x.tid, wi = x.wbase;
    BlkC &b = s.blk[wi];
    Search &q = s.q[wi];
    int n_blk = 0, n_def = 0, n_eval = 0, n_rerun = 0;
    bool late = false;
    // the penalty of the lane's special candidate; read here, since a meeting of the lanes makes the loop read it anew
    const int pp = lane < 9 ? P.pnbour : lane == kPrev ? P.prev : lane == kGlobal ? P.pglobal : lane == kZero ? P.pzero : 0;
    for (int k = g; k < order_len; k += D) {
        const int2 bxy = level == 0 ? initial_order_at(gw, gh, k) : unpack_xy(ds.order[k]);
        const int bx = bxy.x, by = bxy.y;
        const int idx = by * gw + bx;
        const bool edge = level > 0 && (bx == gw - 1 || by == gh - 1);
        // ---- the special candidates, one per lane (see special_sads)
        const int ncell = idx + (lane < 9 ? (lane / 3 - 1) * gw + lane % 3 - 1 : 0);
        unsigned seeds, openm, actm;  // lanes holding a seed, one that is not final yet, a candidate
        unsigned pred_score;
        {
            int px = (level > 0 && bx == gw - 1) ? L.lw - P.block_w : bx * P.step_x;
            int py = (level > 0 && by == gh - 1) ? L.lh - P.block_h : by * P.step_y;
            px += L.pxoff;
            py += L.pyoff;
            const int sxi = imin(bx, gw - 2), syi = imin(by, gh - 2);
            bool act = false, seed = false, open = false;
            int mx = 0, my = 0;
            if (lane < 9) {
                const int ny = by - 1 + lane / 3, nx = bx - 1 + lane % 3;
                if (ny >= 0 && ny < gh && nx >= 0 && nx < gw) {
                    seed = (level == 0 ? (int)initial_order_pos(gw, gh, nx, ny) : ds.pos[ncell]) < k;
                    if (seed) {
                        const unsigned long long v = ld_tag(ds.keys + ncell);
                        const int2 m = vmv(make_uint2((unsigned)v, 0));
                        mx = m.x; my = m.y;
                        act = (int)(v >> 32) != TAG_NONE;
                        open = (int)(v >> 32) != TAG_FINAL;
                    }
                }
            } else if (lane == kPrev) {
                if (prevp) {
                    const uint2 pv = prevp[idx];
                    act = pv.y != 0xFFFFFFFFu && pv.y > 0;
                    const int2 m = vmv(pv);
                    mx = m.x; my = m.y;
                }
            } else if (lane == kGlobal) {
                act = true; mx = gxv; my = gyv;
            } else if (lane == kZero) {
                act = true;
            }
            uint2 interp;
            if (edge) {  // its inner cell comes earlier in the order (level_spec_ok): that cell's final vector
                unsigned long long v = 0;
                if (!spin([&] { v = ld_tag(ds.keys + syi * gw + sxi); return (int)(v >> 32) == TAG_FINAL; }, ctl + CTL_LATE, L.wait_cycles)) late = true;
                interp = make_uint2((unsigned)v, 0);  // the score is taken anew below
            } else {
                interp = field[idx];
            }
            const int2 imv = vmv(interp);
            if (lane == kField) { mx = imv.x; my = imv.y; }
            q.own_x = q.ppx = imv.x; q.own_y = q.ppy = imv.y;
            make_blk(x, px, py, !smallest, b);
            unsigned dcsum = 0;
            if (b.fast_src) dcsum = stage_source(x, b);
            if (!(b.fast_src && b.px2 == px && b.py2 == py))  // block_luma_dc on the reference's read path
                dcsum = eval_slow(x, px, py, 0, 0, SLOW_DC).x;
            if (lane == 0) lumaf[idx] = block_mean(b, L, dcsum);
            pred_score = interp.y;
            if (edge)  // re-score the predictor at its source block (:536-549)
                pred_score = sad_of(eval_slow(x, sxi * P.step_x, syi * P.step_y, imv.x, imv.y, SLOW_CHROMA));
            const bool field_valid = pred_score != 0xFFFFFFFFu;
            if (lane == kField) act = field_valid;
            const bool search = !(level == 0 && P.distance == 0);
            if (!search) act = lane == (field_valid ? kField : kZero);
            seeds = __ballot_sync(kFull, seed);  // at most 8 (level_spec_ok)
            openm = __ballot_sync(kFull, open);
            actm = __ballot_sync(kFull, act);
            s.lmx[wi][lane] = mx;
            s.lmy[wi][lane] = my;
            __syncwarp();
        }
        unsigned freshm = actm;  // lanes whose candidate is to be evaluated
        bool started = false, reran = false, published = false;
        int selx = 0, sely = 0;
        Gen g_{0, 0, 0, 0, 0, 0, 0};  // the step in work, its next 32 candidates, and the one accepted so far
        int base = 0, win = -1;
        bool stepping = false;
        int bad_count = 0;
        bool final = false, expanded = false;
        const bool may_be_bad = level > 0 && P.coarse_bad_sad > 0;
        // Each turn evaluates up to 32 candidates, one per lane: special ones that are new, else the next
        // of the search step in work (one call site of the evaluation, which is inlined). While a search
        // runs, seeds that have become final are looked at between its turns; tentative ones only when
        // there is nothing else to do, since the work they cause may be in vain.
        for (;;) {
            if (!freshm && !stepping) {
                if (search_next(q, x, b, idx, bad_count, g_)) { stepping = true; base = 0; win = -1; }
                else {
                    if (final) break;
                    // ---- the refinement is done. The bad-SAD expansion depends on its outcome and on the
                    // test alone, so it runs at once where the count of bad blocks known by now makes the
                    // block bad, and the outcome before it is kept in case the exact count says otherwise.
                    if (may_be_bad && !expanded && idx > 1 && (int)q.bsad > P.coarse_bad_sad) {
                        const int known = ld_warp_word(ctl + CTL_BAD);
                        if ((int)q.bsad > bad_limit(P, known)) {
                            q.rx = q.bmx; q.ry = q.bmy; q.rsad = q.bsad; q.rcost = q.bcost;
                            expanded = true;
                            bad_count = known;
                            search_begin(q, RS_BAD_ONLY);
                            continue;
                        }
                    }
                    if (openm) {  // publish, then wait for news
                        const unsigned long long word = tag_word(TAG_TENTATIVE, q.bmx, q.bmy);
                        if (!published && lane == 0) st_tag(ds.keys + idx, word);
                        published = true;
                        // not subject to the bad-SAD test: final as soon as its seeds are
                        const bool sure = !expanded && (!may_be_bad || idx <= 1 || (int)q.bsad <= P.coarse_bad_sad);
                        const bool open = (openm >> lane) & 1u, act = (actm >> lane) & 1u;
                        const int mx = s.lmx[wi][lane], my = s.lmy[wi][lane];
                        unsigned long long v = 0;
                        if (!spin([&] {
                                if (open) v = ld_tag(ds.keys + ncell);
                                const int2 m = vmv(make_uint2((unsigned)v, 0));
                                freshm = __ballot_sync(kFull, open && (int)(v >> 32) != TAG_NONE && (!act || m.x != mx || m.y != my));
                                return freshm || !(open && (int)(v >> 32) != TAG_FINAL);
                            }, ctl + CTL_LATE, L.wait_cycles)) {
                            late = true;
                            openm = 0;
                        } else if (!freshm && sure) {  // the next block in the chain waits for this store
                            if (lane == 0) st_tag(ds.keys + idx, word ^ ((unsigned long long)(TAG_TENTATIVE ^ TAG_FINAL) << 32));
                        }
                        openm &= ~__ballot_sync(kFull, (int)(v >> 32) == TAG_FINAL);
                        actm |= freshm;
                        __syncwarp();
                        if ((freshm >> lane) & 1u) { const int2 m = vmv(make_uint2((unsigned)v, 0)); s.lmx[wi][lane] = m.x; s.lmy[wi][lane] = m.y; }
                        __syncwarp();
                        continue;
                    }
                    final = true;  // every seed is final and is the one used
                    if (may_be_bad) {
                        // The exact test. The count only grows, so a block that is not bad by what is known of it
                        // is not bad; the others wait for every earlier block's test.
                        const unsigned sad = expanded ? q.rsad : q.bsad;
                        bool bad = idx > 1 && (int)sad > P.coarse_bad_sad;
                        if (bad) bad = (int)sad > bad_limit(P, ld_warp_word(ctl + CTL_BAD));
                        if (bad) {
                            if (!spin([&] {
                                    bool ok = true;
                                    for (int h = lane; h < D; h += 32) ok = ok && (h == g || ld_word(progress + h) >= k);
                                    return ok;
                                }, ctl + CTL_LATE, L.wait_cycles))
                                late = true;
                            __threadfence();
                            bad_count = ld_warp_word(ctl + CTL_BAD);
                            bad = (int)sad > bad_limit(P, bad_count);
                            if (bad && lane == 0) { st_word(ctl + CTL_BAD, bad_count + 1); __threadfence(); }
                            __syncwarp();
                        }
                        if (lane == 0) st_word(progress + g, k + D);
                        if (bad && !expanded) { search_begin(q, RS_BAD_ONLY); continue; }
                        __syncwarp();
                        if (!bad && expanded) { q.bmx = q.rx; q.bmy = q.ry; q.bsad = q.rsad; q.bcost = q.rcost; }
                    }
                    break;
                }
            }
            // ---- what to evaluate: exact_sad of the new special candidates (an equal vector's that is
            // known, else one for all that are equal), or the step's candidates inside the bounds whose
            // motion penalty does not reach the best cost (see eval_step)
            const bool special = freshm != 0;
            bool eval;
            int vx, vy, from = lane;
            long long motion = 0;
            if (special) {
                vx = s.lmx[wi][lane]; vy = s.lmy[wi][lane];
                const unsigned peers = __match_any_sync(kFull, ((unsigned long long)(unsigned)vx << 32) | (unsigned)vy);
                const unsigned known = peers & actm & ~freshm, asked = peers & freshm;
                const bool fresh = (freshm >> lane) & 1u;
                if (fresh) from = __ffs(known ? known : asked) - 1;
                eval = fresh && !known && from == lane;
                if (started) n_eval += __popc(__ballot_sync(kFull, eval));
            } else {
                const int2 m = gen_mv(g_, imin(base + lane, g_.n - 1));
                vx = m.x; vy = m.y;
                motion = motion_penalty(q.lambda, q.predx, q.predy, vx, vy);
                eval = base + lane < g_.n && vx >= b.bnd0 && vy >= b.bnd1 && vx < b.bnd2 && vy < b.bnd3 && motion < q.bcost;
            }
            unsigned long long news = 0;
            const unsigned lookm = started ? openm : 0;
            if ((lookm >> lane) & 1u) news = ld_tag(ds.keys + ncell);  // in flight during the evaluation
            unsigned l, c;
            eval_cands(x, b, eval, vx, vy, l, c);
            if (special) {
                if (eval) s.lsd[wi][lane] = sat_add(l, c);
                __syncwarp();
                const unsigned sd = s.lsd[wi][from];
                __syncwarp();
                s.lsd[wi][lane] = sd;
                freshm = 0;
                const int place = lane < 9 ? 4 + __popc(seeds & ((1u << lane) - 1u)) : lane - kField;
                const long long cost = (long long)sd + (((long long)pp * sd) >> 8);
                const int wl = first_min((actm >> lane) & 1u, cost, place);
                const int nx = s.lmx[wi][wl], ny = s.lmy[wi][wl];
                const unsigned nsad = __shfl_sync(kFull, sd, wl);
                const bool search = !(level == 0 && P.distance == 0);
                if (!started) {
                    if (search) {
                        const long long cf = __shfl_sync(kFull, cost, kField), cp = __shfl_sync(kFull, cost, kPrev);
                        if (((actm >> kPrev) & 1u) && (!((actm >> kField) & 1u) || cp < cf)) { q.ppx = s.lmx[wi][kPrev]; q.ppy = s.lmy[wi][kPrev]; }
                        q.lambda = adapt_lambda(L.lambda_base, L.lsad, pred_score);
                        int radius = L.base_radius;
                        if (level > 0 && P.coarse_distance < 0)
                            radius = adaptive_radius(radius, block_activity(x.P, x.L, x.S.y, b.px2, b.py2, b.px, b.py));
                        q.radius = radius;
                        q.stype = (edge && level == 1) ? 0 : L.search_type;
                    } else {
                        openm = 0;  // no seed takes part
                    }
                    n_def += openm != 0;
                }
                if (!started || nx != selx || ny != sely) {  // the refinement, from this vector
                    reran = started;
                    selx = nx; sely = ny;
                    q.bmx = nx; q.bmy = ny; q.bsad = nsad; q.bcost = (long long)nsad;
                    search_begin(q, search ? RS_REFINE_ONLY : RS_NONE);
                    stepping = false;
                    published = expanded = false;
                }
                started = true;
            } else {
                const long long K = motion + pen(x.pnew, l) + (b.chroma ? pen(x.pnew, c) : 0LL);  // :1158-1221
                const unsigned sad = sat_add(l, c);
                long long best = q.bcost;
                unsigned best_sad = q.bsad;
                if (x.pnew < -256) {  // exact sequential semantics for penalties that can be negative
                    for (unsigned m = __ballot_sync(kFull, eval); m; m &= m - 1) {
                        const int j = __ffs(m) - 1;
                        const long long mj = __shfl_sync(kFull, motion, j), kj = __shfl_sync(kFull, K, j);
                        const unsigned sj = __shfl_sync(kFull, sad, j);
                        if (mj < best && kj < best) { best = kj; best_sad = sj; win = base + j; }
                    }
                } else {
                    const int j = first_min(eval && K < best, K, lane);
                    if (j >= 0) {
                        best = __shfl_sync(kFull, K, j);
                        best_sad = __shfl_sync(kFull, sad, j);
                        win = base + j;
                    }
                }
                __syncwarp();
                q.bcost = best; q.bsad = best_sad;
                __syncwarp();
                base += 32;
                if (base >= g_.n) { search_took(q, g_, win); stepping = false; }
            }
            if (lookm) {  // seeds that have become final
                const bool fin = (int)(news >> 32) == TAG_FINAL;
                const unsigned finm = __ballot_sync(kFull, fin);
                if (finm) {
                    const int2 m = vmv(make_uint2((unsigned)news, 0));
                    const bool fresh = fin && (!((actm >> lane) & 1u) || m.x != s.lmx[wi][lane] || m.y != s.lmy[wi][lane]);
                    freshm = __ballot_sync(kFull, fresh);
                    __syncwarp();
                    if (fresh) { s.lmx[wi][lane] = m.x; s.lmy[wi][lane] = m.y; }
                    actm |= finm;
                    openm &= ~finm;
                    __syncwarp();
                }
            }
        }
        n_blk++;
        n_rerun += reran;
        // ---- store (:673-679)
        if (lane == 0) {
            const unsigned bsad = q.bsad;
            const uint2 v = mkvec(q.bmx, q.bmy, smallest ? sat_mul(bsad, 3) : bsad);
            st_tag(ds.keys + idx, tag_word(TAG_FINAL, q.bmx, q.bmy));
            field[idx] = v;
        }
        __syncwarp();
    }
    if (lane == 0) {
        if (late) { atomicOr(status, ST_TIMEOUT); ctl[CTL_ABORT] = 1; }
        if (stats && level == 0) {
            atomicAdd(stats + 0, (unsigned long long)n_blk);
            atomicAdd(stats + 1, (unsigned long long)n_def);
            atomicAdd(stats + 2, (unsigned long long)n_eval);
            atomicAdd(stats + 3, (unsigned long long)n_rerun);
        }
    }
}
// What a walk starts from: no cell published, no block tested. Every thread of the direction.
__device__ __forceinline__ void start_walk(const Ctx &x, const DirScratch &ds, int *ctl, int ncell) {
    for (int i = x.tid; i < ncell; i += NT) ds.keys[i] = 0;
    for (int h = x.tid; h < kMaxWalkers; h += NT) ((int *)ds.hist)[h] = h;
    if (x.tid == 0) { ctl[CTL_LATE] = 0; ctl[CTL_BAD] = 0; }
}
// The direction's warps of one CTA walk the level together.
__device__ __forceinline__ void walk_in_cta(const Ctx &xd, DirSh &s, const DirScratch &ds, const uint2 *prevp, int *ctl,
                                            int *status, unsigned long long *stats, unsigned char *area, int groups) {
    start_walk(xd, ds, ctl, xd.L->gw * xd.L->gh);
    __threadfence();
    dbar(xd.d);
    const int g = xd.tid >> 5;
    Ctx x = xd;
    x.nw = 1;
    x.wbase = g;
    x.tid = xd.tid & 31;
    set_stage(x, area, groups, g, g);
    walk_level(x, s, ds, prevp, g, NW, s.order_len, s.gx, s.gy, ctl, status, stats);
    __threadfence();
    dbar(xd.d);
    if (xd.tid == 0 && ctl[CTL_ABORT]) s.abort_ = 1;
    dbar(xd.d);
}

// Whether walk_level may run this level: it takes neither the reference's panics (search_level
// reports them at the block where the reference stops) nor grids below 3 x 3, nor an order that
// visits a cell twice, leaves one out or puts an edge block before its inner cell.
// Called by every thread of the direction; the answer is the same in all of them.
__device__ __forceinline__ bool level_spec_ok(const Ctx &x, DirSh &s, const DirScratch &ds) {
    const LevelInfo &L = *x.L;
    const int level = x.level, gw = L.gw, gh = L.gh;
    const int64_t ncell = (int64_t)gw * gh, order_len = s.order_len;
    if (gw < 3 || gh < 3 || order_len != ncell || (level > 0 && L.smallest)) return false;
    if (x.tid == 0) s.unsafe_ = 0;
    dbar(x.d);
    int bad = 0;
    auto pos_of = [&](int cx, int cy) { return level == 0 ? initial_order_pos(gw, gh, cx, cy) : (int64_t)ds.pos[(int64_t)cy * gw + cx]; };
    for (int64_t k = x.tid; k < order_len && !bad; k += NT) {
        const int2 bxy = level == 0 ? initial_order_at(gw, gh, k) : unpack_xy(ds.order[k]);
        const int bx = bxy.x, by = bxy.y;
        if (bx < 0 || by < 0 || bx >= gw || by >= gh || pos_of(bx, by) != k) {
            bad = 1;
            break;
        }
        if (level > 0 && (bx == gw - 1 || by == gh - 1) && pos_of(imin(bx, gw - 2), imin(by, gh - 2)) >= k) bad = 1;
        int nproc = 0;
        for (int q = 0; q < 9; q++) {
            const int ny = by - 1 + q / 3, nx = bx - 1 + q % 3;
            if (ny < 0 || ny >= gh || nx < 0 || nx >= gw) continue;
            nproc += pos_of(nx, ny) < k;
        }
        if (nproc > 8) bad = 1;
    }
    if (bad) s.unsafe_ = 1;
    dbar(x.d);
    const bool ok = s.unsafe_ == 0;
    dbar(x.d);
    return ok;
}

__device__ __forceinline__ long long floor_div(long long a, long long b) {  // i64::div_euclid for b > 0
    const long long q = a / b;
    return (a % b != 0 && a < 0) ? q - 1 : q;
}

// exact_recalculate (:1326-1451): when refine[0].thsad is set, the level-0 field is
// interpolated onto the half-size output blocks and each block whose interpolated score is
// above the threshold is searched again. Blocks do not read each other's results, so the
// visiting order does not matter: one warp takes one block, with the same evaluation machinery as
// the hierarchy. x: a one-warp group; `shape`: the block shape x is set to, -1 before the first
// block. Output: ds.vec[1] / ds.luma[1].
template <class SH>
__device__ __forceinline__ void refine_block(Ctx &x, SH &s, DirScratch &ds, int bx, int by, int &shape) {
    const AnalyseParams &P = *x.P;
    const uint2 *field = ds.vec[0];
    const int ogw = P.lv[0].gw, ogh = P.lv[0].gh;
    const int obw = P.block_w, obh = P.block_h, osx = P.step_x, osy = P.step_y;
    const int bw = P.out_bw, bh = P.out_bh;
    const int sx = imax(bw - P.out_ox, 1), sy = imax(bh - P.out_oy, 1);
    const int gw = P.out_gw, gh = P.out_gh;
    int ph = 0;
    const int cx = bw / 2 + sx * bx, cy = bh / 2 + sy * by;
    const int ox_ = (cx - obw / 2) / osx, oy_ = (cy - obh / 2) / osy;
    const long long dx_ = imax(cx - (obw / 2 + osx * ox_), 0), dy_ = imax(cy - (obh / 2 + osy * oy_), 0);
    const uint2 p00 = field[(int64_t)iclamp(oy_, 0, ogh - 1) * ogw + iclamp(ox_, 0, ogw - 1)];
    const uint2 p10 = field[(int64_t)iclamp(oy_, 0, ogh - 1) * ogw + iclamp(ox_ + 1, 0, ogw - 1)];
    const uint2 p01 = field[(int64_t)iclamp(oy_ + 1, 0, ogh - 1) * ogw + iclamp(ox_, 0, ogw - 1)];
    const uint2 p11 = field[(int64_t)iclamp(oy_ + 1, 0, ogh - 1) * ogw + iclamp(ox_ + 1, 0, ogw - 1)];
    auto interp = [&](long long a, long long b_, long long c, long long d) {
        const long long top = a * osx + dx_ * (b_ - a);
        const long long bottom = c * osx + dx_ * (d - c);
        return floor_div(top + floor_div(dy_ * (bottom - top), osy), osx);
    };
    const int2 m00 = vmv(p00), m10 = vmv(p10), m01 = vmv(p01), m11 = vmv(p11);
    const int mvx = (int)interp(m00.x, m10.x, m01.x, m11.x);
    const int mvy = (int)interp(m00.y, m10.y, m01.y, m11.y);
    const long long parent = interp(p00.y, p10.y, p01.y, p11.y) * (long long)(bw * bh) / (long long)(obw * obh);
    const int px = bx * sx, py = by * sy;
    const bool border = bx == 0 || by == 0 || bx == gw - 1 || by == gh - 1;
    const int factor = (border && bw > 4) ? 3 : 1;
    const int epx = px + (factor == 3 ? bw / 4 : 0), epy = py + (factor == 3 ? bh / 4 : 0);
    x.L = &P.rlv[factor == 3 ? 1 : 0];
    const LevelInfo &L = *x.L;
    if (shape != factor) {
        shape = factor;
        __syncwarp();
        set_groups(x);
    }
    x.pnew = P.pnew / factor;
    BlkC &b = s.blk[x.wbase];
    Search &q = s.q[x.wbase];
    make_blk(x, epx, epy, true, b);
    // exact_clip (:1269-1273) of the interpolated vector into mv_bounds
    const int pmx = iclamp(mvx, b.bnd0, imax(b.bnd2 - 1, b.bnd0)), pmy = iclamp(mvy, b.bnd1, imax(b.bnd3 - 1, b.bnd1));
    const int threshold = P.refine_thsad / factor;
    const bool search = parent > (long long)threshold;
    unsigned dcsum = 0;
    if (b.fast_src) dcsum = stage_source(x, b);
    __syncwarp();
    if (!b.fast_src) {
        dcsum = eval_slow(x, b.px, b.py, 0, 0, SLOW_DC).x;
    }
    unsigned best_sad = parent < 0 ? 0u : (parent > 0xFFFFFFFFLL ? 0xFFFFFFFFu : (unsigned)parent);
    long long best = parent < 0 ? 0 : parent;
    if (search) {
        unsigned l, c;
        eval_cands(x, b, (x.tid & 31) == 0, pmx, pmy, l, c);
        best_sad = __shfl_sync(kFull, sat_add(l, c), 0);  // exact_sad at the clipped predictor
        best = (long long)best_sad;
    }
    q.bmx = pmx; q.bmy = pmy;
    q.bsad = best_sad; q.bcost = best;
    const int lambda = by == 0 ? 0 : (P.lambda >> 2) / factor;
    int bad = 0;
    q.stype = P.refine_search_type; q.radius = abs(P.refine_distance); q.lambda = lambda;
    q.ppx = q.own_x = pmx; q.ppy = q.own_y = pmy;
    search_begin(q, search ? RS_ALL : RS_NONE);
    run_search(x, b, s, ph, q, 0, bad);
    if ((x.tid & 31) == 0) {
        ds.vec[1][(int64_t)by * gw + bx] = mkvec(q.bmx, q.bmy, sat_mul(q.bsad, (unsigned)factor));
        ds.luma[1][(int64_t)by * gw + bx] = block_mean(b, L, dcsum);
    }
    __syncwarp();  // the next block stages over this one's source
}

// exact_global_doubled (:1285-1324) over the dir's threads
__device__ void global_doubled(const Ctx &x, DirSh &s, const uint2 *field, int64_t n, unsigned *hist) {
    int mode[2];
    for (int comp = 0; comp < 2; comp++) {
        int mn = 0x7FFFFFFF, mx = (int)0x80000000;
        for (int64_t i = x.tid; i < n; i += NT) {
            const int2 v = vmv(field[i]);
            const int c = comp == 0 ? v.x : v.y;
            mn = imin(mn, c); mx = imax(mx, c);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) { mn = imin(mn, __shfl_xor_sync(~0u, mn, o)); mx = imax(mx, __shfl_xor_sync(~0u, mx, o)); }
        if ((x.tid & 31) == 0) { s.r32[x.tid >> 5][0] = mn; s.r32[x.tid >> 5][1] = mx; }
        dbar(x.d);
        mn = s.r32[0][0]; mx = s.r32[0][1];
        for (int w = 1; w < NW; w++) { mn = imin(mn, s.r32[w][0]); mx = imax(mx, s.r32[w][1]); }
        dbar(x.d);
        if (n == 0) { mode[comp] = 0; continue; }
        for (int v = mn + x.tid; v <= mx; v += NT) hist[v + 32768] = 0;
        dbar(x.d);
        for (int64_t i = x.tid; i < n; i += NT) {
            const int2 v = vmv(field[i]);
            atomicAdd(&hist[(comp == 0 ? v.x : v.y) + 32768], 1u);
        }
        dbar(x.d);
        // most frequent value, the smallest one among ties
        unsigned bc = 0;
        int bv = 0x7FFFFFFF;
        for (int v = mn + x.tid; v <= mx; v += NT) {
            const unsigned c = hist[v + 32768];
            if (c > bc || (c == bc && v < bv)) { bc = c; bv = v; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            unsigned oc = __shfl_xor_sync(~0u, bc, o);
            int ov = __shfl_xor_sync(~0u, bv, o);
            if (oc > bc || (oc == bc && ov < bv)) { bc = oc; bv = ov; }
        }
        if ((x.tid & 31) == 0) { s.r32[x.tid >> 5][0] = (int)bc; s.r32[x.tid >> 5][1] = bv; }
        dbar(x.d);
        bc = (unsigned)s.r32[0][0]; bv = s.r32[0][1];
        for (int w = 1; w < NW; w++) {
            const unsigned oc = (unsigned)s.r32[w][0];
            const int ov = s.r32[w][1];
            if (oc > bc || (oc == bc && ov < bv)) { bc = oc; bv = ov; }
        }
        mode[comp] = bv;
        dbar(x.d);
    }
    long long sx = 0, sy = 0, cnt = 0;
    for (int64_t i = x.tid; i < n; i += NT) {
        const int2 v = vmv(field[i]);
        if (abs(v.x - mode[0]) < 6 && abs(v.y - mode[1]) < 6) { sx += v.x; sy += v.y; cnt++; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sx += __shfl_xor_sync(~0u, sx, o); sy += __shfl_xor_sync(~0u, sy, o); cnt += __shfl_xor_sync(~0u, cnt, o);
    }
    if ((x.tid & 31) == 0) { s.r64[x.tid >> 5][0] = sx; s.r64[x.tid >> 5][1] = sy; s.r64[x.tid >> 5][2] = cnt; }
    dbar(x.d);
    if (x.tid == 0) {
        sx = 0; sy = 0; cnt = 0;
        for (int w = 0; w < NW; w++) { sx += s.r64[w][0]; sy += s.r64[w][1]; cnt += s.r64[w][2]; }
        if (cnt == 0) { s.gx = 2 * mode[0]; s.gy = 2 * mode[1]; }
        else {
            const long long ssx = (sx > 0) - (sx < 0), ssy = (sy > 0) - (sy < 0);
            s.gx = 2 * (int)((sx + ssx * cnt / 2) / cnt);
            s.gy = 2 * (int)((sy + ssy * cnt / 2) / cnt);
        }
    }
    dbar(x.d);
}

// reorder_search_order (:404-419): stable sort of the interior cells by score >> shift
// (`sorted`: the next level takes its order from this one's, as all but level 0 do)
__device__ void reorder(const Ctx &x, DirSh &s, const uint2 *field, int gw, int gh, DirScratch &ds, int *status, bool sorted) {
    const unsigned count = (unsigned)(gw - 1) * (unsigned)(gh - 1);
    if ((int64_t)count > s.order_len) {
        if (x.tid == 0) { atomicOr(status, ST_PANIC); s.abort_ = 1; }
        dbar(x.d);
        return;
    }
    if (!sorted) return;
    unsigned v = (unsigned)imax(x.P->block_w * x.P->block_h / 8, 1), lg = 0;
    while (v >>= 1) lg++;
    const unsigned shift = lg + 1;
    int lgn = 5;
    while ((1u << lgn) < count) lgn++;
    const unsigned np = 1u << lgn;
    unsigned long long *keys = ds.keys;
    for (unsigned i = (unsigned)x.tid; i < np; i += NT) {
        if (i < count) {
            const unsigned xx = i % (unsigned)(gw - 1), yy = i / (unsigned)(gw - 1);
            keys[i] = ((unsigned long long)(field[yy * (unsigned)gw + xx].y >> shift) << 32) | (unsigned long long)i;
        } else {
            keys[i] = ~0ull;
        }
    }
    dbar(x.d);
    // Bitonic sort: the steps between keys 32 and more apart in memory, those within 32 in a warp's
    // registers, one pass for a stage's five (2048 keys: 27 passes with barriers between in place of 66).
    const int lane = x.tid & 31;
    for (int stage = 5; stage <= lgn; stage++) {  // the first sorts runs of 32 outright
        for (int lj = stage - 1; lj >= 5; lj--) {
            const unsigned j = 1u << lj;
            for (unsigned i = (unsigned)x.tid; i < np / 2; i += NT) {
                const unsigned lo = ((i >> lj) << (lj + 1)) | (i & (j - 1)), hi = lo + j;
                const unsigned long long a = keys[lo], b = keys[hi];
                if ((a > b) == (((lo >> stage) & 1u) == 0)) { keys[lo] = b; keys[hi] = a; }
            }
            dbar(x.d);
        }
        for (unsigned i = (unsigned)x.tid; i < np; i += NT) {
            unsigned long long k = keys[i];
            for (int st = stage == 5 ? 1 : stage; st <= stage; st++)
                for (int lj = imin(st, 5) - 1; lj >= 0; lj--) {
                    const unsigned long long o = __shfl_xor_sync(kFull, k, 1 << lj);
                    const bool up = ((i >> st) & 1u) == 0, low = ((lane >> lj) & 1) == 0;
                    if ((up == low) == (o < k)) k = o;
                }
            keys[i] = k;
        }
        dbar(x.d);
    }
    for (unsigned i = (unsigned)x.tid; i < count; i += NT) {
        const unsigned r = (unsigned)(keys[i] & 0xFFFFFFFFull);
        ds.order[i] = pack_xy((int)(r % (unsigned)(gw - 1)), (int)(r / (unsigned)(gw - 1)));
    }
    dbar(x.d);
}

// refine_search_order (:338-402): the children of the coarser level's sw x sh interior cells, in the order of
// those (a permutation of them after reorder), inner cells of the grid first, then the cells on its inner
// border, then its last row and column. Every cell of the dw x dh interior is the child of exactly one
// coarse cell (those past twice the coarse grid, of the last column or row), so the places are two sums
// over the coarse cells: each thread counts and then writes a run of them. What ran before the search of
// a 1080p pair's second level was bound by one thread's chain through a mask of the cells seen, 0.55 ms;
// it takes 0.10 so, with the sort above in fewer passes.
__device__ void refine_order(const Ctx &x, DirSh &s, DirScratch &ds, int sw, int sh, int gw, int gh) {
    const int dw = gw - 1, dh = gh - 1;
    const int ex = imax(dw - 2 * sw, 0), ey = imax(dh - 2 * sh, 0);
    const int n = sw > 0 && sh > 0 ? sw * sh : 0, run = (n + NT - 1) / NT;
    const int first = imin(x.tid * run, n), last = imin(first + run, n);
    const int lane = x.tid & 31;
    uint32_t *to = ds.order2;
    auto children = [&](int2 c, auto add) {
        const int left = 2 * c.x, top = 2 * c.y;
        auto one = [&](int cx, int cy) {
            if (cx < dw && cy < dh) add(cx, cy, cx > 0 && cy > 0 && cx < dw - 1 && cy < dh - 1);
        };
        one(left, top); one(left + 1, top); one(left + 1, top + 1); one(left, top + 1);
        if (c.x == sw - 1)
            for (int dx = 2; dx < 2 + ex; dx++)
                for (int dy = 0; dy < 2 + (c.y == sh - 1) * ey; dy++) one(left + dx, top + dy);
        if (c.y == sh - 1)
            for (int dy = 2; dy < 2 + ey; dy++)
                for (int dx = 0; dx < 2; dx++) one(left + dx, top + dy);
    };
    int inner = 0, border = 0;
    for (int k = first; k < last; k++) children(unpack_xy(ds.order[k]), [&](int, int, bool in) { inner += in; border += !in; });
    long long mine = ((long long)border << 32) | inner, sum = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long v = __shfl_up_sync(kFull, sum, o);
        if (lane >= o) sum += v;
    }
    if (lane == 31) s.r64[x.tid >> 5][0] = sum;
    dbar(x.d);
    long long before = sum - mine, total = 0;
    for (int w = 0; w < NW; w++) {
        if (w < (x.tid >> 5)) before += s.r64[w][0];
        total += s.r64[w][0];
    }
    const int ninner = (int)total, nborder = (int)(total >> 32);
    int pi = (int)before, pb = ninner + (int)(before >> 32);
    for (int k = first; k < last; k++)
        children(unpack_xy(ds.order[k]), [&](int cx, int cy, bool in) { to[in ? pi++ : pb++] = pack_xy(cx, cy); });
    const int base = ninner + nborder;
    for (int k = x.tid; k <= dw + dh; k += NT) to[base + k] = k <= dw ? pack_xy(k, dh) : pack_xy(dw, k - dw - 1);
    const int len = base + dw + 1 + dh;
    dbar(x.d);
    if (x.tid == 0) s.order_len = len;
    for (int k = x.tid; k < len; k += NT) ds.order[k] = to[k];
}

__device__ __forceinline__ DirScratch dir_scratch(const AnalyseParams &P, uint8_t *scr, int d) {
    DirScratch ds;
    ds.vec[0] = (uint2 *)(scr + P.off_field[d]);
    ds.vec[1] = (uint2 *)(scr + P.off_next[d]);
    ds.luma[0] = scr + P.off_out[d];
    ds.luma[1] = scr + P.off_out[d] + P.max_cells;
    ds.proj[0] = (uint2 *)(scr + P.off_proj[d][0]);
    ds.proj[1] = (uint2 *)(scr + P.off_proj[d][1]);
    ds.order = (uint32_t *)(scr + P.off_order[d]);
    ds.order2 = (uint32_t *)(scr + P.off_order2[d]);
    ds.pos = (int *)(scr + P.off_pos[d]);
    ds.keys = (unsigned long long *)(scr + P.off_keys[d]);
    ds.hist = (unsigned *)(scr + P.off_hist[d]);
    return ds;
}

// The per-level fields of the search context, and the warp's group tables.
__device__ __forceinline__ void set_level(Ctx &x, const AnalyseParams &P, int level) {
    const LevelInfo &L = P.lv[level];
    x.L = &L;
    x.level = level;
    x.satd = L.satd;
    x.pel = L.pel;
    set_geo(x.G, P, L);
    x.pnew = P.pnew;
    set_groups(x);
}

// Pair b of a launch (analyse_filter.rs:277-282: frame n pairs with min(n + delta, num_frames - 1)).
__device__ __forceinline__ PairRef pair_at(const PairSrc &psrc, int64_t pair) {
    if (psrc.table) return psrc.table[pair];
    const int64_t n = (int64_t)psrc.first + pair;
    int64_t n2 = n + psrc.delta;
    if (n2 > psrc.nframes - 1) n2 = psrc.nframes - 1;
    PairRef pr;
    pr.cur = psrc.clip + n * psrc.frame_bytes;
    pr.ref = psrc.clip + n2 * psrc.frame_bytes;
    return pr;
}

// One frame pair, both directions: the whole of analyse_pair (:68-226) plus the payload
// (:2740-2811). Called by every thread of the CTA; threads of a direction the
// configuration does not search (vectors 1 or 2 under a 2-direction batch CTA) only
// take part in the CTA-wide barriers. Status bits go to *status.
// Levels hi .. lo: the whole hierarchy in one call (split false), or the part between two walks:
// what follows the search of level hi + 1 (global predictor, order) unless hi is the first level, the
// levels above lo whole, and level lo up to its search, which the walk kernel does (see CTL_GO);
// a level that the walk may not take is searched here.
__device__ __forceinline__ void analyse_pair_dev(const AnalyseParams &P, const PairRef pr, uint8_t *__restrict__ pay,
                                                 uint8_t *__restrict__ scr, int *status, int &cta_abort,
                                                 unsigned long long *spec_stats, bool split, int hi, int lo, int groups) {
    extern __shared__ __align__(16) unsigned char smem[];
    const bool bidir = P.vectors == 3;
    const int half = (int)(threadIdx.x / NT);
    const bool idle = !bidir && half == 1;
    const int d = bidir ? half : ((P.vectors & 2) ? 0 : 1);  // 0 = forward (cur -> ref), 1 = backward
    const int tid = threadIdx.x % NT;
    DirSh &s = reinterpret_cast<DirSh *>(smem)[half];
    const px_t *src = (const px_t *)(d == 0 ? pr.cur : pr.ref);
    const px_t *ref = (const px_t *)(d == 0 ? pr.ref : pr.cur);
    DirScratch ds = dir_scratch(P, scr, d);
    int *ctl = (int *)(scr + P.off_ctl[d]);
    Ctx x;
    x.P = &P;
    x.d = half;
    x.tid = tid;
    x.nw = NW;
    x.wbase = 0;
    unsigned char *area = smem + sizeof(DirSh) * (blockDim.x / NT) + (size_t)half * NW * groups * kGroupBytes;
    set_stage(x, area, groups, 0, tid >> 5);
    set_frames(x, P, src, ref);
    if (threadIdx.x == 0) cta_abort = 0;
    const bool resume = hi < P.nlevels - 1;
    if (tid == 0) {
        s.abort_ = 0; s.gx = 0; s.gy = 0; s.order_len = 0;
        if (idle) s.abort_ = 2;
        else if (resume) {
            s.abort_ = ctl[CTL_ABORT]; s.gx = ctl[CTL_GX]; s.gy = ctl[CTL_GY]; s.order_len = ctl[CTL_ORDER];
            ctl[CTL_GO] = 0;
        } else { ctl[CTL_GO] = 0; ctl[CTL_ABORT] = 0; }
    }
    __syncthreads();
    const uint2 *other_proj[2] = {nullptr, nullptr};
    {
        const int od = bidir ? 1 - d : d;
        other_proj[0] = (const uint2 *)(scr + P.off_proj[od][0]);
        other_proj[1] = (const uint2 *)(scr + P.off_proj[od][1]);
    }
    int pgw = 0, pgh = 0;  // grid of the previous (coarser) level
    auto after_search = [&](int level) {
        const LevelInfo &L = P.lv[level];
        const uint2 *f = ds.vec[level & 1];
        global_doubled(x, s, f, (int64_t)L.gw * L.gh, ds.hist);
        reorder(x, s, f, L.gw, L.gh, ds, status, level > 1);
    };
    if (resume) {
        pgw = P.lv[hi + 1].gw; pgh = P.lv[hi + 1].gh;
        if (!s.abort_) after_search(hi + 1);
    }
    for (int level = hi; level >= lo; level--) {
        const LevelInfo &L = P.lv[level];
        set_level(x, P, level);
        const int gw = L.gw, gh = L.gh;
        const int64_t ncell = (int64_t)gw * gh;
        const bool first = level == P.nlevels - 1;
        if (!s.abort_) {
            // ---- search order of this level
            if (level == 0) {
                if (tid == 0) s.order_len = (int)initial_order_len(gw, gh);
            } else if (first) {
                const int64_t n0 = initial_order_len(gw - 1, gh - 1) + gw + (gh - 1);
                for (int64_t k = tid; k < n0; k += NT) {
                    const int2 b = level_order_at(gw, gh, k);
                    ds.order[k] = pack_xy(b.x, b.y);
                }
                if (tid == 0) s.order_len = (int)n0;
            } else {
                refine_order(x, s, ds, pgw - 1, pgh - 1, gw, gh);
            }
            dbar(half);
            if (level > 0) {  // first position of every cell in the order ("processed" test)
                for (int64_t i = tid; i < ncell; i += NT) ds.pos[i] = 0x7FFFFFFF;
                dbar(half);
                for (int64_t k = tid; k < s.order_len; k += NT) {
                    const int2 c = unpack_xy(ds.order[k]);
                    atomicMin(&ds.pos[(int64_t)c.y * gw + c.x], (int)k);
                }
            }
            // ---- interpolate the coarser field (:421-478), or start from zeros
            uint2 *nf = ds.vec[level & 1];
            uint8_t *nl = ds.luma[level & 1];
            uint2 *pj = ds.proj[level & 1];
            if (first) {
                for (unsigned i = (unsigned)tid; i < (unsigned)ncell; i += NT) { nf[i] = make_uint2(0, 0); nl[i] = 0; }
            } else {
                const uint2 *cf = ds.vec[(level + 1) & 1];
                const uint8_t *cl = ds.luma[(level + 1) & 1];
                const int cw = pgw - 1, ch = pgh - 1, pel = L.pel;
                for (unsigned i = (unsigned)tid; i < (unsigned)ncell; i += NT) {
                    const int xx = (int)(i % (unsigned)gw), yy = (int)(i / (unsigned)gw);
                    uint2 out = make_uint2(0, 0);
                    uint8_t ol = 0;
                    if (xx < gw - 1 && yy < gh - 1) {
                        int64_t ci;
                        if (xx < 2 * cw && yy < 2 * ch) ci = (int64_t)(yy >> 1) * pgw + (xx >> 1);
                        else {
                            const int e = ch + imin(xx >> 1, cw) - imin(yy >> 1, ch);
                            ci = e <= cw ? (int64_t)ch * pgw + e : (int64_t)(cw + ch - e) * pgw + cw;
                        }
                        const uint2 p = cf[ci];
                        const int2 pm = vmv(p);
                        out = mkvec(iclamp(pm.x * 2 * pel, -32768, 32767), iclamp(pm.y * 2 * pel, -32768, 32767), p.y);
                        ol = cl[ci];
                    }
                    nf[i] = out;
                    nl[i] = ol;
                    ds.keys[i] = ~0ull;
                }
                dbar(half);
                for (unsigned i = (unsigned)tid; i < (unsigned)ncell; i += NT) {
                    const int xx = (int)(i % (unsigned)gw), yy = (int)(i / (unsigned)gw);
                    if (xx >= gw - 1 || yy >= gh - 1 || xx >= 2 * cw || yy >= 2 * ch) continue;
                    const uint2 p = cf[(int64_t)(yy >> 1) * pgw + (xx >> 1)];
                    if (p.y == 0xFFFFFFFFu) continue;  // `score < target.score` never holds
                    const int2 pm = vmv(p);
                    const int vx = pm.x * 2 * pel, vy = pm.y * 2 * pel;
                    const int bw = P.block_w, bh = P.block_h;
                    const int tx = iclamp((vx + (bw >> 1) + (bw - P.ox) * xx) / (bw - P.ox), 0, gw - 1);
                    const int ty = iclamp((vy + (bh >> 1) + (bh - P.oy) * yy) / (bh - P.oy), 0, gh - 1);
                    atomicMin(&ds.keys[(int64_t)ty * gw + tx], ((unsigned long long)p.y << 32) | (unsigned long long)i);
                }
                dbar(half);
                for (unsigned i = (unsigned)tid; i < (unsigned)ncell; i += NT) {
                    const unsigned long long kk = ds.keys[i];
                    if (kk == ~0ull) pj[i] = make_uint2(0, 0xFFFFFFFFu);
                    else {
                        const uint2 v = nf[kk & 0xFFFFFFFFull];
                        const int2 m = vmv(v);
                        pj[i] = mkvec(-m.x, -m.y, v.y);
                    }
                }
            }
        }
        __syncthreads();  // both directions' projections of this level are ready
        if (!s.abort_) {
            const uint2 *prevp = (first) ? nullptr : other_proj[level & 1];
            const bool leave = split && level == lo;
            const bool walk = SVPF_LOOKAHEAD && NW > 1 && (leave || (!split && (P.lookahead & (level == 0 ? 1 : 2))));
            if (walk && level_spec_ok(x, s, ds)) {
                if (leave) {  // the walk kernel's
                    start_walk(x, ds, ctl, (int)ncell);
                    if (tid == 0) { ctl[CTL_PREV] = prevp != nullptr; ctl[CTL_GO] = 1; }
                } else {
                    walk_in_cta(x, s, ds, prevp, ctl, status, spec_stats, area, groups);
                }
            } else {
                search_level(x, s, ds, prevp, status);
            }
        }
        dbar(half);
        if (!s.abort_ && level > 0 && !(split && level == lo)) after_search(level);
        pgw = gw; pgh = gh;
        if (tid == 0 && s.abort_ == 1) cta_abort = 1;
        __syncthreads();
    }
    if (split && tid == 0 && !idle) {
        ctl[CTL_GX] = s.gx; ctl[CTL_GY] = s.gy; ctl[CTL_ORDER] = s.order_len;
        if (s.abort_ == 1) ctl[CTL_ABORT] = 1;
    }
}

// rescale_scores (:2716-2738) + pack_vector_frame (:2740-2811) of one direction's cells first, first +
// step, ...; the thread with `head` also writes the payload's header and the direction's.
__device__ __forceinline__ void pack_cells(const AnalyseParams &P, const DirScratch &ds, int d, uint8_t *pay, int64_t first,
                                           int64_t step, bool head) {
    const bool bidir = P.vectors == 3;
    const uint2 *f = ds.vec[P.has_refine ? 1 : 0];
    const uint8_t *fl = ds.luma[P.has_refine ? 1 : 0];
    const int64_t count = (int64_t)P.out_gw * P.out_gh;
    const int64_t region = bidir ? (d == 1 ? 0x40 : 0x40 + 4 + count * 8) : 0x40;
    if (head) {
        if (!bidir || d == 0)
            for (int i = 0; i < 16; i++) reinterpret_cast<int *>(pay)[i] = P.header[i];
        *reinterpret_cast<int *>(pay + region) = (int)(2 * count + 1);
    }
    for (int64_t i = first; i < count; i += step) {
        const uint2 v = f[i];
        const int2 m = vmv(v);
        const int mag = abs(m.x) + abs(m.y);
        const int ratio = (100 * mag) / P.rescale_denom;
        int score = (int)v.y;
        if (ratio >= 51) score = sat_i32((long long)score * 20);
        else if (ratio >= 16) {
            const unsigned long long v71 = (3926827243ull * (unsigned long long)(unsigned)score * (unsigned long long)(unsigned)(ratio - 15)) >> 32;
            const int w = (int)(unsigned)v71;
            score = sat_i32((long long)score + 9 * ((w >> 31) + (w >> 5)));
        }
        const unsigned sc = (unsigned)score & 0x00FFFFFFu;
        uint8_t *o = pay + region + 4 + i * 8;
        const unsigned d0 = ((unsigned)(int)m.x << 16) | (unsigned)(uint16_t)(short)m.y;
        const unsigned d1 = sc | ((unsigned)fl[i] << 24);
        memcpy(o, &d0, 4);
        memcpy(o + 4, &d1, 4);
    }
}

// A one-warp context at the refine pass's level.
__device__ __forceinline__ void refine_ctx(Ctx &x, const AnalyseParams &P, const PairRef pr, int d) {
    const px_t *src = (const px_t *)(d == 0 ? pr.cur : pr.ref);
    const px_t *ref = (const px_t *)(d == 0 ? pr.ref : pr.cur);
    x.P = &P;
    x.tid = (int)(threadIdx.x & 31);
    x.nw = 1;
    set_frames(x, P, src, ref);
    x.level = 0;
    x.pel = P.lv[0].pel;
    x.satd = P.refine_satd;
    set_geo(x.G, P, P.lv[0]);
}

// After the hierarchy in one CTA: the refine pass when configured, then the payload. Out of line,
// called where little else is live, so neither adds to the hierarchy's register pressure. Every
// thread of the CTA calls it.
__device__ __noinline__ void finish_pair(const AnalyseParams *Pp, const PairRef pr, uint8_t *pay, uint8_t *scr, int groups) {
    extern __shared__ __align__(16) unsigned char smem[];
    const AnalyseParams &P = *Pp;
    const bool bidir = P.vectors == 3;
    const int half = (int)(threadIdx.x / NT);
    if (!bidir && half == 1) return;
    const int d = bidir ? half : ((P.vectors & 2) ? 0 : 1);
    const int tid = threadIdx.x % NT;
    DirSh &s = reinterpret_cast<DirSh *>(smem)[half];
    DirScratch ds = dir_scratch(P, scr, d);
    if (P.has_refine) {
        Ctx x;
        refine_ctx(x, P, pr, d);
        x.d = half;
        x.wbase = tid >> 5;
        set_stage(x, smem + sizeof(DirSh) * (blockDim.x / NT) + (size_t)half * NW * groups * kGroupBytes, groups, x.wbase,
                  x.wbase);
        int shape = -1;
        const int n = P.out_gw * P.out_gh;
        for (int i = x.wbase; i < n; i += NW) refine_block(x, s, ds, i % P.out_gw, i / P.out_gw, shape);
        dbar(half);
    }
    pack_cells(P, ds, d, pay, tid, NT, tid == 0);
}

// One CTA per frame pair: the whole pair, or (split) the levels hi .. lo between two walks.
__global__ void __launch_bounds__(2 * NT, SVPF_MINB)
    analyse_kernel(const __grid_constant__ AnalyseParams P, const PairSrc psrc, uint8_t *__restrict__ payloads,
                   uint8_t *__restrict__ scratch, int *status, int split, int hi, int lo) {
    __shared__ int cta_abort;
    const int64_t pair = blockIdx.x;
    const PairRef pr = pair_at(psrc, pair);
    uint8_t *scr = scratch + pair * P.scratch_per_pair;
    analyse_pair_dev(P, pr, payloads + pair * P.payload_len, scr, status, cta_abort, psrc.stats, split != 0, hi, lo,
                     P.stage_groups);
    __syncthreads();
    if (!split && !cta_abort) finish_pair(&P, pr, payloads + pair * P.payload_len, scr, P.stage_groups);
}

#if SVPF_LOOKAHEAD
// One level spread over the GPU: a CTA per warp, D of them per search direction of the pairs first ..
// of the launch. The warps of a direction wait on one another, so the launch is cooperative: all its
// CTAs are resident at once, or it does not start.
// PER_SM: CTAs per SM the registers are cut for, 16 (128 per thread) or 20 (96; more spills, but a quarter
// more warps). Few pairs leave the chain of blocks as the bound, where the first is faster (32 frames of
// 640x360 3.69 against 3.96 ms, 16 of them at 10 bits 134 against 158, one 1080p pair 23.4 against 24.2), many
// pairs the latency of the loads, which more warps hide (240 frames of 1080p 800 against 731 ms; 24 CTAs with 80
// registers were slower than 20): the line is where the first could give a direction kDenseWalkers warps.
constexpr int kWalkPerSM = 16, kDensePerSM = 20, kDenseWalkers = 8;
__device__ __forceinline__ void walk_cta(const AnalyseParams &P, const PairRef pr, uint8_t *scr, int dir, int g, int D, int level,
                                         int groups, int *status, unsigned long long *stats) {
    __shared__ WarpSh s;
    extern __shared__ __align__(16) unsigned char stage[];
    const int ndir = P.vectors == 3 ? 2 : 1;
    if (dir >= ndir) return;
    const int d = ndir == 2 ? dir : ((P.vectors & 2) ? 0 : 1);
    int *ctl = (int *)(scr + P.off_ctl[d]);
    if (!ctl[CTL_GO]) return;  // the pair kernel searched the level itself, or the direction stopped
    const DirScratch ds = dir_scratch(P, scr, d);
    Ctx x;
    x.P = &P;
    x.d = 0;
    x.tid = (int)threadIdx.x;
    x.nw = 1;
    x.wbase = 0;
    set_frames(x, P, (const px_t *)(d == 0 ? pr.cur : pr.ref), (const px_t *)(d == 0 ? pr.ref : pr.cur));
    set_stage(x, stage, groups, 0, 0);
    set_level(x, P, level);
    const int od = ndir == 2 ? 1 - d : d;
    const uint2 *prevp = ctl[CTL_PREV] ? (const uint2 *)(scr + P.off_proj[od][level & 1]) : nullptr;
    walk_level(x, s, ds, prevp, g, D, ctl[CTL_ORDER], ctl[CTL_GX], ctl[CTL_GY], ctl, status, stats);
}
template <int PER_SM>
__global__ void __launch_bounds__(32, PER_SM)
    analyse_walk_kernel(const __grid_constant__ AnalyseParams P, const PairSrc psrc, int64_t first, int level, int D,
                        uint8_t *__restrict__ scratch, int *status) {
    const int ndir = P.vectors == 3 ? 2 : 1;
    const int64_t pair = first + blockIdx.x / (ndir * D);
    const int rem = (int)(blockIdx.x % (ndir * D));
    walk_cta(P, pair_at(psrc, pair), scratch + pair * P.scratch_per_pair, rem / D, rem % D, D, level, P.stage_groups, status,
             psrc.stats);
}

// Neither direction of a pair stopped.
__device__ __forceinline__ bool pair_whole(const AnalyseParams &P, const uint8_t *scr) {
    const bool bidir = P.vectors == 3;
    const int d0 = bidir ? 0 : ((P.vectors & 2) ? 0 : 1);
    return !((const int *)(scr + P.off_ctl[d0]))[CTL_ABORT] && !(bidir && ((const int *)(scr + P.off_ctl[1]))[CTL_ABORT]);
}

// The refine pass of a split launch: its blocks are independent, so they go to `per_dir` one-warp
// CTAs per direction, every per_dir-th block to each.
__device__ __forceinline__ void refine_cta(const AnalyseParams &P, const PairRef pr, uint8_t *scr, int dir, int g, int per_dir,
                                           int groups) {
    __shared__ WarpSh s;
    extern __shared__ __align__(16) unsigned char stage[];
    const int ndir = P.vectors == 3 ? 2 : 1;
    if (dir >= ndir || !pair_whole(P, scr)) return;
    const int d = ndir == 2 ? dir : ((P.vectors & 2) ? 0 : 1);
    DirScratch ds = dir_scratch(P, scr, d);
    Ctx x;
    refine_ctx(x, P, pr, d);
    x.d = 0;
    x.wbase = 0;
    set_stage(x, stage, groups, 0, 0);
    int shape = -1;
    const int n = P.out_gw * P.out_gh;
    for (int i = g; i < n; i += per_dir) refine_block(x, s, ds, i % P.out_gw, i / P.out_gw, shape);
}
__global__ void __launch_bounds__(32, kWalkPerSM)
    analyse_refine_kernel(const __grid_constant__ AnalyseParams P, const PairSrc psrc, int per_dir, uint8_t *__restrict__ scratch) {
    const int ndir = P.vectors == 3 ? 2 : 1;
    const int64_t pair = blockIdx.x / (ndir * per_dir);
    const int rem = (int)(blockIdx.x % (ndir * per_dir));
    refine_cta(P, pair_at(psrc, pair), scratch + pair * P.scratch_per_pair, rem / per_dir, rem % per_dir, per_dir, P.stage_groups);
}

// The payloads of a split launch: kPackThreads cells of one direction per CTA.
constexpr int kPackThreads = 256;
__global__ void __launch_bounds__(kPackThreads)
    analyse_pack_kernel(const __grid_constant__ AnalyseParams P, uint8_t *__restrict__ payloads, uint8_t *__restrict__ scratch) {
    const int64_t pair = blockIdx.y;
    const int d = P.vectors == 3 ? (int)blockIdx.z : ((P.vectors & 2) ? 0 : 1);
    uint8_t *scr = scratch + pair * P.scratch_per_pair;
    if (!pair_whole(P, scr)) return;
    const DirScratch ds = dir_scratch(P, scr, d);
    const int64_t i = (int64_t)blockIdx.x * kPackThreads + threadIdx.x;
    pack_cells(P, ds, d, payloads + pair * P.payload_len, i, (int64_t)gridDim.x * kPackThreads, i == 0);
}

// Levels of fewer blocks than this are searched by the pair's CTA, without a launch of their own: the least
// that a walk takes, 3 x 3. (32 frames of 640x360, lines at 9, 30 and 120 blocks: 3.50, 3.69 and 4.45 ms; one
// 1080p pair 23.2, 23.4 and 25.0.)
constexpr int kWalkCells = 9;

// The coarsest level of P that a walk takes; the levels above it are the pair kernel's.
__host__ __device__ inline int first_walk(const AnalyseParams &P) {
    int lo = P.nlevels - 1;
    while (lo > 0 && P.lv[lo].gw * P.lv[lo].gh < kWalkCells) lo--;
    return lo;
}
#endif

// Persistent form: a grid sized to the resident CTAs drains the item list in order (the
// host sorts it largest-first); each CTA pulls the next item with one atomic, copies the
// item's clip parameters into shared memory and runs the pair on its own scratch slot.
__global__ void __launch_bounds__(2 * NT, SVPF_MINB)
    analyse_batch_kernel(const AnalyseParams *__restrict__ clips, const BatchItem *__restrict__ items, int nitems,
                         unsigned *__restrict__ next_item, uint8_t *__restrict__ scratch, int64_t scratch_per_cta,
                         int *__restrict__ clip_status, int groups) {
    __shared__ int cta_abort;
    __shared__ int item_sh;
    __shared__ __align__(16) AnalyseParams P;
    uint8_t *scr = scratch + (int64_t)blockIdx.x * scratch_per_cta;
    for (;;) {
        if (threadIdx.x == 0) item_sh = (int)atomicAdd(next_item, 1u);
        __syncthreads();
        const int it = item_sh;
        if (it >= nitems) break;
        const BatchItem bi = items[it];
        {
            const int4 *src = reinterpret_cast<const int4 *>(clips + bi.clip);
            int4 *dst = reinterpret_cast<int4 *>(&P);
            for (int i = threadIdx.x; i < (int)(sizeof(AnalyseParams) / 16); i += blockDim.x) dst[i] = src[i];
        }
        __syncthreads();
        analyse_pair_dev(P, bi.pair, bi.payload, scr, clip_status + bi.clip, cta_abort, nullptr, false, P.nlevels - 1, 0, groups);
        __syncthreads();
        if (!cta_abort) finish_pair(&P, bi.pair, bi.payload, scr, groups);
        __syncthreads();  // P, item_sh and the shared search state are reused by the next item
    }
}

#if SVPF_LOOKAHEAD && !defined(SVPF_PX16)
// The batch form of the split launch: every item of a group of items (one scratch slot each) goes level
// by level, the clips' finest levels aligned: `lo` is the level of this round, and an item whose clip has
// its first walk at a finer level waits. Between two walks:
__global__ void __launch_bounds__(2 * NT, SVPF_MINB)
    batch_ground_kernel(const AnalyseParams *__restrict__ clips, const BatchItem *__restrict__ items, int lo,
                        uint8_t *__restrict__ scratch, int64_t scratch_per_slot, int *__restrict__ clip_status, int groups) {
    __shared__ int cta_abort;
    __shared__ __align__(16) AnalyseParams P;
    const BatchItem bi = items[blockIdx.x];
    {
        const int4 *src = reinterpret_cast<const int4 *>(clips + bi.clip);
        int4 *dst = reinterpret_cast<int4 *>(&P);
        for (int i = threadIdx.x; i < (int)(sizeof(AnalyseParams) / 16); i += blockDim.x) dst[i] = src[i];
    }
    __syncthreads();
    const int start = first_walk(P);
    if (lo > start) return;
    analyse_pair_dev(P, bi.pair, bi.payload, scratch + (int64_t)blockIdx.x * scratch_per_slot, clip_status + bi.clip, cta_abort,
                     nullptr, true, lo == start ? P.nlevels - 1 : lo, lo, groups);
}
// The walks of a round: 2 D one-warp CTAs per item (see analyse_walk_kernel).
template <int PER_SM>
__global__ void __launch_bounds__(32, PER_SM)
    batch_walk_kernel(const AnalyseParams *__restrict__ clips, const BatchItem *__restrict__ items, int lo, int D,
                      uint8_t *__restrict__ scratch, int64_t scratch_per_slot, int *__restrict__ clip_status, int groups) {
    const int slot = blockIdx.x / (2 * D), rem = blockIdx.x % (2 * D);
    const BatchItem bi = items[slot];
    const AnalyseParams &P = clips[bi.clip];
    if (lo > first_walk(P)) return;
    walk_cta(P, bi.pair, scratch + (int64_t)slot * scratch_per_slot, rem / D, rem % D, D, lo, groups, clip_status + bi.clip, nullptr);
}
__global__ void __launch_bounds__(32, kWalkPerSM)
    batch_refine_kernel(const AnalyseParams *__restrict__ clips, const BatchItem *__restrict__ items, int per_dir,
                        uint8_t *__restrict__ scratch, int64_t scratch_per_slot, int groups) {
    const int slot = blockIdx.x / (2 * per_dir), rem = blockIdx.x % (2 * per_dir);
    const BatchItem bi = items[slot];
    const AnalyseParams &P = clips[bi.clip];
    if (P.has_refine) refine_cta(P, bi.pair, scratch + (int64_t)slot * scratch_per_slot, rem / per_dir, rem % per_dir, per_dir, groups);
}
__global__ void __launch_bounds__(kPackThreads)
    batch_pack_kernel(const AnalyseParams *__restrict__ clips, const BatchItem *__restrict__ items, uint8_t *__restrict__ scratch,
                      int64_t scratch_per_slot) {
    const int slot = blockIdx.y;
    const BatchItem bi = items[slot];
    const AnalyseParams &P = clips[bi.clip];
    if ((int)blockIdx.z >= (P.vectors == 3 ? 2 : 1)) return;
    const int d = P.vectors == 3 ? (int)blockIdx.z : ((P.vectors & 2) ? 0 : 1);
    uint8_t *scr = scratch + (int64_t)slot * scratch_per_slot;
    if (!pair_whole(P, scr)) return;
    const int64_t i = (int64_t)blockIdx.x * kPackThreads + threadIdx.x;
    pack_cells(P, dir_scratch(P, scr, d), d, bi.payload, i, (int64_t)gridDim.x * kPackThreads, i == 0);
}
#endif

}  // namespace

// Dynamic shared memory of a pair CTA of `ndir` directions.
size_t pair_shared(int ndir, int groups) { return (size_t)ndir * (sizeof(DirSh) + (size_t)NW * groups * kGroupBytes); }

// The kernels' shared-memory limits. They are raised once, to the most groups a supported block
// can have; each launch asks for its own configuration's bytes.
cudaError_t prepare() {
    static cudaError_t once = [] {
        const int smem = (int)pair_shared(2, kMaxStageGroups);
        cudaError_t e = cudaFuncSetAttribute(analyse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(analyse_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        return e;
    }();
    return once;
}

#if SVPF_LOOKAHEAD
namespace {
constexpr int kMinWalkers = 4;  // warps per direction of a walk, at least
// The build of a walk over `ndirs` search directions, its shared memory and how many CTAs of that very kernel are
// resident at once: the plain and the batch's kernels need not have the same registers.
template <class KERNEL>
struct WalkShape {
    KERNEL kernel;
    bool dense;
    size_t smem;
    int64_t resident;
};
template <class KERNEL>
cudaError_t walk_shape(KERNEL sparse, KERNEL dense, int groups, int64_t ndirs, WalkShape<KERNEL> &w) {
    w.smem = (size_t)groups * kGroupBytes;
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaError_t e = cudaGetDevice(&dev)) return e;
    if (cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) return e;
    if (cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sparse, 32, w.smem)) return e;
    w.dense = (int64_t)sms * per_sm < ndirs * kDenseWalkers;
    w.kernel = w.dense ? dense : sparse;
    if (w.dense)
        if (cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dense, 32, w.smem)) return e;
    w.resident = (int64_t)sms * per_sm;
    return cudaSuccess;
}
// The CTAs of a walk wait on one another, so the launch is cooperative and takes the directions whose
// CTAs are all resident at once.
template <class KERNEL, class... A>
cudaError_t launch_walk(const WalkShape<KERNEL> &w, int64_t ctas, cudaStream_t stream, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(32);
    cfg.dynamicSmemBytes = w.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, w.kernel, args...);
}
}  // namespace
#endif

cudaError_t launch_plain(const AnalyseParams &P, const PairSrc &psrc, int npairs, uint8_t *payloads, uint8_t *scratch,
                         int *status_dev, cudaStream_t stream, int *launches) {
    if (npairs <= 0) return cudaSuccess;
    if (cudaError_t e = prepare()) return e;
    const int ndir = P.vectors == 3 ? 2 : 1;
    const bool split = SVPF_LOOKAHEAD && (P.lookahead & 5) == 5;
    const size_t pair_smem = pair_shared(ndir, P.stage_groups);
    auto count = [&] { if (launches) *launches += 1; return cudaGetLastError(); };
    if (!split) {
        analyse_kernel<<<npairs, NT * ndir, pair_smem, stream>>>(P, psrc, payloads, scratch, status_dev, 0, P.nlevels - 1, 0);
        return count();
    }
#if SVPF_LOOKAHEAD
    // D warps per direction, as many as are resident at once (at least kMinWalkers, with the pairs in
    // several launches when they would not be)
    WalkShape<decltype(&analyse_walk_kernel<kWalkPerSM>)> w;
    if (cudaError_t e = walk_shape(analyse_walk_kernel<kWalkPerSM>, analyse_walk_kernel<kDensePerSM>, P.stage_groups,
                                   (int64_t)npairs * ndir, w))
        return e;
    const size_t stage = w.smem;
    const int64_t resident = w.resident;
    const int64_t most = resident / (ndir * kMinWalkers);
    if (most < 1) return cudaErrorCooperativeLaunchTooLarge;
    const int64_t walks = (npairs + most - 1) / most;
    const int64_t group = (npairs + walks - 1) / walks;  // even groups
    int64_t D = resident / (ndir * group);
    D = D < kMinWalkers ? kMinWalkers : D > kMaxWalkers ? kMaxWalkers : D;
    int hi = P.nlevels - 1, lo = first_walk(P);
    for (; lo >= 0; hi = lo - 1, lo = hi) {
        analyse_kernel<<<npairs, NT * ndir, pair_smem, stream>>>(P, psrc, payloads, scratch, status_dev, 1, hi, lo);
        if (cudaError_t e = count()) return e;
        for (int64_t f = 0; f < npairs; f += group) {
            const int64_t n = npairs - f < group ? npairs - f : group;
            if (cudaError_t e = launch_walk(w, n * ndir * D, stream, P, psrc, f, lo, (int)D, scratch, status_dev)) return e;
            if (launches) *launches += 1;
        }
    }
    const int cells = P.out_gw * P.out_gh;
    if (P.has_refine) {
        int64_t per_dir = (2 * resident + npairs * ndir - 1) / (npairs * ndir);  // about two waves
        if (per_dir > cells) per_dir = cells;
        analyse_refine_kernel<<<(unsigned)(npairs * ndir * per_dir), 32, stage, stream>>>(P, psrc, (int)per_dir, scratch);
        if (cudaError_t e = count()) return e;
    }
    for (int f = 0; f < npairs; f += 65535) {  // grid rows
        const int n = npairs - f < 65535 ? npairs - f : 65535;
        analyse_pack_kernel<<<dim3((cells + kPackThreads - 1) / kPackThreads, n, ndir), kPackThreads, 0, stream>>>(
            P, payloads + (int64_t)f * P.payload_len, scratch + (int64_t)f * P.scratch_per_pair);
        if (cudaError_t e = count()) return e;
    }
#endif
    return cudaSuccess;
}

cudaError_t batch_blocks_per_sm(const BatchInfo &info, int *blocks) {
    if (cudaError_t e = prepare()) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, analyse_batch_kernel, 2 * NT, pair_shared(2, info.groups));
}

cudaError_t launch_batch(const AnalyseParams *clips_dev, const BatchItem *items_dev, int nitems, unsigned *next_item_dev,
                         uint8_t *scratch, int64_t scratch_per_cta, int *clip_status_dev, const BatchInfo &info, int grid,
                         cudaStream_t stream, int *launches) {
    if (nitems <= 0 || grid <= 0) return cudaSuccess;
    if (cudaError_t e = prepare()) return e;
    analyse_batch_kernel<<<grid, 2 * NT, pair_shared(2, info.groups), stream>>>(clips_dev, items_dev, nitems, next_item_dev,
                                                                                scratch, scratch_per_cta, clip_status_dev,
                                                                                info.groups);
    if (launches) *launches += 1;
    return cudaGetLastError();
}

#if SVPF_LOOKAHEAD && !defined(SVPF_PX16)
// The batch walked level by level (batch_ground_kernel): `grid` pairs at a time.
int first_walk_level(const AnalyseParams &P) { return first_walk(P); }

using BatchWalkShape = WalkShape<decltype(&batch_walk_kernel<kWalkPerSM>)>;
cudaError_t batch_walk_shape(int groups, int64_t ndirs, BatchWalkShape &w) {
    return walk_shape(batch_walk_kernel<kWalkPerSM>, batch_walk_kernel<kDensePerSM>, groups, ndirs, w);
}

// Pairs of a group per SM: enough to fill the SMs with at least kMinWalkers warps per direction.
cudaError_t batch_walk_pairs_per_sm(const BatchInfo &info, int *pairs) {
    BatchWalkShape w;
    if (cudaError_t e = prepare()) return e;
    if (cudaError_t e = batch_walk_shape(info.groups, (int64_t)1 << 30, w)) return e;
    int dev = 0, sms = 0;
    if (cudaError_t e = cudaGetDevice(&dev)) return e;
    if (cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) return e;
    *pairs = (int)(w.resident / sms / (2 * kMinWalkers));
    return cudaSuccess;
}

cudaError_t launch_batch_walk(const AnalyseParams *clips_dev, const BatchItem *items_dev, int nitems, unsigned *,
                              uint8_t *scratch, int64_t scratch_per_slot, int *clip_status_dev, const BatchInfo &info,
                              int grid, cudaStream_t stream, int *launches) {
    if (nitems <= 0 || grid <= 0) return cudaSuccess;
    if (cudaError_t e = prepare()) return e;
    static const cudaError_t ground = cudaFuncSetAttribute(batch_ground_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                           (int)pair_shared(2, kMaxStageGroups));
    if (ground != cudaSuccess) return ground;
    auto count = [&] { if (launches) *launches += 1; return cudaGetLastError(); };
    const int ngroups = (nitems + grid - 1) / grid, group = (nitems + ngroups - 1) / ngroups;  // even groups
    BatchWalkShape w;
    if (cudaError_t e = batch_walk_shape(info.groups, (int64_t)group * 2, w)) return e;
    int64_t D = w.resident / (group * 2);
    if (D < 1) return cudaErrorCooperativeLaunchTooLarge;
    if (D > kMaxWalkers) D = kMaxWalkers;
    for (int f = 0; f < nitems; f += group) {
        const int n = nitems - f < group ? nitems - f : group;
        const BatchItem *it = items_dev + f;
        for (int lo = info.rounds - 1; lo >= 0; lo--) {
            batch_ground_kernel<<<n, 2 * NT, pair_shared(2, info.groups), stream>>>(clips_dev, it, lo, scratch, scratch_per_slot,
                                                                                    clip_status_dev, info.groups);
            if (cudaError_t e = count()) return e;
            if (cudaError_t e = launch_walk(w, n * 2 * D, stream, clips_dev, it, lo, (int)D, scratch, scratch_per_slot,
                                            clip_status_dev, info.groups))
                return e;
            if (launches) *launches += 1;
        }
        if (info.refine) {
            const int per_dir = (int)((2 * w.resident + 2 * n - 1) / (2 * n));
            batch_refine_kernel<<<n * 2 * per_dir, 32, w.smem, stream>>>(clips_dev, it, per_dir, scratch, scratch_per_slot, info.groups);
            if (cudaError_t e = count()) return e;
        }
        batch_pack_kernel<<<dim3((info.cells + kPackThreads - 1) / kPackThreads, n, 2), kPackThreads, 0, stream>>>(
            clips_dev, it, scratch, scratch_per_slot);
        if (cudaError_t e = count()) return e;
    }
    return cudaSuccess;
}
#endif

}  // namespace SVPF_VARIANT
}  // namespace svpf
