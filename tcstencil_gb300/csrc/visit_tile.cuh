// A tile of a plain FP16 grid stepped several times in shared memory: what the
// epilogue warps do with a step's accumulators (back into the staged image, or
// to the output plane), for the single-grid visits (sweep_visit.cu, which says
// how the image shrinks) and the batched ones (batch.cu).
#pragma once

#include <type_traits>

#include "tc_core.cuh"

namespace tcs {
namespace tc {

// 8 accumulators as a panel row of FP16 cells.
__device__ __forceinline__ uint4 pack_panel(const uint32_t *v) {
    uint32_t w[4];
#pragma unroll
    for (int c = 0; c < 4; c++) w[c] = pack_h2(__uint_as_float(v[2 * c]), __uint_as_float(v[2 * c + 1]));
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// Masks of a panel row's cells in shared memory, 16 bytes each: entry n is the
// cells c >= n (n = 0 .. 8), entry 9 + n the cells c < n.
constexpr int kMaskBytes = 18 * 16;
__device__ __forceinline__ void build_masks(uint32_t *mask, int tid) {
    if (tid < 72) {
        const int n = (tid / 4) % 9, c = 2 * (tid % 4);
        const uint32_t ge = (c >= n ? 0x0000ffffu : 0u) | (c + 1 >= n ? 0xffff0000u : 0u);
        mask[tid] = tid < 36 ? ge : ~ge;
    }
}
__device__ __forceinline__ uint4 blend(const uint4 &w, const uint4 &old, const uint4 &m) {
    return make_uint4((w.x & m.x) | (old.x & ~m.x), (w.y & m.y) | (old.y & ~m.y),
                      (w.z & m.z) | (old.z & ~m.z), (w.w & m.w) | (old.w & ~m.w));
}
// The mask of cells [a, b), 0 <= a, b <= 8 (none if b <= a).
__device__ __forceinline__ uint4 cells_mask(uint32_t mask, int a, int b) {
    const uint4 x = lds128(mask + 16 * a), y = lds128(mask + 16 * (9 + b));
    return make_uint4(x.x & y.x, x.y & y.y, x.z & y.z, x.w & y.w);
}
__device__ __forceinline__ int clamp8(int v) { return v < 0 ? 0 : v > 8 ? 8 : v; }

// This warp's G blocks of 16 columns of a step's accumulators, two blocks at
// a time: sink(p, w) takes panel row p = 0 .. 2G-1.  (A TMEM load takes about
// 25 cycles; holding all blocks at once would spill registers, which cost
// ten times that, as little L1 is left beside the stages.)
template <int G, typename Sink>
__device__ __forceinline__ void walk_blocks(uint32_t col, Sink &&sink) {
#pragma unroll
    for (int g = 0; g < G; g += 2) {
        uint32_t v[2][16];
        tmem_ld_x16(col + 16 * g, v[0]);
        if (g + 1 < G) tmem_ld_x16(col + 16 * (g + 1), v[1]);
        if (g + 1 < G) tmem_ld_wait(v);
        else tmem_ld_wait(v[0]);
#pragma unroll
        for (int p = 2 * g; p < 2 * g + 4 && p < 2 * G; p++)
            sink(p, pack_panel(v[(p >> 1) - g] + 8 * (p & 1)));
    }
}

// A tile's MMAs: the windows its grid cells need (tile_windows), rounded up
// to a sequence of 5 or of all.  (In a loop over the coefficient rows instead
// of unrolled, the issuing thread took 87 cycles per MMA instead of 67.)
template <int R, int NWIN>
__device__ __forceinline__ void issue_visit_tile(uint64_t a0, uint32_t band, uint32_t d, int nwin) {
    if (NWIN > 5 && nwin <= 5) issue_plain_windows<R, StageLines, 5>(a0, band, d);
    else issue_plain_windows<R, StageLines, NWIN>(a0, band, d);
}

// What one epilogue warp does with a tile: fixed over the tile's steps.
struct WarpTile {
    uint32_t col, ecol;  // TMEM: its blocks' first column, its halo panel's
    uint32_t img, eimg;  // image: this row of its blocks' first panel, of its halo panel
    uint32_t mask;       // the mask table
    int xf, ex;          // first column of its blocks, of its halo panel
    int tmax;            // the row may be written up to this step (0: never)
    bool inner;          // its blocks' and halo panel's columns all lie in the rectangle
    // otherwise: panels [p0, p1) of its blocks lie in the rectangle, the others
    // of [q0, q1) in part, and cells [ea, eb) of the halo panel
    int p0, p1, q0, q1, ea, eb;
};

// An intermediate step t: the new values go back into the image.  A step's
// MMAs wait for this chain, so it is kept to TMEM loads, conversions and
// predicated stores; only columns at the rectangle's edge take the blends of
// the second branch.
template <int G, typename Radius>  // (a constant's type, or int)
__device__ __forceinline__ void step_to_image(const WarpTile &c, int half, int t, Radius r, int x0, int x1) {
    const bool row = t <= c.tmax;
    // halo cells whose neighbourhood is all of step t-1: r t fewer
    const int ea = half ? 0 : r * t, eb = half ? 8 - r * t : 8;
    if (c.inner) {
        uint32_t e[8];
        tmem_ld_x8(c.ecol, e);
        const uint4 old = lds128(c.eimg);
        const uint4 m = lds128(c.mask + 16 * (half ? 9 + eb : ea));
        tmem_ld_wait(e);
        if (row) sts128(c.eimg, blend(pack_panel(e), old, m));
        walk_blocks<G>(c.col, [&](int p, const uint4 &w) {
            if (row) sts128(c.img + p * StageLines::CHUNK, w);
        });
    } else {
        if (c.ea < c.eb) {
            uint32_t e[8];
            tmem_ld_x8(c.ecol, e);
            const uint4 old = lds128(c.eimg);
            const uint4 m = cells_mask(c.mask, max(ea, c.ea), min(eb, c.eb));
            tmem_ld_wait(e);
            if (row) sts128(c.eimg, blend(pack_panel(e), old, m));
        }
        walk_blocks<G>(c.col, [&](int p, const uint4 &w) {
            const uint32_t at = c.img + p * StageLines::CHUNK;
            if (p >= c.p0 && p < c.p1) {
                if (row) sts128(at, w);
            } else if (p >= c.q0 && p < c.q1) {
                const int xb = c.xf + 8 * p;
                if (row) sts128(at, blend(w, lds128(at), cells_mask(c.mask, clamp8(x0 - xb), clamp8(x1 - xb))));
            }
        });
    }
}

// The visit's last step: the new values go to the output plane (dst: the
// blocks' first panel in this row), and the image's where they may not be
// written (every grid cell of an owned row is stored: the fixed border has to
// be in both planes).
template <int G>
__device__ __forceinline__ void step_to_plane(const WarpTile &c, int t, int x0, int x1, int nx,
                                              bool owned, uint4 *dst, int nyp) {
    const bool row = t <= c.tmax;
    if (c.inner && __all_sync(0xffffffffu, row || !owned)) {
        walk_blocks<G>(c.col, [&](int p, const uint4 &w) {
            if (owned) dst[(size_t)p * nyp] = w;
        });
    } else {
        walk_blocks<G>(c.col, [&](int p, const uint4 &w) {
            const int xb = c.xf + 8 * p;
            if (!owned || xb >= nx) return;
            const int a = row ? clamp8(x0 - xb) : 8, b = row ? clamp8(x1 - xb) : 0;
            dst[(size_t)p * nyp] =
                a == 0 && b == 8 ? w : blend(w, lds128(c.img + p * StageLines::CHUNK), cells_mask(c.mask, a, b));
        });
    }
}

// mbar_wait that polls for a while before it sleeps between polls: a step's
// waits end within a microsecond, and a sleep that outlasts one costs a
// quarter of a step.
__device__ __forceinline__ bool mbar_wait_soon(uint64_t *bar, uint32_t parity,
                                               const volatile int *abort_flag,
                                               uint64_t limit_ns = kWaitLimitNs) {
#pragma unroll 1
    for (int n = 0; n < 64; n++)
        if (mbar_try_wait(bar, parity)) return true;
    return mbar_wait(bar, parity, abort_flag, limit_ns);
}

}  // namespace tc
}  // namespace tcs
