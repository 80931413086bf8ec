// Temporally blocked split-precision sweep: TWO Jacobi steps per HBM round
// trip.  A split step moves 8 bytes per point update, which at the memory
// rate takes twice as long as a radius-1 tile's MMAs and as long as a
// radius-2 tile's; two steps per load and store halve the traffic.
//
// Tile.  As in the single-step split kernel (sweep_tc.cu), W = 128, 80 or 32
// columns wide (tb_width; the numbers here are for 128): the stage holds
// rows Yb-4 .. Yb+131 of the panels X0-8 .. X0+135, hi and lo, and one step's
// nine windows give rows Yb .. Yb+127 of the columns X0-16 .. X0+143.  The
// first step's values go back over the staged image (X0-8 .. X0+135: the
// halo panels lack only windows whose products with their valid cells are all
// zero), the second step's nine windows run on it, and the rows Yb+2 ..
// Yb+125 (from row 0 / to the last row for the first and last tile rows) go
// to the output planes.  Windows, their order and the split are the
// single-step kernel's, so two blocked steps give exactly the bits of two
// single steps.  Tile rows start at multiples of 124, so their copies move
// half lines (encode_panel_map with rows = 4; 120 and whole lines: 3 % more
// rows, the same time per tile).
//
// Pipeline.  Window accumulators stream through the ring of five 96-column
// TMEM regions of the single-step kernel, 18 windows per tile.  A block's new
// values overwrite its two panels as soon as its two windows are complete
// (no other window reads those panels), and window w of the second step
// waits for its two blocks: the second step follows the first a few windows
// behind, and the tensor pipe does not drain between them.  Radius 2 runs at
// the tensor pipe's 60 cycles per MMA (8196²: 98.6 -> 84.6 us per step against
// one step per launch); radius 1 (95.8 -> 72.5) at 480 cycles per window of 360
// cycles' MMAs, the five regions' turnaround.  An epilogue warp
// waits once per block, on a barrier that both windows' commits arrive at.
// (Waiting for windows, each released by all warps read or not, cost a warp
// 800 of 2200 cycles per block: 16386² box2d1r 399 us per step, 336 with the
// barriers per block; one range check per panel row instead of per pair
// -> 292; both panels summed before the first is split -> 272; the groups
// taking turns over both steps' blocks -> 264.  Reading each window the moment
// it completes, for three groups of 128 registers, was slower: 309.)  Rows
// outside the update rectangle are left out of the blocks and copied after
// them, and only panels that straddle its sides choose per cell: at 1026²,
// where half of the tiles touch the border, 6.5 -> 4.95 us per step, and 4.32
// with 80 columns (8.0 a step in single launches).  (The form this
// replaces, with 80-column tiles, a second image for the intermediate and a
// handoff per step, took 140 / 156 us per step at 8196², box2d1r / box2d2r.)
// Two stages: the next tile loads while a tile runs both its steps.
#include "tc_core.cuh"

namespace tcs {

namespace {

using namespace tc;
using SG = StageLines;

__device__ int g_tb_error = 0;

constexpr int kTbStages = 2;
constexpr int kTbGroups = 4;                // epilogue block groups
constexpr int kTbEpiWarps = 4 * kTbGroups;  // a lane quarter each
// MMA issuer warps 1 .. 3 take the windows w with w % 3 == id of every step;
// each waits for every stage fill, in order, and for the phases of its own
// windows' blocks.  A region's barrier completes a phase per window that used
// it; an issuer waits for window G's region only once window G - 5, whose
// issuer saw the release of window G - 10, has been issued (`issued`), so the
// parity it waits for cannot be that of an older phase.
constexpr int kTbIssuers = 3;
constexpr int kTbEpi0 = 1 + kTbIssuers;
constexpr int kTbThreads = 32 * (kTbEpi0 + kTbEpiWarps);

template <int S>
struct TbCfg {
    static constexpr int R = stencil_r(S);
    static constexpr bool BOX = stencil_box(S);
    static constexpr int NDY = 2 * R + 1;
    static constexpr size_t BAND = (size_t)4 * NDY * kBandBytes;
    static constexpr int BARS = 512;
    static constexpr size_t SMEM = 1024 + (size_t)kTbStages * 2 * SG::PLANE + BAND + BARS;
    static_assert(SMEM <= 232448, "shared memory budget");
};

struct TbParams {
    CUtensorMap map_hi, map_lo;  // input planes
    GridGeom g;
    int tiles_x, tiles_y, n_tiles;
    const uint16_t *in_hi, *in_lo;
    uint16_t *out_hi, *out_lo;
    SplitScale *scale;  // the grid's per-step scale (null: fixed scale)
    int t0;             // steps of the run done before this pair
    float coef[25];
};

template <int S, int W>
__global__ void __launch_bounds__(kTbThreads, 1) tc_split_tb_kernel(const __grid_constant__ TbParams p) {
    using C = TbCfg<S>;
    constexpr int R = C::R;
    constexpr int WIN = W / 16 + 1, BLK = W / 16 + 2, PANELS = W / 8 + 2;
    static_assert(WIN % kTbIssuers == 0 && 2 * WIN > kTbRing, "an issuer's windows and the barriers' phases");
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = align_smem(smem_raw);
    uint8_t *stage_base = smem;  // [stage][hi, lo]
    uint8_t *band_base = smem + (size_t)kTbStages * 2 * SG::PLANE;
    uint64_t *bars = reinterpret_cast<uint64_t *>(band_base + C::BAND);
    uint64_t *full = bars;                          // [stages]
    uint64_t *empty = full + kTbStages;             // [stages]
    uint64_t *win_empty = empty + kTbStages;        // [kTbRing] region read by its blocks' groups
    uint64_t *blk_full = win_empty + kTbRing;       // [2][BLK] a step's block: its windows complete
    uint64_t *blk_ready = blk_full + 2 * BLK; // [BLK] first-step values in the image
    uint64_t *drain = blk_ready + BLK;        // [1]
    CtaScale cs;                                    // the CTA's side of the scale
    cs.bar = drain + 1;                             // [2]
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(cs.bar + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    cs.max = tmem_slot + 2;                         // [2]
    cs.cnt = cs.max + 2;                            // [2]
    cs.ss = reinterpret_cast<StepScale *>(cs.cnt + 2);  // [2]
    uint32_t *issued = reinterpret_cast<uint32_t *>(cs.ss + 2);  // [kTbIssuers] 1 + its last window
    static_assert((2 * kTbStages + kTbRing + 3 * BLK + 3) * 8 + 24 + 2 * sizeof(StepScale) +
                          4 * kTbIssuers <= C::BARS,
                  "barrier area");

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int n_mine = (p.n_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kTbStages; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kTbIssuers);
        }
        for (int r = 0; r < kTbRing; r++) mbar_init(&win_empty[r], 8);  // two groups
        for (int b = 0; b < BLK; b++) {
            // the halo blocks have one window
            for (int st = 0; st < 2; st++)
                mbar_init(&blk_full[st * BLK + b], b == 0 || b == BLK - 1 ? 1 : 2);
            mbar_init(&blk_ready[b], 4);
        }
        for (int k = 0; k < kTbIssuers; k++) issued[k] = 0;
        mbar_init(drain, kTbIssuers);
        cta_scale_init(cs);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 1) {
        __syncwarp();
        tmem_alloc(tmem_slot, kTmemCols);
        tmem_relinquish();
    }
    build_bands(reinterpret_cast<uint16_t *>(band_base), p.coef, R, C::BOX, true, threadIdx.x,
                kTbThreads);
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // the previous step's CTAs may still run: planes only after pdl_wait
    pdl_launch_dependents();
    pdl_wait();

    auto fail = [&](int code) {
        record_error(&g_tb_error, code);
        *abort_flag = 1;
    };

    if (warp == 0) {
        // ------------------------------------------------------ producer ---
        if (lane == 0) {
            int last_issued = -1;
            for (int i = 0; i < n_mine; i++) {
                const int s = i % kTbStages;
                if (!mbar_wait(&empty[s], ((i / kTbStages) & 1) ^ 1, abort_flag)) {
                    fail(kErrWaitEmpty);
                    break;
                }
                const int t = (int)blockIdx.x + i * (int)gridDim.x;
                const int ty = t / p.tiles_x, tx = t - ty * p.tiles_x;
                uint8_t *st = stage_base + (size_t)s * 2 * SG::PLANE;
                mbar_arrive_expect_tx(&full[s], 2 * PANELS * SG::CHUNK);
                tma_load_3d(st, &p.map_hi, &full[s], 0, ty * kTbRows / kTbMapRows, tx * (W / 8));
                tma_load_3d(st + SG::PLANE, &p.map_lo, &full[s], 0, ty * kTbRows / kTbMapRows,
                            tx * (W / 8));
                last_issued = i;
            }
            for (int k = 0; k < kTbStages && last_issued - k >= 0; k++) {
                const int ii = last_issued - k;
                const uint64_t t0 = global_timer_ns();
                while (!mbar_try_wait(&full[ii % kTbStages], (ii / kTbStages) & 1)) {
                    if (global_timer_ns() - t0 > kWaitLimitNs) {
                        record_error(&g_tb_error, kErrWaitDrain);
                        break;
                    }
                }
            }
        }
    } else if (warp < kTbEpi0) {
        // --------------------------------------------------- MMA issuers ---
        if (lane == 0) {
            const int id = warp - 1;
            const uint32_t band = smem_u32(band_base);
            bool stop = false;
            // global window, its region, the region's uses before it
            int G = id, r = id % kTbRing, uses = id / kTbRing;
            const int before = (id + kTbIssuers - kTbRing % kTbIssuers) % kTbIssuers;  // issuer of G - 5
            // bounded wait until issuer k has issued window G
            auto issued_by = [&](int k, int G) {
                if (ld_acquire_cta(&issued[k]) > (uint32_t)G) return true;
                const uint64_t t0 = global_timer_ns();
                while (ld_acquire_cta(&issued[k]) <= (uint32_t)G)
                    if (*abort_flag || global_timer_ns() - t0 > kWaitLimitNs) return false;
                return true;
            };
            for (int i = 0; i < n_mine && !stop; i++) {
                const int s = i % kTbStages;
                if (!mbar_wait(&full[s], (i / kTbStages) & 1, abort_flag)) {
                    fail(kErrWaitFull);
                    break;
                }
                const uint64_t a_hi0 =
                    smem_desc(smem_u32(stage_base + (size_t)s * 2 * SG::PLANE), SG::CHUNK, 128);
                for (int sw = id; sw < 2 * WIN; sw += kTbIssuers) {
                    const bool second = sw >= WIN;
                    const int w = second ? sw - WIN : sw;
                    // window w's blocks are w and w + 1
                    if ((G >= kTbRing && !issued_by(before, G - kTbRing)) ||
                        !mbar_wait(&win_empty[r], (uses & 1) ^ 1, abort_flag) ||
                        (second && (!mbar_wait(&blk_ready[w], i & 1, abort_flag) ||
                                    !mbar_wait(&blk_ready[w + 1], i & 1, abort_flag)))) {
                        fail(kErrWaitAccum);
                        stop = true;
                        break;
                    }
                    tc_fence_after();
                    issue_split_window<R, SG>(a_hi0, band, tmem_base + r * kTbRegion, w);
                    st_release_cta(&issued[id], (uint32_t)G + 1);
                    // the window's two blocks (the second step has no halo blocks)
                    uint64_t *bf = blk_full + (second ? BLK : 0);
                    if (!second || w > 0) umma_commit(&bf[w]);
                    if (!second || w < WIN - 1) umma_commit(&bf[w + 1]);
                    G += kTbIssuers;
                    r += kTbIssuers;
                    while (r >= kTbRing) {
                        r -= kTbRing;
                        uses++;
                    }
                }
                if (!stop) umma_commit(&empty[s]);  // both steps' MMAs have read the stage
            }
            umma_commit(drain);  // completes at once if nothing is in flight
            const uint64_t t0 = global_timer_ns();
            while (!mbar_try_wait(drain, 0)) {
                if (global_timer_ns() - t0 > kWaitLimitNs) {
                    record_error(&g_tb_error, kErrWaitDrain);
                    break;
                }
            }
        }
    } else {
        // ------------------------------------------------------ epilogue ---
        const int q = warp & 3;
        // A tile's 18 blocks in order: blocks 0 .. 9 of the first step (block
        // b: columns X0-16+16b ..; 0 and 9 are the halo panels), then 1 .. 8
        // of the second; this group takes every fourth.
        const int grp = (warp - kTbEpi0) >> 2;
        const int m = q * 32 + lane;            // tile row
        const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16);
        const GridGeom &g = p.g;
        bool stop = false;
        // The pair's two scales, both from steps finished before the launch
        // (step t reads steps t-2 and t-3), read by the first epilogue warp;
        // the second step's copies come from the input, two steps back, so
        // they take both shifts.
        if (warp == kTbEpi0 && lane == 0) {
            cta_scale_publish(cs, 0, step_scale(p.scale, p.t0 + 1));
            cta_scale_publish(cs, 1, step_scale(p.scale, p.t0 + 2));
        }
        StepScale ss1, ss2;
        if (!cta_scale_take(cs, 0, ss1, abort_flag) || !cta_scale_take(cs, 1, ss2, abort_flag)) {
            if (lane == 0) fail(kErrWaitResult);
            stop = true;
        }
        StepScale cs2 = ss2;
        cs2.k = ss1.k + ss2.k;
        cs2.s = __int_as_float((127 + 11 + cs2.k) << 23);
        float mx1 = 0.0f, mx2 = 0.0f;
        int r0 = 0;  // ring region of the tile's window 0
        // One block: wait for its windows, load and sum its panels, give the
        // windows back, and sink each panel (its index in the image, its
        // eight values).  rb: region of the step's window 0, at most 4.
        auto take_block = [&](int st, int b, int rb, int i, const StepScale &ss, auto &&sink) {
            bool ok = mbar_wait(&blk_full[st * BLK + b], i & 1, abort_flag);
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) fail(kErrWaitResult);
                return false;
            }
            tc_fence_after();
            auto region = [&](int w) {
                const int x = rb + w;  // < 14
                return x >= 10 ? x - 10 : x >= 5 ? x - 5 : x;
            };
            const int wa = region(b - 1), wb = region(b);
            const uint32_t ta = lane_base + (uint32_t)(wa * kTbRegion) + 16;  // its second half
            const uint32_t tb = lane_base + (uint32_t)(wb * kTbRegion);       // its first half
            auto release = [&]() {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    // in the second step the outer windows have one block
                    if (b > 0) mbar_arrive_n(&win_empty[wa], st == 1 && b == 1 ? 2 : 1);
                    if (b < BLK - 1) mbar_arrive_n(&win_empty[wb], st == 1 && b == BLK - 2 ? 2 : 1);
                }
            };
            float u[8];
            uint32_t v[6][8];
            if (b == 0 || b == BLK - 1) {
                // halo panel: the inner one of the block; cells that lack a
                // column of the input are zero (nothing valid reads them)
                panel_load(b == 0 ? tb + 8 : ta, 0, false, v);
                tmem_ld_wait(v);
                release();
                panel_sum(v, false, ss, u);
#pragma unroll
                for (int c = 0; c < 8; c++)
                    if (b == 0 ? c < R : c >= 8 - R) u[c] = 0.0f;
                sink(b == 0 ? 0 : 2 * b - 1, u);
            } else {
                // (both panels are summed before the first is split: with
                // five regions the windows wait for this release)
                float u2[8];
                panel_load(ta, tb, true, v);
                tmem_ld_wait(v);
                panel_sum(v, true, ss, u);
                panel_load(ta + 8, tb + 8, true, v);
                tmem_ld_wait(v);
                release();
                panel_sum(v, true, ss, u2);
                sink(2 * b - 1, u);
                sink(2 * b, u2);
            }
            return true;
        };
        for (int i = 0; i < n_mine && !stop; i++) {
            const int t = (int)blockIdx.x + i * (int)gridDim.x;
            const int ty = t / p.tiles_x, tx = t - ty * p.tiles_x;
            const int Yb = ty * kTbRows, X0 = tx * W;
            const int y = Yb + m;
            const bool top = ty == 0, bottom = ty == p.tiles_y - 1;
            const bool row_in = y >= g.y0 && y < g.y1;
            const bool mine = (top || m >= kTbHalo) && (bottom || m < kTile - kTbHalo) && y < g.ny;
            const uint32_t img = smem_u32(stage_base) +
                                 (uint32_t)((i % kTbStages) * 2 * SG::PLANE + (m + SG::TOP) * 16);
            const size_t row0 = plane_index16(g.p16, mine ? y : 0, X0 - 8);
            // (rolled: unrolled, as it would be for 80 columns, it spills registers)
#pragma unroll 1
            for (int idx = grp; idx < 2 * WIN && !stop; idx += kTbGroups) {
                if (idx < BLK) {
                    // first step -> the image
                    const bool ok = take_block(0, idx, r0, i, ss1, [&](int pan, const float (&u)[8]) {
                        const int xb = X0 - 8 + 8 * pan;
                        const uint32_t a = img + (uint32_t)(pan * SG::CHUNK);
                        PanelPair w;
                        if (!row_in) {  // a row that keeps its values
                            if (ss1.k == 0) return;
                            w = resplit_panel(PanelPair{lds128(a), lds128(a + SG::PLANE)}, ss1);
                        } else if (xb >= g.x0 && xb + 8 <= g.x1) {
                            w = split_panel(u, mx1);
                        } else {
                            const PanelPair old{lds128(a), lds128(a + SG::PLANE)};
                            w = split_panel_edge(u, old, xb, g.x0, g.x1, ss1, mx1);
                        }
                        sts128(a, w.hi);
                        sts128(a + SG::PLANE, w.lo);
                    });
                    if (!ok) {
                        stop = true;
                        break;
                    }
                    fence_proxy_async_smem();  // an MMA operand next
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&blk_ready[idx]);
                } else {
                    // second step -> the output planes
                    const int rb = (r0 + WIN) % kTbRing;
                    const bool ok = take_block(1, idx - WIN, rb, i, ss2, [&](int pan, const float (&u)[8]) {
                        const int xb = X0 - 8 + 8 * pan;
                        if (!mine || !row_in || xb >= g.nx) return;
                        const size_t off = row0 + (size_t)pan * g.p16.nyp * 8;
                        PanelPair w;
                        if (xb >= g.x0 && xb + 8 <= g.x1) {
                            w = split_panel(u, mx2);
                        } else {
                            const PanelPair old{*reinterpret_cast<const uint4 *>(p.in_hi + off),
                                                *reinterpret_cast<const uint4 *>(p.in_lo + off)};
                            w = split_panel_edge(u, old, xb, g.x0, g.x1, cs2, mx2);
                        }
                        *reinterpret_cast<uint4 *>(p.out_hi + off) = w.hi;
                        *reinterpret_cast<uint4 *>(p.out_lo + off) = w.lo;
                    });
                    if (!ok) stop = true;
                    __syncwarp();  // rows may have parted; warp-wide TMEM loads next
                }
            }
            r0 = (r0 + 2 * WIN) % kTbRing;
            // rows that keep their values: this group's panels
            if (!stop && mine && !row_in) {
#pragma unroll 1
                for (int pan = 1 + grp; pan <= W / 8 && X0 - 8 + 8 * pan < g.nx; pan += kTbGroups) {
                    const size_t off = row0 + (size_t)pan * g.p16.nyp * 8;
                    PanelPair w{*reinterpret_cast<const uint4 *>(p.in_hi + off),
                                *reinterpret_cast<const uint4 *>(p.in_lo + off)};
                    if (cs2.k != 0) w = resplit_panel(w, cs2);
                    *reinterpret_cast<uint4 *>(p.out_hi + off) = w.hi;
                    *reinterpret_cast<uint4 *>(p.out_lo + off) = w.lo;
                }
            }
            __syncwarp();
        }
        if (!stop && p.scale) {  // tile 0 is CTA 0's
            cta_scale_flush<kTbEpiWarps>(cs, 0, p.scale, p.t0 + 1, ss1, mx1, blockIdx.x == 0);
            cta_scale_flush<kTbEpiWarps>(cs, 1, p.scale, p.t0 + 2, ss2, mx2, blockIdx.x == 0);
        }
    }

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) {
        __syncwarp();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

int g_tb_sms = 0;

// Tile columns: what a launch takes is about its waves of tiles times a tile's
// windows (2 (W/16 + 1), one after another), so a grid of few tiles is cut
// narrower; a tie goes to the wider tile, which recomputes less halo.  32
// columns only while they leave half of the SMs free: past that their loads
// and launches, 1.5 times as many bytes per cell, take back what the shorter
// chain gives.  us per step of a pair, W = 128 / 80 / 32 (box2d1r; box2d2r):
// 256² 4.72 / 3.82 / 3.15 (5.26 / 4.14 / 3.48), 512² 4.79 / 3.78 / 3.55, 724²
// 4.78 / 3.87 / 3.89 (5.28 / 4.23 / 4.81), 1024² 4.75 / 4.36 / 4.99, 1600² 7.51
// / 5.91 / 7.77 (8.43 / 7.04 / 9.53), 2048² 7.61 / 7.70 / 11.1, 4096² 20.8 /
// 22.6 / 34.1, 8196² 73.1 / 75.4 / 129.  (A tile takes 3, 6 or 9 windows a step:
// a multiple of the issuers, so that an issuer's windows are the same in every
// tile.)
int tb_width(const GridGeom &g) {
    const int ty = tb_tiles_y(g.ny);
    auto tiles = [&](int w) { return (long long)((g.nx + w - 1) / w) * ty; };
    auto waves = [&](int w) { return (tiles(w) + g_tb_sms - 1) / g_tb_sms; };
    if (tiles(32) <= g_tb_sms / 2) return 32;
    return waves(80) * 6 < waves(128) * 9 ? 80 : 128;
}

template <int S, int W>
cudaError_t launch_tb_w(TbParams &p, cudaStream_t s) {
    using C = TbCfg<S>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(tc_split_tb_kernel<S, W>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(C::SMEM));
        if (e != cudaSuccess) return e;
        configured = true;
    }
    cudaError_t e = encode_panel_map(p.in_hi, p.g.p16, &p.map_hi, W / 8 + 2, kTbMapRows);
    if (e == cudaSuccess) e = encode_panel_map(p.in_lo, p.g.p16, &p.map_lo, W / 8 + 2, kTbMapRows);
    if (e != cudaSuccess) return e;
    p.tiles_x = (p.g.nx + W - 1) / W;
    p.n_tiles = p.tiles_x * p.tiles_y;
    const int grid = p.n_tiles < g_tb_sms ? p.n_tiles : g_tb_sms;
    return launch_step(tc_split_tb_kernel<S, W>, grid, kTbThreads, C::SMEM, s, p);
}

template <int S>
cudaError_t launch_tb(const GridGeom &g, const float *B, const uint16_t *in_hi,
                      const uint16_t *in_lo, uint16_t *out_hi, uint16_t *out_lo, cudaStream_t s,
                      SplitScale *scale, int t0) {
    using C = TbCfg<S>;
    if (!g_tb_sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_tb_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_tb_sms <= 0) g_tb_sms = 1;
    }
    TbParams p;
    p.g = g;
    p.tiles_y = tb_tiles_y(g.ny);
    p.in_hi = in_hi;
    p.in_lo = in_lo;
    p.out_hi = out_hi;
    p.out_lo = out_lo;
    p.scale = scale;
    p.t0 = t0;
    for (int k = 0; k < 25; k++) p.coef[k] = k < C::NDY * C::NDY ? B[k] : 0.0f;
    switch (tb_width(g)) {
    case 32: return launch_tb_w<S, 32>(p, s);
    case 80: return launch_tb_w<S, 80>(p, s);
    default: return launch_tb_w<S, 128>(p, s);
    }
}

}  // namespace

cudaError_t launch_tc_split2(const GridGeom &g, int stencil, const float *B, const uint16_t *in_hi,
                             const uint16_t *in_lo, uint16_t *out_hi, uint16_t *out_lo,
                             cudaStream_t s, SplitScale *scale, int t0) {
    switch (stencil) {
    case TCS_STAR2D1R: return launch_tb<TCS_STAR2D1R>(g, B, in_hi, in_lo, out_hi, out_lo, s, scale, t0);
    case TCS_STAR2D2R: return launch_tb<TCS_STAR2D2R>(g, B, in_hi, in_lo, out_hi, out_lo, s, scale, t0);
    case TCS_BOX2D1R: return launch_tb<TCS_BOX2D1R>(g, B, in_hi, in_lo, out_hi, out_lo, s, scale, t0);
    case TCS_BOX2D2R: return launch_tb<TCS_BOX2D2R>(g, B, in_hi, in_lo, out_hi, out_lo, s, scale, t0);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t tb_error_word(int **word) {
    return cudaGetSymbolAddress(reinterpret_cast<void **>(word), g_tb_error);
}

}  // namespace tcs
