// Plain FP16 sweeps of several steps per tile visit: a tile is loaded once,
// stepped T times in shared memory and stored once.
//
// A step that reads and writes every plane moves 4 bytes per point update,
// which at 8196² takes as long as the two issuers of tc_sweep_kernel need for
// the radius-2 MMAs and 1.6 times as long as the radius-1 MMAs; a small grid's
// step is a launch boundary, a load and a store around about a microsecond of
// MMAs.  Both come down to one load and one store per T steps here.
//
// Tile.  As in tc_sweep_kernel (sweep_tc.cu): the stage holds rows
// Yb-4 .. Yb+131 of the panels X0-8 .. X0+W+7, an MMA step gives rows
// Yb .. Yb+127 of the columns X0-16 .. X0+W+15, and the windows and their
// order are the same, so every cell sums the same products in the same order
// as in a single-step launch.  After a step the epilogue warps write the new
// values back over the staged image (all MMAs that read it are complete),
// X0-8 .. X0+W+7 included, and the next step's MMAs run on the image.  Cells
// whose neighbourhood is not all of the previous step are not written: r more
// rows at the image's top and bottom and r more columns at its sides with
// every step (r(t-1) rows, r t columns after t steps), so the image only ever
// holds values of the field.  The halo columns are the staged panels on
// either side, which bounds r T by 8; an incomplete halo column lacks only
// windows whose products with it are all zero.  Tile rows overlap by 2 halo
// rows, halo = 2, 4 or 8 (>= r(T-1)): the tile at Yb = ty (128 - 2 halo) owns rows
// Yb+halo .. Yb+127-halo (from row 0, to the last row, for the first and last
// tile rows), stored to the other plane after the visit's last step.
//
// Pipeline.  Two MMA issuers, each with its own accumulator slot and its own
// eight epilogue warps (a lane quarter and a column half each): while one
// slot's tile is in its epilogue, the other's MMAs run.  Each slot walks its
// tiles in order and never waits for the other, because with few tiles per SM
// the other slot's tile may be of the next visit and wait for this one's
// result.  Stage i % 4 holds tile i, so each stage belongs to one issuer.
// A tile's visit j needs visit j-1 of itself and its eight neighbours: they
// hold its input, and they were the last readers of the plane it overwrites.
// Every tile has a counter of its finished visits, added to with one release
// reduction by the last of its epilogue warps; nine lanes of the producer
// warp poll the nine counters at once.  (Counters per tile row, as the split
// kernel's several-step form has, made a visit's boundary 3.3 us on a
// 333 x 1517 grid: a tile waited for its rows' slowest CTA, and 192 reductions
// met on one word.  A reduction by each of a tile's eight warps: 8196²
// star2d1r 28.3 us per step, 26.9 with one.)  The launch is cooperative: all
// CTAs are resident at once.  Every wait is bounded.
//
// Cells that are not finite: an MMA multiplies all 16 columns of a window, so
// one infinity or NaN makes every output of its windows in the reaching rows
// NaN, here as in single steps; which further cells it reaches over several
// steps depends on the visit's halo.
#include <algorithm>
#include <cmath>

#include "tc_core.cuh"
#include "tile_walk.h"
#include "visit_tile.cuh"

namespace tcs {

namespace {

using namespace tc;
using SG = StageLines;

__device__ int g_visit_error = 0;

constexpr int kVisitSlots = 2;
constexpr int kVisitStages = 4;                 // a multiple of the slots
constexpr int kVisitEpi0 = 1 + kVisitSlots;     // first epilogue warp
constexpr int kVisitEpi = 8;                    // epilogue warps per slot
constexpr int kVisitThreads = 32 * (kVisitEpi0 + kVisitSlots * kVisitEpi);
constexpr int kBarBytes = 256;                  // barriers and flags, before the masks

struct VisitParams {
    CUtensorMap map[2];  // the planes; visit j reads map[j & 1]
    GridGeom g;
    int tiles_x, tiles_y, halo;
    int map_rows;             // rows of a panel per box line (encode_panel_map)
    int visits, base, extra;  // visit j takes base + (j < extra) steps
    unsigned *ended;          // CTAs at the end of the launch (zero at its start)
    unsigned *done;           // [tiles] the tile's finished visits (zeros)
    uint16_t *plane[2];
    float coef[25];
};

// TMEM columns of a slot (16 (W/16 + 2) used): all there are between the two,
// or, beside another launch's CTA, what 32-column tiles need.
__host__ __device__ constexpr int visit_slot_cols(int ctas) { return ctas == 2 ? 64 : kTmemCols / kVisitSlots; }
__host__ __device__ constexpr int visit_stage_bytes(int W) { return (W / 8 + 2) * SG::CHUNK; }

// Waits (bounded) for visit w.step - 1 of the tile and its neighbours: lane l
// < 9 acquires the counter of neighbour l.  Called by a whole warp.
__device__ __forceinline__ bool wait_neighbours(const unsigned *done, const TileWalk &w, int lane,
                                                const volatile int *abort_flag) {
    const int y = w.ty + lane / 3 - 1, x = w.tx + lane % 3 - 1;
    const bool mine = lane < 9 && y >= 0 && y < w.tiles_y && x >= 0 && x < w.tiles_x;
    const unsigned *ctr = done + (mine ? y * w.tiles_x + x : 0);
    const unsigned target = (unsigned)w.step;
    const uint64_t t0 = global_timer_ns();
    // the error word and the clock, which take as long as a poll each, are
    // read only now and then
    for (int n = 1; !__all_sync(0xffffffffu, !mine || ld_acquire(ctr) >= target); n++) {
        if (n % 32) continue;
        const bool stop = *abort_flag || *(volatile int *)&g_visit_error != 0 ||
                          global_timer_ns() - t0 > kWaitLimitNs;
        if (__any_sync(0xffffffffu, stop)) return false;
    }
    // (a vote orders no memory: the barrier puts every lane's acquire before
    // what lane 0 does next)
    __syncwarp();
    return true;
}

// The last CTA whose tiles need no counter any more leaves them zero for the
// next launch (a memset before each launch took a tenth of a 256², 10-step
// run).  By then every tile's last addition has been made: a tile's last visit
// waits for its own, and the CTAs count here after their last waits, beside
// their last visits' steps (at the kernel's end it was 1 us of a small
// launch).  Called by a whole warp.
__device__ __forceinline__ void leave_counters(const VisitParams &p, int lane) {
    if (p.visits < 2) return;
    int last = 0;
    if (lane == 0) {
        fence_acq_rel_gpu();
        last = atomicAdd(p.ended, 1u) == gridDim.x - 1;
        fence_acq_rel_gpu();
    }
    if (!__shfl_sync(0xffffffffu, last, 0)) return;
    __syncwarp();  // lane 0's acquire before the other lanes' stores
    for (int t = lane; t < p.tiles_x * p.tiles_y; t += 32) p.done[t] = 0;
    if (lane == 0) *p.ended = 0;
}

// G: a tile is W = 32 G columns wide, G blocks of 16 for each column half.
// CTAS: 2 leaves room on an SM for a CTA of another launch (launch_visit).
template <int S, int G, int CTAS>
__global__ void __launch_bounds__(kVisitThreads, CTAS) tc_visit_kernel(const __grid_constant__ VisitParams p) {
    constexpr int R = stencil_r(S);
    constexpr int W = 32 * G;
    constexpr int stage_bytes = visit_stage_bytes(W);
    constexpr int NS = kVisitStages;
    constexpr int slot_cols = visit_slot_cols(CTAS);
    static_assert(16 * (W / 16 + 2) <= slot_cols, "TMEM slot");
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = align_smem(smem_raw);
    uint8_t *stage_base = smem;                          // [NS]
    uint8_t *band_base = smem + (size_t)NS * stage_bytes;  // [2R+1]
    uint64_t *bars = reinterpret_cast<uint64_t *>(band_base + (2 * R + 1) * kBandBytes);
    uint64_t *full = bars;                        // [NS] tile loaded
    uint64_t *empty = full + NS;                  // [NS] tile stored
    uint64_t *acc_full = empty + NS;              // [slots] a step's MMAs complete
    uint64_t *step_done = acc_full + kVisitSlots; // [slots] its results in the image (or registers)
    uint64_t *drain = step_done + kVisitSlots;    // [1]
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    unsigned *stored = tmem_slot + 2;             // [slots] warps that stored their last step
    volatile unsigned *left_over = stored + kVisitSlots;  // the producer gave up
    static_assert((2 * NS + 2 * kVisitSlots + 1) * 8 + 12 + 4 * kVisitSlots <= kBarBytes, "barrier area");
    uint32_t *masks = reinterpret_cast<uint32_t *>(reinterpret_cast<uint8_t *>(bars) + kBarBytes);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < NS; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kVisitEpi);
        }
        for (int b = 0; b < kVisitSlots; b++) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&step_done[b], kVisitEpi);
            stored[b] = 0;
        }
        mbar_init(drain, kVisitSlots);
        *abort_flag = 0;
        *left_over = 0;
        fence_mbar_init();
        // the first tile's load runs beside the rest of the set-up
        mbar_arrive_expect_tx(&full[0], (uint32_t)stage_bytes);
        tma_load_3d(stage_base, &p.map[0], &full[0], 0, (int)blockIdx.x / p.tiles_x * (kTile - 2 * p.halo) / p.map_rows,
                    (int)blockIdx.x % p.tiles_x * W / 8);
    }
    if (warp == 1) {
        __syncwarp();
        tmem_alloc(tmem_slot, kVisitSlots * slot_cols);
        tmem_relinquish();
    }
    build_bands(reinterpret_cast<uint16_t *>(band_base), p.coef, R, stencil_box(S), false,
                threadIdx.x, kVisitThreads);
    build_masks(masks, threadIdx.x);
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    const int tiles_x = p.tiles_x, tiles_y = p.tiles_y;
    const int n_items = p.visits * tiles_x * tiles_y;  // (visit, tile), visit-major
    const int H = kTile - 2 * p.halo;                  // rows from one tile row to the next
    const int grid = (int)gridDim.x;
    auto fail = [&](int code) {
        record_error(&g_visit_error, code);
        *abort_flag = 1;
    };

    if (warp == 0) {
        // ------------------------------------------------------ producer ---
        int i = 0, last_issued = 0;
        TileWalk w;
        w.init(blockIdx.x, grid, tiles_x, tiles_y);
        for (int k = blockIdx.x; k < n_items; k += grid, i++, w.advance()) {
            if (i == 0) continue;  // loaded above
            const int s = i % NS;
            if (w.step > 0 && !wait_neighbours(p.done, w, lane, abort_flag)) {
                if (lane == 0) fail(kErrWaitDep);
                break;
            }
            int ok = 1;
            if (lane == 0) {
                ok = mbar_wait(&empty[s], ((i / NS) & 1) ^ 1, abort_flag);
                if (ok) {
                    fence_proxy_async_global();  // the copy reads what other SMs stored
                    mbar_arrive_expect_tx(&full[s], (uint32_t)stage_bytes);
                    tma_load_3d(stage_base + (size_t)s * stage_bytes, &p.map[w.step & 1], &full[s],
                                0, w.ty * H / p.map_rows, w.tx * W / 8);
                } else {
                    fail(kErrWaitEmpty);
                }
            }
            if (!__shfl_sync(0xffffffffu, ok, 0)) break;
            last_issued = i;
        }
        // no counter is read or added to by this CTA from here on
        if (i * grid + (int)blockIdx.x >= n_items) leave_counters(p, lane);
        else if (lane == 0) *left_over = 1;
        // every stage armed last must have landed before exit
        if (lane == 0) {
            for (int k = 0; k < NS && last_issued - k >= 0; k++) {
                const int ii = last_issued - k;
                const uint64_t t0 = global_timer_ns();
                while (!mbar_try_wait(&full[ii % NS], (ii / NS) & 1)) {
                    if (global_timer_ns() - t0 > kWaitLimitNs) {
                        record_error(&g_visit_error, kErrWaitDrain);
                        break;
                    }
                }
            }
        }
    } else if (warp < kVisitEpi0) {
        // --------------------------------------------------- MMA issuers ---
        if (lane == 0) {
            const int id = warp - 1;  // its slot: tiles i with i % slots == id
            const uint32_t band = smem_u32(band_base);
            const uint32_t d = tmem_base + (uint32_t)(id * slot_cols);
            bool stop = false;
            uint32_t e = 0;  // the slot's steps so far
            TileWalk w;
            w.init(blockIdx.x + id * grid, kVisitSlots * grid, tiles_x, tiles_y);
            int i = id;
            for (int k = blockIdx.x + id * grid; k < n_items && !stop;
                 k += kVisitSlots * grid, i += kVisitSlots, w.advance()) {
                const int s = i % NS;
                if (!mbar_wait_soon(&full[s], (i / NS) & 1, abort_flag)) {
                    fail(kErrWaitFull);
                    break;
                }
                const uint64_t a0 = smem_desc(smem_u32(stage_base + (size_t)s * stage_bytes), SG::CHUNK, 128);
                const int T = p.base + (w.step < p.extra ? 1 : 0);
                const int nwin = tile_windows(p.g.nx, w.tx * W, W);
                for (int t = 0; t < T; t++, e++) {
                    // the slot's previous step has been read out (and, within
                    // a visit, written to the image)
                    if (e > 0 && !mbar_wait_soon(&step_done[id], (e - 1) & 1, abort_flag)) {
                        fail(kErrWaitAccum);
                        stop = true;
                        break;
                    }
                    tc_fence_after();
                    issue_visit_tile<R, W / 16 + 1>(a0, band, d, nwin);
                    umma_commit(&acc_full[id]);
                }
            }
            umma_commit(drain);  // completes at once if nothing is in flight
            const uint64_t t0 = global_timer_ns();
            while (!mbar_try_wait(drain, 0)) {
                if (global_timer_ns() - t0 > kWaitLimitNs) {
                    record_error(&g_visit_error, kErrWaitDrain);
                    break;
                }
            }
        }
    } else {
        // ------------------------------------------------------ epilogue ---
        const int slot = (warp - kVisitEpi0) / kVisitEpi;
        const int half = ((warp - kVisitEpi0) >> 2) & 1;
        const int q = warp & 3;       // TMEM lane quarter
        const int m = q * 32 + lane;  // tile row
        const uint32_t lane_col =
            tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(slot * slot_cols);
        const GridGeom &g = p.g;
        uint32_t e = 0;  // the slot's steps so far
        bool stop = false;
        WarpTile c;
        c.col = lane_col + 16 * (half * G + 1);
        c.ecol = lane_col + (half ? 16 + W : 8);
        c.mask = smem_u32(masks);
        TileWalk w;
        w.init(blockIdx.x + slot * grid, kVisitSlots * grid, tiles_x, tiles_y);
        int i = slot;
        for (int k = blockIdx.x + slot * grid; k < n_items && !stop;
             k += kVisitSlots * grid, i += kVisitSlots, w.advance()) {
            const int s = i % NS;
            const int T = p.base + (w.step < p.extra ? 1 : 0);
            const int X0 = w.tx * W;
            const int y = w.ty * H + m;
            const bool top = w.ty == 0, bottom = w.ty == tiles_y - 1;
            c.xf = X0 + 16 * half * G;
            c.ex = half ? X0 + W : X0 - 8;
            const uint32_t row0 = smem_u32(stage_base) + (uint32_t)(s * stage_bytes + (m + SG::TOP) * 16);
            c.img = row0 + (uint32_t)((1 + 2 * half * G) * SG::CHUNK);
            c.eimg = row0 + (uint32_t)((half ? 4 * G + 1 : 0) * SG::CHUNK);
            c.inner = min(c.xf, c.ex) >= g.x0 && max(c.xf + 16 * G, c.ex + 8) <= g.x1;
            if (!c.inner) {
                c.q0 = (g.x0 - c.xf) >> 3;
                c.p0 = (g.x0 - c.xf + 7) >> 3;
                c.p1 = (g.x1 - c.xf) >> 3;
                c.q1 = (g.x1 - c.xf + 7) >> 3;
                c.ea = clamp8(g.x0 - c.ex);
                c.eb = clamp8(g.x1 - c.ex);
            }
            // rows whose neighbourhood is all of step t-1: R fewer a step,
            // except at the grid's own top and bottom
            c.tmax = y >= g.y0 && y < g.y1
                         ? min(top ? kTile : m / R + 1, bottom ? kTile : (kTile - 1 - m) / R + 1)
                         : 0;
            for (int t = 1; t <= T; t++, e++) {
                bool ok = mbar_wait_soon(&acc_full[slot], e & 1, abort_flag);
                if (!__all_sync(0xffffffffu, ok)) {
                    if (lane == 0) fail(kErrWaitResult);
                    stop = true;
                    break;
                }
                tc_fence_after();
                if (t < T) {
                    step_to_image<G>(c, half, t, std::integral_constant<int, R>{}, g.x0, g.x1);
                    fence_proxy_async_smem();  // the next step's MMAs read the image
                } else {
                    const bool owned = y < g.ny && (top || m >= p.halo) && (bottom || m < kTile - p.halo);
                    uint4 *dst = reinterpret_cast<uint4 *>(p.plane[(w.step & 1) ^ 1] +
                                                           plane_index16(g.p16, owned ? y : 0, c.xf));
                    step_to_plane<G>(c, t, g.x0, g.x1, g.nx, owned, dst, g.p16.nyp);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&step_done[slot]);
                    if (t == T) {
                        mbar_arrive(&empty[s]);
                        // the tile's last warp publishes it: the warps' stores
                        // are ordered by the barrier above and this count, and
                        // visible to whoever acquires the tile's counter
                        if (w.step + 1 < p.visits &&
                            add_acq_rel_cta(&stored[slot], 1u) % kVisitEpi == kVisitEpi - 1)
                            red_release_add(p.done + w.ty * tiles_x + w.tx, 1u);
                    }
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) {
        __syncwarp();
        tmem_dealloc(tmem_base, kVisitSlots * slot_cols);
    }
    // a producer that gave up did not leave the counters
    if (*left_over && warp == 0) leave_counters(p, lane);
}

// A launch's CTAs wait on one another, so none may wait for TMEM that a CTA
// which itself waits holds.  One CTA per SM takes all of TMEM, and more than
// half of the shared memory, so that it stands alone.  The form for two takes
// 128 of the 512 columns and just under half: two of them fit, but neither fits
// beside any other kernel that takes TMEM (tc_sweep_kernel, the smallest, has
// 121 KB and up).
template <int CTAS>
size_t visit_smem(int R, int W) {
    const size_t need = 1024 + (size_t)kVisitStages * visit_stage_bytes(W) + (2 * R + 1) * kBandBytes + kBarBytes + kMaskBytes;
    const size_t least = (CTAS == 2 ? 110 : 120) * 1024;
    return need > least ? need : least;
}

template <int S, int G, int CTAS = 1>
cudaError_t launch_visit_w(VisitParams &p, int sms, cudaStream_t s) {
    const int tiles = p.tiles_x * p.tiles_y;
    const int grid = tiles < sms ? tiles : sms;
    return launch_step(tc_visit_kernel<S, G, CTAS>, grid, kVisitThreads, visit_smem<CTAS>(stencil_r(S), 32 * G),
                       s, p, true);
}
// 32-column tiles on more than half of the SMs, but not on nearly all, go out in
// the form that shares an SM with another launch's: plans in several streams
// then run side by side, two launches to an SM, where such whole-SM launches
// take turns (smaller ones have room beside one another).  512² in 20 steps, us
// per step of one of 8 plans in 8 streams (a launch per step / whole SMs /
// shared): star2d1r 0.64 / 0.93 / 0.38, box2d2r 0.72 / 1.32 / 0.55.  Its 48
// registers instead of 84 cost one plan alone 0 to 3 % (512², 64 steps: star2d1r
// 0.994 -> 0.997, box2d2r 1.41 -> 1.44 us per step), and 5 % with more tiles (700²
// box2d2r 1.44 -> 1.52), where a launch per step takes turns as well.
template <int S>
cudaError_t launch_visit(VisitParams &p, int w, int sms, cudaStream_t s) {
    const int tiles = p.tiles_x * p.tiles_y;
    if (w == 32 && 2 * tiles > sms && 4 * tiles <= 3 * sms) return launch_visit_w<S, 1, 2>(p, sms, s);
    return w == 128  ? launch_visit_w<S, 4>(p, sms, s)
           : w == 96 ? launch_visit_w<S, 3>(p, sms, s)
           : w == 64 ? launch_visit_w<S, 2>(p, sms, s)
                     : launch_visit_w<S, 1>(p, sms, s);
}

template <int S, int G, int CTAS = 1>
cudaError_t prepare_visit_w() {
    return cudaFuncSetAttribute(tc_visit_kernel<S, G, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)visit_smem<CTAS>(stencil_r(S), 32 * G));
}
template <int S>
cudaError_t prepare_visit() {
    static bool configured = false;
    if (configured) return cudaSuccess;
    cudaError_t e = prepare_visit_w<S, 1>();
    if (e == cudaSuccess) e = prepare_visit_w<S, 1, 2>();
    if (e == cudaSuccess) e = prepare_visit_w<S, 2>();
    if (e == cudaSuccess) e = prepare_visit_w<S, 3>();
    if (e == cudaSuccess) e = prepare_visit_w<S, 4>();
    configured = e == cudaSuccess;
    return e;
}

}  // namespace

// The tile width and halo of a sweep, from a model of its SM cycles that was
// fitted to 2640 sweeps of 256² to 4096² in 2 to 64 steps (M: a tile's MMAs; L:
// from the last MMA of a step to the slot's next one; n tiles per SM; I: the
// visits a CTA makes, between their average and that of the CTAs with one tile
// more, as neighbours wait for one another):
//   one tile after another:  visits (T (M + L) + 3417)
//   two slots at a time:     I (T max(M, 0.575 (M + L)) + 243)
// of which the larger.
// Narrow tiles have short steps and more SMs, wide ones fewer MMAs per cell;
// halo 8 takes more steps per visit, halo 4 fewer rows twice, and halo 2
// (whose copies move half lines) pays only for radius 2 with many tiles,
// where T = 2 already takes the sweep off the memory bound.  Against widths of
// 64 and 96 columns set by the caller, over 13 grids of 256² to 8196², four
// stencils and calls of 4 to 100 steps, the choice is 1.0 % behind the best on
// average; where it misses most is radius 2 at 2048² (100 steps: 3.55 us per
// step, 64 columns 2.85) and in calls of four steps around 1300² (3.7, 3.1);
// profiles/visit_widths.md has all.  us per step in calls of 100 steps, against
// one launch per step, star2d1r / box2d2r: 256² 4.45 -> 0.98 / 5.06 -> 1.40, 1026²
// 4.83 -> 1.23 / 5.43 -> 1.58, 4096² 11.1 -> 6.81 / 12.8 -> 9.39, 8196² 46.4 ->
// 26.7 / 47.9 -> 36.8.
VisitShape visit_shape(int ny, int nx, int stencil, int steps, int tile_w, int sms) {
    const int r = stencil_r(stencil);
    VisitShape best{};
    double best_cost = 0.0;
    for (int w = 32; w <= kTile; w += 32) {
        if (tile_w != kTile && w != tile_w) continue;  // a width the caller set stays
        for (int halo = 2; halo <= 8; halo *= 2) {
            const int h = kTile - 2 * halo;
            VisitShape v;
            v.tile_w = w;
            v.halo = halo;
            v.tiles_x = (nx + w - 1) / w;
            v.tiles_y = ny <= kTile ? 1 : (ny - 2 * halo + h - 1) / h;
            const int by_rows = halo / r + 1, by_cols = 8 / r;
            v.depth = by_rows < by_cols ? by_rows : by_cols;
            v.visits = steps > 0 ? (steps - 1) / v.depth + 1 : 0;
            const double n = (double)v.tiles_x * v.tiles_y / sms;
            if (halo == 2 && (r == 1 || n <= 4.0)) continue;
            const double t = (double)steps / v.visits;
            const double m = 61.7 * (w / 16 + 1) * (2 * r + 1) - 50.0, l = 586.0 + 8.0 * w;
            const double per_cta = std::max(std::ceil(v.visits * n), v.visits * (n + 0.42 * (std::ceil(n) - n)));
            const double chain = v.visits * (t * (m + l) + 3417.0);
            const double slots = per_cta * (t * std::max(m, 0.575 * (m + l)) + 243.0);
            const double cost = std::max(chain, slots);
            if (!best.visits || cost < best_cost) {
                best = v;
                best_cost = cost;
            }
        }
    }
    return best;
}

cudaError_t visit_prepare(int stencil) {
    switch (stencil) {
    case TCS_STAR2D1R: return prepare_visit<TCS_STAR2D1R>();
    case TCS_STAR2D2R: return prepare_visit<TCS_STAR2D2R>();
    case TCS_BOX2D1R: return prepare_visit<TCS_BOX2D1R>();
    case TCS_BOX2D2R: return prepare_visit<TCS_BOX2D2R>();
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_tc_f16_visits(const GridGeom &g, int stencil, const float *B, uint16_t *in,
                                 uint16_t *out, int steps, const VisitShape &v,
                                 unsigned *counters, cudaStream_t s, int sms) {
    if (steps < 1 || v.visits < 1 || !counters) return cudaErrorInvalidValue;
    VisitParams p;
    p.g = g;
    p.tiles_x = v.tiles_x;
    p.tiles_y = v.tiles_y;
    p.halo = v.halo;
    p.map_rows = v.halo == 2 ? 4 : 8;  // tile rows start at multiples of 124, 120 or 112
    p.visits = v.visits;
    p.base = steps / v.visits;
    p.extra = steps % v.visits;
    // A tile's finished warps are counted on its slot after they have let the
    // slot's next tile start: were that one's visit a single step and published
    // too, a fast warp could be counted for it before a slow one for this tile.
    // So single steps only in the last visit, which publishes nothing; a depth of
    // two and more gives no others.  (Counting by stage, before the stage is given
    // back, allows them: 8196² box2d2r 0.2 % slower.)
    if (p.base < 2 && p.visits - p.extra > 1) return cudaErrorInvalidValue;
    p.ended = counters;
    p.done = counters + kRowCounterStride;  // a line of its own each
    p.plane[0] = in;
    p.plane[1] = out;
    cudaError_t e = encode_panel_map(in, g.p16, &p.map[0], v.tile_w / 8 + 2, p.map_rows);
    if (e == cudaSuccess) e = encode_panel_map(out, g.p16, &p.map[1], v.tile_w / 8 + 2, p.map_rows);
    if (e != cudaSuccess) return e;
    const int n = 2 * stencil_r(stencil) + 1;
    for (int k = 0; k < 25; k++) p.coef[k] = k < n * n ? B[k] : 0.0f;
    switch (stencil) {
    case TCS_STAR2D1R: return launch_visit<TCS_STAR2D1R>(p, v.tile_w, sms, s);
    case TCS_STAR2D2R: return launch_visit<TCS_STAR2D2R>(p, v.tile_w, sms, s);
    case TCS_BOX2D1R: return launch_visit<TCS_BOX2D1R>(p, v.tile_w, sms, s);
    case TCS_BOX2D2R: return launch_visit<TCS_BOX2D2R>(p, v.tile_w, sms, s);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t visit_error_word(int **word) {
    return cudaGetSymbolAddress(reinterpret_cast<void **>(word), g_visit_error);
}

}  // namespace tcs
