// CUDA-core sweep kernels (the counterpart of the reference's baseline/
// kernel_*.cu `kernel_run`, rebuilt for GB300).
//
// One CTA per tile of 128 rows by 16 panels (128 FP16 or 64 FP32 columns).
// One thread stages the tile's rows, with four halo rows above and below,
// and the panel on each side, as 18 bulk copies (a panel's rows are one
// contiguous run) into shared memory, where runs sit 2192 bytes apart so
// that the 16 panels of a row fall on different banks.  Four warps then
// take 32 rows each.  Lane l owns half a panel: cells [x_l, x_l + H) with
// H = 4 (FP16) or 2 (FP32), 8 bytes of each panel row; horizontal halo
// cells come from lanes l-1 and l+1 by shuffle (the same shuffle for every
// lane) and, for the outer lanes, from the side panels' runs.  The vertical
// taps come from a register window of six rows, two rows per step.  Each
// warp first reads the rows it shares with its neighbours, then writes its
// results over its own rows of the stage, and one thread stores the 16
// panels' rows back with 16 bulk copies.  Both directions go by the copy
// engine, not the load/store pipeline, which was this kernel's limit when
// it moved its rows through L1 (79 % of the L1 throughput at 0.43 of HBM;
// measured on GB300 at 8196², us per step, L1 -> bulk loads -> bulk loads
// and stores: star2d1r FP16 111.7 -> 73.9 -> 61.4, FP32 182 -> 124 -> 97.6).
// Five such CTAs fit an SM.  (Persistent CTAs walking tiles through two or
// three stages measured no faster.)  A warp whose rows and whose tile's
// columns all lie in the update rectangle (most warps of a large grid) runs
// its rows with no per-row tests and immediate row offsets; with that,
// star2d1r FP16 runs 57.9 -> 49.5 us per step at 8196², star2d2r 66.3 ->
// 55.0, box2d2r 95.1 -> 83.5 (FP32 97.7 -> 87.3, 109.4 -> 90.9, 160.1 -> 134.5),
// from the row overhead each lane carried: about 62 instructions per row
// beside the FMAs.
//
// Arithmetic follows gold's tap order (common/gold_*.cpp):
//  - FP16 storage: acc = fmaf chain from 0, FP32 coefficients, RNE to FP16.
//  - FP32 storage: gold's own unfused products and sums (__fmul_rn/__fadd_rn),
//    so the result is bit-identical to gold compiled without FMA contraction.
#include <type_traits>

#include "tcs_device.cuh"
#include "tcs_internal.h"

namespace tcs {

__device__ int g_cc_error = 0;  // first give-up code of a CUDA-core launch

namespace {

constexpr int kCcTileRows = 128;
constexpr int kCcPanels = 16;                          // panels a tile computes
constexpr int kCcRunRows = kCcTileRows + 8;            // staged rows: 4 above, 4 below
constexpr int kCcRunBytes = kCcRunRows * 16;           // one panel's run
constexpr int kCcRunStride = kCcRunBytes + 16;         // next panel 4 banks on
constexpr int kCcWarps = 4;                            // warps per CTA
constexpr int kCcWarpRows = kCcTileRows / kCcWarps;    // rows per warp (even)
constexpr int kCcRunsOffset = 128;                     // after the mbarrier
constexpr int kCcSmem = kCcRunsOffset + (kCcPanels + 2) * kCcRunStride;
static_assert(kCcWarpRows % 2 == 0, "two rows per step");

struct CcParams {
    GridGeom g;
    PlaneGeom p;   // plane of this precision
    int nchunks;   // panels that hold grid cells
    int tiles_x;
    int n_tiles;
    float neg_zero;
};

__device__ __forceinline__ uint2 lds_v2(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts_v2(uint32_t addr, uint2 v) {
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(v.x), "r"(v.y) : "memory");
}
// 1-D bulk copy of `bytes` (a multiple of 16) from shared to global memory,
// both addresses 16-byte aligned, in this thread's bulk group.
__device__ __forceinline__ void bulk_store(void *dst, const void *src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(
                     reinterpret_cast<uint64_t>(dst)),
                 "r"(smem_u32(src)), "r"(bytes)
                 : "memory");
}
// Waits until this thread's bulk stores have read their shared memory.
__device__ __forceinline__ void bulk_store_commit_and_wait_read() {
    asm volatile("cp.async.bulk.commit_group;\n\tcp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}

// One lane's part of a tile: PPL = 1: half a panel's cells of every row (a
// warp covers 16 panels), PPL = 2: a whole panel's (32 panels).  Windows,
// products and stores are the same for every form of the sweep.
template <int S, bool F32, int PPL>
struct CcLane {
    static constexpr int R = stencil_r(S);
    static constexpr int V = F32 ? 4 : 8;            // cells per panel row
    static constexpr int H = V / 2 * PPL;            // cells per lane
    static constexpr int OW = 2 * PPL;               // its 32-bit words
    static constexpr int WPC = F32 ? 1 : 2;          // cells per 32-bit word
    static constexpr int HW = (R + WPC - 1) / WPC;   // halo words each side
    static constexpr int HC = HW * WPC;              // halo cells each side
    static constexpr int W = H + 2 * R;              // window columns of a lane
    static constexpr int NT = tap_count(S);
    static constexpr bool BOX = stencil_box(S);
    static constexpr int PANELS = 16 * PPL;          // of a warp's row
    // Taps of odd dx in scalar operations: their cell pairs straddle two
    // register pairs, and the two moves that align one cost more than packing
    // saves (8196² visits, us per step, FP16 star2d1r 30.9 -> 27.9, star2d2r 45.0
    // -> 42.7, box2d1r 41.3 -> 38.8; FP32 star2d1r 37.5 -> 35.4, star2d2r 72.0 ->
    // 67.4, box2d2r 130 -> 122 a single step).  The FP32 box2d1r's single steps
    // are faster packed (24.3 against 25.1 at 4096²).
    static constexpr bool ODD_SCALAR = !(F32 && BOX && R == 1);
    using T = typename std::conditional<F32, float, uint16_t>::type;

    // shared address of tile row 0 of this lane's cells, and of the outer
    // lanes' edge words in the side panels' runs
    uint32_t own0, edge0;
    bool is_l, is_r;
    float neg0;  // -0, a run-time value (compute)

    __device__ __forceinline__ void init(uint32_t runs, int lane, float neg_zero) {
        neg0 = neg_zero;
        own0 = PPL == 2 ? runs + (1 + lane) * kCcRunStride + 4 * 16
                        : runs + (1 + (lane >> 1)) * kCcRunStride + 4 * 16 + (lane & 1) * 8;
        edge0 = lane == 0 ? runs + 4 * 16 + (V - HC) * (uint32_t)sizeof(T)
                          : runs + (PANELS + 1) * kCcRunStride + 4 * 16;
        is_l = lane == 0;
        is_r = lane == 31;
    }

    // A row's words: this lane's own and (the outer lanes') halo words in the
    // side panels' runs.  Every lane loads one of the latter (the inner lanes
    // all the same word, discarded), so the warp does not branch.
    struct Raw {
        uint32_t own[OW], e[HW];
    };
    __device__ __forceinline__ void fetch(uint32_t r16, Raw &x) const {
        if constexpr (PPL == 2) {
            const uint4 v = lds128(own0 + r16);
            x.own[0] = v.x; x.own[1] = v.y; x.own[2] = v.z; x.own[3] = v.w;
        } else {
            const uint2 v = lds_v2(own0 + r16);
            x.own[0] = v.x; x.own[1] = v.y;
        }
#pragma unroll
        for (int k = 0; k < HW; k++) x.e[k] = lds_u32(edge0 + r16 + 4 * k);
    }
    // Its window columns [0, W): cells xl-R .. xl+H+R-1.
    __device__ __forceinline__ void expand(const Raw &x, float (&w)[W]) const {
        const uint32_t (&own)[OW] = x.own;
        uint32_t left[HW], right[HW];
#pragma unroll
        for (int k = 0; k < HW; k++) {
            left[k] = __shfl_up_sync(0xffffffffu, own[OW - HW + k], 1);
            right[k] = __shfl_down_sync(0xffffffffu, own[k], 1);
            left[k] = is_l ? x.e[k] : left[k];
            right[k] = is_r ? x.e[k] : right[k];
        }
        float cells[HC + H + HC];
        if constexpr (F32) {
#pragma unroll
            for (int k = 0; k < HW; k++) {
                cells[k] = __uint_as_float(left[k]);
                cells[HC + H + k] = __uint_as_float(right[k]);
            }
#pragma unroll
            for (int k = 0; k < OW; k++) cells[HC + k] = __uint_as_float(own[k]);
        } else {
            const float2 l = unpack_half2(left[0]), rr = unpack_half2(right[0]);
            cells[0] = l.x; cells[1] = l.y;
#pragma unroll
            for (int k = 0; k < OW; k++) {
                const float2 a = unpack_half2(own[k]);
                cells[2 + 2 * k] = a.x;
                cells[3 + 2 * k] = a.y;
            }
            cells[2 + H] = rr.x; cells[3 + H] = rr.y;
        }
#pragma unroll
        for (int k = 0; k < W; k++) w[k] = cells[HC - R + k];
    }
    // The window columns of the stage row at byte offset r16 = (y - Y0) * 16.
    __device__ __forceinline__ void to_window(uint32_t r16, float (&w)[W]) const {
        Raw x;
        fetch(r16, x);
        expand(x, w);
    }

    // Rows y0, y0+1 from the window rows y0-2 .. y0+3, held as three row
    // pairs p0, p1, p2, in gold's tap order.
    template <bool PACK = true>
    __device__ __forceinline__ void compute(const TapCoeffs &c, const float (&p0)[2][W],
                                            const float (&p1)[2][W], const float (&p2)[2][W],
                                            float (&acc)[2][H]) const {
        auto row = [&](int wr) -> const float (&)[W] {
            return wr < 2 ? p0[wr] : wr < 4 ? p1[wr - 2] : p2[wr - 4];
        };
        if constexpr (PACK && !(F32 && PPL == 2 && BOX && R == 1)) {
            // packed FP32 operations on cell pairs, taps outside the rows so
            // that one coefficient pair serves both rows; each lane rounds as
            // the scalar operation does, so the bits are the same (measured
            // at 8196², us per step, one step per launch: star2d1r 61.4 ->
            // 57.9 and box2d1r 66.4 -> 63.4 before the interior path,
            // star2d2r 55.0 -> 51.8 after it; the FP16 box2d2r since its odd
            // taps are scalar: 80.9 -> 73.3, 4096² 25.7 -> 21.8, though not on
            // visits of 64-row tiles, 700² 2.50 -> 2.62).
            // FP32 storage wants gold's unfused products: x c + -0 rounds as
            // x c does, and with the -0 a run-time value the compiler cannot
            // make one fused operation of it and the sum (it does of a packed
            // product and sum, .rn or not).  Scalar -> packed, one step per
            // launch at 4096²: star2d1r 23.3 -> 22.2, box2d1r 26.3 -> 24.2,
            // box2d2r 39.6 -> 37.0; whole-panel lanes of the visit kernel at
            // 8196²: star2d1r 39.3 -> 37.9, star2d2r 69.2 -> 65.0, box2d2r
            // 185 -> 148, but box2d1r 58.1 -> 60.8, which stays scalar.
            float2 a2[2][H / 2];
#pragma unroll
            for (int k = 0; k < NT; k++) {
                const int dy = tap_dy(S, k), dx = tap_dx(S, k);
                const float2 cc = make_float2(c.c[k], c.c[k]);
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const float (&x)[W] = row(2 + q + dy);
#pragma unroll
                    for (int i = 0; i < H; i += 2) {
                        const float2 x2 = make_float2(x[R + i + dx], x[R + i + 1 + dx]);
                        const float2 a = k == 0 ? make_float2(0.0f, 0.0f) : a2[q][i / 2];
                        if (ODD_SCALAR && dx % 2 != 0) {
                            // the pair straddles two register pairs
                            if constexpr (F32) {
                                const float2 p = make_float2(__fmul_rn(x2.x, cc.x), __fmul_rn(x2.y, cc.x));
                                a2[q][i / 2] = k == 0 && !BOX ? p : make_float2(__fadd_rn(a.x, p.x), __fadd_rn(a.y, p.y));
                            } else {
                                a2[q][i / 2] = make_float2(fmaf(x2.x, cc.x, a.x), fmaf(x2.y, cc.x, a.y));
                            }
                            continue;
                        }
                        if constexpr (F32) {
                            const float2 p = __ffma2_rn(x2, cc, make_float2(neg0, neg0));
                            a2[q][i / 2] = k == 0 && !BOX ? p : __fadd2_rn(a, p);
                        } else {
                            a2[q][i / 2] = __ffma2_rn(x2, cc, a);
                        }
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < 2; q++)
#pragma unroll
                for (int i = 0; i < H; i += 2) {
                    acc[q][i] = a2[q][i / 2].x;
                    acc[q][i + 1] = a2[q][i / 2].y;
                }
            return;
        }
        // scalar chains: the FP16 box2d2r of short tiles, and the FP32 box2d1r
        // of whole-panel lanes
#pragma unroll
        for (int q = 0; q < 2; q++) {
            constexpr int dy0 = tap_dy(S, 0), dx0 = tap_dx(S, 0);
            const float (&x0)[W] = row(2 + q + dy0);
#pragma unroll
            for (int i = 0; i < H; i++) {
                if constexpr (F32) acc[q][i] = BOX ? __fadd_rn(0.0f, __fmul_rn(x0[R + i + dx0], c.c[0]))
                                                   : __fmul_rn(x0[R + i + dx0], c.c[0]);
                else acc[q][i] = fmaf(x0[R + i + dx0], c.c[0], 0.0f);
            }
#pragma unroll
            for (int k = 1; k < NT; k++) {
                const int dy = tap_dy(S, k), dx = tap_dx(S, k);
                const float (&x)[W] = row(2 + q + dy);
#pragma unroll
                for (int i = 0; i < H; i++) {
                    if constexpr (F32) acc[q][i] = __fadd_rn(acc[q][i], __fmul_rn(x[R + i + dx], c.c[k]));
                    else acc[q][i] = fmaf(x[R + i + dx], c.c[k], acc[q][i]);
                }
            }
        }
    }

    __device__ __forceinline__ void store_row(uint32_t r16, const float (&a)[H]) const {
        uint32_t w[OW];
#pragma unroll
        for (int k = 0; k < OW; k++) {
            if constexpr (F32) w[k] = __float_as_uint(a[k]);
            else w[k] = pack_half2(a[2 * k], a[2 * k + 1]);
        }
        if constexpr (PPL == 2) sts128(own0 + r16, make_uint4(w[0], w[1], w[2], w[3]));
        else sts_v2(own0 + r16, make_uint2(w[0], w[1]));
    }
};

template <int S, bool F32>
__global__ void __launch_bounds__(kCcWarps * 32, 5)
    cc_sweep_kernel(const void *__restrict__ in_, void *__restrict__ out_, CcParams p,
                    TapCoeffs c) {
    using L = CcLane<S, F32, 1>;
    constexpr int R = L::R, V = L::V, H = L::H, W = L::W;
    using T = typename L::T;
    const T *__restrict__ in = static_cast<const T *>(in_);
    T *__restrict__ out = static_cast<T *>(out_);

    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem);
    const uint32_t runs = smem_u32(smem + kCcRunsOffset);

    const int tile = blockIdx.x;
    const int tx = tile % p.tiles_x, ty = tile / p.tiles_x;
    const int Y0 = ty * kCcTileRows;
    const int chunk0 = tx * kCcPanels;  // first panel of the tile
    const ptrdiff_t nyp = p.p.nyp;

    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    // the previous step's CTAs may still run: planes only after pdl_wait
    pdl_wait();
    if (threadIdx.x == 0) {
        // staged run q = plane panel chunk0 + q (the panel left of chunk0 is
        // the plane's panel chunk0), plane rows Y0 .. Y0+135 (grid rows
        // Y0-4 .. Y0+131); runs past the plane are not staged and never read
        // by a cell of the update rectangle
        const int nq = min(kCcPanels + 2, p.p.npan - chunk0);
        mbar_arrive_expect_tx(bar, (uint32_t)(nq * kCcRunBytes));
        for (int q = 0; q < nq; q++)
            bulk_load(smem + kCcRunsOffset + q * kCcRunStride,
                      in + ((ptrdiff_t)(chunk0 + q) * nyp + Y0) * V, kCcRunBytes, bar);
    }
    __syncthreads();
    if (!__syncthreads_and(mbar_wait(bar, 0, &g_cc_error))) {  // every thread leaves, or none
        if (threadIdx.x == 0) record_error(&g_cc_error, kErrWaitFull);
        return;
    }

    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int chunk = chunk0 + (lane >> 1);  // this lane's panel
    const bool active = chunk < p.nchunks;
    const int xl = chunk * V + (lane & 1) * H;  // first column this lane computes
    const int ys = Y0 + warp * kCcWarpRows;
    const int ye = min(ys + kCcWarpRows, p.g.ny);
    const bool has_rows = ys < p.g.ny;  // the same for the whole warp
    L ln;
    ln.init(runs, lane, p.neg_zero);
    auto to_window = [&](uint32_t r16, float (&w)[W]) { ln.to_window(r16, w); };
    auto compute = [&](const float (&p0)[2][W], const float (&p1)[2][W], const float (&p2)[2][W],
                       float (&acc)[2][H]) { ln.compute(c, p0, p1, p2, acc); };
    auto store_row = [&](uint32_t r16, const float (&a)[H]) { ln.store_row(r16, a); };

    // this lane's cells of the update rectangle
    const bool cols_in = xl >= p.g.x0 && xl + H <= p.g.x1;
    // A warp whose 32 rows and whose tile's 128 columns all lie in the update
    // rectangle takes a path with no per-row checks and immediate row offsets
    // (the general path tests rows, columns and the grid's end on every row).
    const bool fast = __all_sync(0xffffffffu, active && cols_in) && ys >= p.g.y0 &&
                      ys + kCcWarpRows <= p.g.y1;

    // Results go back into the stage, over the rows they replace, and leave
    // by bulk stores: so each warp first reads the rows it shares with its
    // neighbours (two above its rows, two below), and only then, after a
    // barrier, overwrites its own rows.
    // window: pair slot j holds rows (y0-2+2j, y0-1+2j), rotated over steps
    const uint32_t rs = (uint32_t)(ys - Y0) * 16;  // this warp's first row
    float win[3][2][W];
    float below[2][W];  // rows ye, ye+1
    if (has_rows) {
        to_window(rs - 2 * 16, win[0][0]);
        to_window(rs - 1 * 16, win[0][1]);
        to_window(rs, win[1][0]);
        to_window(rs + 16, win[1][1]);
        to_window((uint32_t)(ye - Y0) * 16, below[0]);
        to_window((uint32_t)(ye + 1 - Y0) * 16, below[1]);
    }
    __syncthreads();

    if (fast) {
        // 16 row pairs: five rounds of three (the window's three slots), then
        // the last pair, whose next rows are the next warp's, read before the
        // barrier
        static_assert(kCcWarpRows == 32, "five rounds of three row pairs and one more");
        uint32_t r = rs;
        for (int round = 0; round < 5; round++, r += 6 * 16) {
#pragma unroll
            for (int u = 0; u < 3; u++) {
                float (&n)[2][W] = win[(u + 2) % 3];
                to_window(r + (2 * u + 2) * 16, n[0]);
                to_window(r + (2 * u + 3) * 16, n[1]);
                float acc[2][H];
                compute(win[u], win[(u + 1) % 3], n, acc);
                store_row(r + 2 * u * 16, acc[0]);
                store_row(r + (2 * u + 1) * 16, acc[1]);
            }
        }
        float acc[2][H];
        compute(win[0], win[1], below, acc);
        store_row(r, acc[0]);
        store_row(r + 16, acc[1]);
    } else if (has_rows) {
        for (int y = ys; y < ye; y += 6) {
#pragma unroll
            for (int u = 0; u < 3; u++) {
                const int y0 = y + 2 * u;
                if (y0 < ye) {
                    float (&n)[2][W] = win[(u + 2) % 3];
                    // rows from ye on belong to the next warp, which may have
                    // written them by now, unless the grid ends at ye (then
                    // no warp writes them, and a warp of an odd row count
                    // reads up to ye + 2)
                    if (y0 + 2 < ye || ye == p.g.ny) {
                        to_window((uint32_t)(y0 + 2 - Y0) * 16, n[0]);
                        to_window((uint32_t)(y0 + 3 - Y0) * 16, n[1]);
                    } else {
#pragma unroll
                        for (int k = 0; k < W; k++) {
                            n[0][k] = below[0][k];
                            n[1][k] = below[1][k];
                        }
                    }
                    float acc[2][H];
                    compute(win[u], win[(u + 1) % 3], n, acc);
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        // cells outside the update rectangle keep their value
                        const int yy = y0 + q;
                        const bool row_in = yy >= p.g.y0 && yy < p.g.y1;
                        if (!(row_in && cols_in)) {
#pragma unroll
                            for (int i = 0; i < H; i++) {
                                const int x = xl + i;
                                if (!(row_in && x >= p.g.x0 && x < p.g.x1))
                                    acc[q][i] = win[(u + 1) % 3][q][R + i];
                            }
                        }
                        if (active && yy < ye) store_row((uint32_t)(yy - Y0) * 16, acc[q]);
                    }
                }
            }
        }
    }
    // the stage's rows Y0 .. Y0+127 of the 16 panels (results, and the input
    // where nothing was computed: rows past the grid, panels past its cells)
    // to the output plane
    fence_proxy_async_smem();
    __syncthreads();
    // the next step may launch once every CTA is here: signalled at the start
    // instead, CTAs of several later steps filled the SMs while they waited,
    // and a step of about one tile per SM ran slower (measured on GB300,
    // 1602² star2d1r FP16: 6.8 -> 8.6 us per step)
    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        const int nq = min(kCcPanels + 1, p.p.npan - chunk0);
        for (int q = 1; q < nq; q++)
            bulk_store(out + ((ptrdiff_t)(chunk0 + q) * nyp + Y0 + 4) * V,
                       smem + kCcRunsOffset + q * kCcRunStride + 4 * 16, kCcTileRows * 16);
        bulk_store_commit_and_wait_read();
    }
}

// ------------------------------------------- several steps per tile visit ---
// A tile of 128 rows by 16 PPL panels is staged once, stepped T times in
// shared memory and stored once; the rows and columns whose neighbourhood was
// not all staged shrink by R a step and hold garbage (no valid cell reads it,
// and each cell is computed by itself, whatever the values).  Tiles overlap
// by `halo` rows (4 or 8) and one panel (8 or 4 cells) on each side, so T =
// halo / R + 1, halo = 4 for FP32: tile (ty, tx) starts at row (128 - 2 halo)
// ty and panel (PANELS - 2) tx and owns all but that margin (up to the grid's
// edge for the outer tiles).  Visits of one launch depend on each
// other by tiles: a tile's visit j needs visit j-1 of itself and its eight
// neighbours, which hold its input and last read the plane it overwrites; one
// counter per tile, polled by nine lanes.  The launch is cooperative.
//
// WARPS warps take 128 / WARPS rows each: with few tiles per SM a step's time
// is the length of a warp's row sequence, with many the rows read twice at the
// warps' edges count.  Two barriers a step: between reading the rows a warp
// shares with its neighbours and overwriting them, and after.
template <int PPL>
constexpr int cv_smem() { return kCcRunsOffset + (16 * PPL + 2) * kCcRunStride; }

struct CvParams {
    GridGeom g;
    PlaneGeom p;
    int nchunks, tiles_x, tiles_y;
    int halo;                 // rows given up at the top and bottom: 4 or 8
    int visits, base, extra;  // visit j takes base + (j < extra) steps
    float neg_zero;
    void *plane[2];           // visit j reads plane[j & 1]
    unsigned *ended, *done;   // CTAs at their end; [tiles] finished visits (zeros)
};

// The last CTA whose tiles need no counter any more leaves them zero for the
// next launch: as leave_counters of sweep_visit.cu.  Called by a whole warp.
__device__ __forceinline__ void cv_leave_counters(const CvParams &p, int lane) {
    if (p.visits < 2) return;
    int last = 0;
    if (lane == 0) {
        fence_acq_rel_gpu();
        last = atomicAdd(p.ended, 1u) == gridDim.x - 1;
        fence_acq_rel_gpu();
    }
    if (!__shfl_sync(0xffffffffu, last, 0)) return;
    __syncwarp();
    for (int t = lane; t < p.tiles_x * p.tiles_y; t += 32) p.done[t] = 0;
    if (lane == 0) *p.ended = 0;
}

template <int S, bool F32, int PPL, int WARPS, int TR, int CTAS>
__global__ void __launch_bounds__(WARPS * 32, CTAS)
    cc_visit_kernel(const __grid_constant__ CvParams p, const __grid_constant__ TapCoeffs c) {
    using L = CcLane<S, F32, PPL>;
    constexpr int V = L::V, H = L::H, W = L::W, R = L::R;
    constexpr int PANELS = L::PANELS;
    constexpr int ROWS = TR / WARPS, PAIRS = ROWS / 2;  // of a warp
    using T = typename L::T;
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(bar + 1);
    const uint32_t runs = smem_u32(smem + kCcRunsOffset);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n_tiles = p.tiles_x * p.tiles_y, n_items = p.visits * n_tiles;
    const ptrdiff_t nyp = p.p.nyp;
    L ln;
    ln.init(runs, lane, p.neg_zero);
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        *abort_flag = 0;
        fence_mbar_init();
    }
    __syncthreads();

    uint32_t phase = 0;
    bool counted = false;  // (warp 0)
    for (int k = blockIdx.x; k < n_items; k += gridDim.x, phase ^= 1) {
        const int visit = k / n_tiles, tile = k - visit * n_tiles;
        const int ty = tile / p.tiles_x, tx = tile - ty * p.tiles_x;
        const int Yb = ty * (TR - 2 * p.halo);
        const int chunk0 = tx * (PANELS - 2);  // first panel of the tile
        const int rows = min(TR + 8, p.p.nyp - Yb);
        if (warp == 0) {
            bool ok = true;
            if (visit > 0) {
                const int y = ty + lane / 3 - 1, x = tx + lane % 3 - 1;
                const bool mine = lane < 9 && y >= 0 && y < p.tiles_y && x >= 0 && x < p.tiles_x;
                const unsigned *ctr = p.done + (mine ? y * p.tiles_x + x : 0);
                const uint64_t t0 = global_timer_ns();
                for (int n = 1; !__all_sync(0xffffffffu, !mine || ld_acquire(ctr) >= (unsigned)visit); n++) {
                    if (n % 32) continue;
                    const bool stop = *(volatile int *)&g_cc_error != 0 || global_timer_ns() - t0 > kWaitLimitNs;
                    if (__any_sync(0xffffffffu, stop)) {
                        ok = false;
                        break;
                    }
                }
                __syncwarp();  // all lanes' acquires before lane 0's copies (a vote orders no memory)
            }
            // no counter is read or added to for this CTA's other tiles any more
            if (ok && k + (int)gridDim.x >= n_items) {
                cv_leave_counters(p, lane);
                counted = true;
            }
            if (lane == 0) {
                if (ok) {
                    // staged run q = panel chunk0 - 1 + q, plane rows Yb .. (grid
                    // rows Yb-4 ..); what lies past the plane is not staged and
                    // never read by a cell of the update rectangle
                    fence_proxy_async_global();  // other SMs stored it
                    const T *in = static_cast<const T *>(p.plane[visit & 1]);
                    const int nq = min(PANELS + 2, p.p.npan - chunk0);
                    mbar_arrive_expect_tx(bar, (uint32_t)(nq * rows * 16));
                    for (int q = 0; q < nq; q++)
                        bulk_load(smem + kCcRunsOffset + q * kCcRunStride,
                                  in + ((ptrdiff_t)(chunk0 + q) * nyp + Yb) * V, (uint32_t)(rows * 16), bar);
                } else {
                    record_error(&g_cc_error, kErrWaitDep);
                    *abort_flag = 1;
                }
            }
        }
        // every thread leaves, or none
        const bool here = mbar_wait(bar, phase, abort_flag);
        if (!__syncthreads_and(here)) {
            if (threadIdx.x == 0) record_error(&g_cc_error, kErrWaitFull);
            break;
        }

        const int chunk = chunk0 + (PPL == 2 ? lane : lane >> 1);  // this lane's panel
        const bool active = chunk < p.nchunks;
        const int xl = chunk * V + (PPL == 2 ? 0 : (lane & 1) * H);  // its first column
        const int ys = Yb + warp * ROWS;
        const bool cols_in = xl >= p.g.x0 && xl + H <= p.g.x1;
        // fast: all of the warp's cells lie in the update rectangle; else a
        // cell is stored, or kept, by its row and its column's bit
        const bool fast = __all_sync(0xffffffffu, active && cols_in) && ys >= p.g.y0 && ys + ROWS <= p.g.y1;
        uint32_t cells = 0;
#pragma unroll
        for (int i = 0; i < H; i++) cells |= (xl + i >= p.g.x0 && xl + i < p.g.x1 ? 1u : 0u) << i;
        const uint32_t rs = (uint32_t)(warp * ROWS) * 16;  // this warp's first row
        const int steps = p.base + (visit < p.extra ? 1 : 0);
        // window: pair slot j holds rows (y0-2+2j, y0-1+2j), rotated; the next
        // pair's words are fetched while a pair is computed
        float win[3][2][W];
        typename L::Raw next[2], below[2];
        auto pairs = [&](auto all) {
#pragma unroll
            for (int u = 0; u < PAIRS; u++) {
                float (&n)[2][W] = win[(u + 2) % 3];
                if (u < PAIRS - 1) {
                    ln.expand(next[0], n[0]);
                    ln.expand(next[1], n[1]);
                    if (u < PAIRS - 2) {
                        ln.fetch(rs + (2 * u + 4) * 16, next[0]);
                        ln.fetch(rs + (2 * u + 5) * 16, next[1]);
                    }
                } else {
                    ln.expand(below[0], n[0]);
                    if (R == 2) ln.expand(below[1], n[1]);
                }
                const float (&own)[2][W] = win[(u + 1) % 3];
                float acc[2][H];
                ln.template compute<F32 || S != TCS_BOX2D2R || TR == kCcTileRows>(c, win[u % 3], own, n, acc);
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    if constexpr (decltype(all)::value) {
                        ln.store_row(rs + (2 * u + q) * 16, acc[q]);
                    } else {
                        const int y = ys + 2 * u + q;
                        if (y >= p.g.y0 && y < p.g.y1 && cells != 0) {
#pragma unroll
                            for (int i = 0; i < H; i++)
                                if (!((cells >> i) & 1u)) acc[q][i] = own[q][R + i];
                            ln.store_row(rs + (2 * u + q) * 16, acc[q]);
                        }
                    }
                }
            }
        };
        for (int t = 0; t < steps; t++) {
            if (R == 2) ln.to_window(rs - 2 * 16, win[0][0]);
            ln.to_window(rs - 1 * 16, win[0][1]);
            ln.to_window(rs, win[1][0]);
            ln.to_window(rs + 16, win[1][1]);
            ln.fetch(rs + ROWS * 16, below[0]);
            if (R == 2) ln.fetch(rs + (ROWS + 1) * 16, below[1]);
            ln.fetch(rs + 2 * 16, next[0]);
            ln.fetch(rs + 3 * 16, next[1]);
            __syncthreads();
            if (fast) pairs(std::true_type{});
            else pairs(std::false_type{});
            if (t + 1 < steps) __syncthreads();
        }
        // the owned rows and panels to the other plane
        fence_proxy_async_smem();
        __syncthreads();
        if (threadIdx.x == 0) {
            T *out = static_cast<T *>(p.plane[(visit & 1) ^ 1]);
            const int top = ty == 0 ? 0 : p.halo;  // tile rows [top, bottom)
            const int bottom = min(ty == p.tiles_y - 1 ? TR : TR - p.halo, rows - 4);
            const int q0 = tx == 0 ? 1 : 2;
            const int q1 = min(tx == p.tiles_x - 1 ? PANELS + 1 : PANELS, p.p.npan - chunk0);
            for (int q = q0; q < q1; q++)
                bulk_store(out + ((ptrdiff_t)(chunk0 + q) * nyp + Yb + 4 + top) * V,
                           smem + kCcRunsOffset + q * kCcRunStride + (4 + top) * 16,
                           (uint32_t)((bottom - top) * 16));
            bulk_store_commit_and_wait_read();
            if (visit + 1 < p.visits) {
                // the copies have been written, not only read, before the tile
                // is published
                asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
                fence_proxy_async_global();
                red_release_add(p.done + tile, 1u);
            }
        }
    }
    // an early exit did not leave the counters
    if (!counted && warp == 0) cv_leave_counters(p, lane);
}

template <int S, bool F32, int PPL, int WARPS, int TR, int CTAS>
cudaError_t launch_cv(const CvParams &p, const TapCoeffs &c, int sms, cudaStream_t s) {
    static int per_sm = 0;
    if (!per_sm) {
        cudaError_t e = cudaFuncSetAttribute(cc_visit_kernel<S, F32, PPL, WARPS, TR, CTAS>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, cv_smem<PPL>());
        int n = 0;
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, cc_visit_kernel<S, F32, PPL, WARPS, TR, CTAS>,
                                                              WARPS * 32, cv_smem<PPL>());
        if (e != cudaSuccess) return e;
        if (n < 1) return cudaErrorInvalidConfiguration;
        per_sm = n;
    }
    const int tiles = p.tiles_x * p.tiles_y;
    if (!tiles) return cudaSuccess;  // preparation only
    cudaLaunchConfig_t cfg = {};
    // (up to three tiles per SM, two CTAs each: where three fit, some SMs would
    // have three tiles' steps and others one or two; FP16 2048² star2d1r 3.31 ->
    // 2.94 us per step, box2d1r 4.44 -> 3.88, FP32 1500² box2d1r 3.72 -> 3.32)
    const int ctas = (WARPS == 8 && tiles <= 3 * sms && per_sm > 2 ? 2 : per_sm) * sms;
    cfg.gridDim = dim3((unsigned)(tiles < ctas ? tiles : ctas));
    cfg.blockDim = dim3(WARPS * 32);
    cfg.dynamicSmemBytes = cv_smem<PPL>();
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, cc_visit_kernel<S, F32, PPL, WARPS, TR, CTAS>, p, c);
}

template <int S, bool F32>
cudaError_t dispatch_cv(const CcVisitShape &v, const CvParams &p, const TapCoeffs &c, int sms, cudaStream_t s) {
    if (v.ppl == 2) {
        // Where a whole-panel FP32 lane fits 80 registers, 24 warps on an SM
        // instead of 16, from three tiles per SM on (us per step: 8196²
        // star2d1r 39.7 -> 37.5, box2d1r 60.0 -> 55.9, 3000² 6.07 -> 5.80, 8.75
        // -> 8.42); with fewer tiles the tighter code is the slower one (2500²
        // box2d1r 6.28 -> 6.59).
        if constexpr (F32 && (S == TCS_STAR2D1R || S == TCS_BOX2D1R)) {
            const int tiles = p.tiles_x * p.tiles_y;
            if (tiles > 3 * sms) return launch_cv<S, F32, 2, 8, 128, 3>(p, c, sms, s);
            if (!tiles) {  // preparation of both
                const cudaError_t e = launch_cv<S, F32, 2, 8, 128, 3>(p, c, sms, s);
                if (e != cudaSuccess) return e;
            }
        }
        return launch_cv<S, F32, 2, 8, 128, 2>(p, c, sms, s);
    }
    if (v.warps == 8) return launch_cv<S, F32, 1, 8, 128, 2>(p, c, sms, s);
    if (v.rows == 32) return launch_cv<S, F32, 1, 16, 32, 1>(p, c, sms, s);
    return v.rows == 64 ? launch_cv<S, F32, 1, 16, 64, 1>(p, c, sms, s) : launch_cv<S, F32, 1, 16, 128, 1>(p, c, sms, s);
}
template <bool F32>
cudaError_t dispatch_cv(int stencil, const CcVisitShape &v, const CvParams &p, const TapCoeffs &c, int sms,
                        cudaStream_t s) {
    switch (stencil) {
    case TCS_STAR2D1R: return dispatch_cv<TCS_STAR2D1R, F32>(v, p, c, sms, s);
    case TCS_STAR2D2R: return dispatch_cv<TCS_STAR2D2R, F32>(v, p, c, sms, s);
    case TCS_BOX2D1R: return dispatch_cv<TCS_BOX2D1R, F32>(v, p, c, sms, s);
    case TCS_BOX2D2R: return dispatch_cv<TCS_BOX2D2R, F32>(v, p, c, sms, s);
    default: return cudaErrorInvalidValue;
    }
}

template <bool F32>
cudaError_t launch_cc(const GridGeom &g, int stencil, const TapCoeffs &c, const void *in,
                      void *out, cudaStream_t s) {
    CcParams p;
    p.g = g;
    p.p = F32 ? g.p32 : g.p16;
    p.nchunks = (g.nx + p.p.cpp - 1) / p.p.cpp;
    p.tiles_x = (p.nchunks + kCcPanels - 1) / kCcPanels;
    p.n_tiles = p.tiles_x * ((g.ny + kCcTileRows - 1) / kCcTileRows);
    p.neg_zero = -0.0f;
    // programmatic stream serialization, as the tensor steps: the next
    // step's CTAs initialise their barrier while this step's last tiles
    // finish, and wait in pdl_wait before their copies
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)p.n_tiles);
    cfg.blockDim = dim3(kCcWarps * 32);
    cfg.dynamicSmemBytes = kCcSmem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    switch (stencil) {
    case TCS_STAR2D1R: return cudaLaunchKernelEx(&cfg, cc_sweep_kernel<TCS_STAR2D1R, F32>, in, out, p, c);
    case TCS_STAR2D2R: return cudaLaunchKernelEx(&cfg, cc_sweep_kernel<TCS_STAR2D2R, F32>, in, out, p, c);
    case TCS_BOX2D1R: return cudaLaunchKernelEx(&cfg, cc_sweep_kernel<TCS_BOX2D1R, F32>, in, out, p, c);
    case TCS_BOX2D2R: return cudaLaunchKernelEx(&cfg, cc_sweep_kernel<TCS_BOX2D2R, F32>, in, out, p, c);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

cudaError_t launch_cc_f16(const GridGeom &g, int stencil, const TapCoeffs &c, const uint16_t *in,
                          uint16_t *out, cudaStream_t s) {
    return launch_cc<false>(g, stencil, c, in, out, s);
}

cudaError_t launch_cc_f32(const GridGeom &g, int stencil, const TapCoeffs &c, const float *in,
                          float *out, cudaStream_t s) {
    return launch_cc<true>(g, stencil, c, in, out, s);
}

// The form of a sweep's visits by its tiles per SM (n, of half-panel-lane
// tiles).  Few tiles: sixteen warps each (FP16 with halo 8, more steps per
// visit), and on grids below about a wave of them tiles of 64 or 32 rows, as
// a step takes an SM as long as its rows have instructions; a few per SM: eight warps,
// two or three CTAs per SM; many: whole-panel lanes, which spend fewer
// instructions per cell on halo words and overlap tiles by less.  With many
// tiles the radius-2 boxes (25 taps, bound by their FMAs, of which a visit's
// overlap computes a fifth twice) are faster in single steps: visits = 0.
// us per step of 128 / 64 / 32 rows: FP16 star2d1r 256² 1.54 / 1.09 / 0.89,
// box2d2r 3.63 / 2.29 / 1.54; 700² (n = 0.9 of 64 rows, 2.0 of 32) 1.59 / 1.12 /
// 1.12, 3.68 / 2.35 / 2.76; 1026² (1.45 of 64) 1.63 / 1.54, 1500² (2.9) 1.96 /
// 2.71; FP32 star2d1r 256² 1.43 / 1.13 / 0.96, 512² (1.25 of 32) 1.48 / 1.14 /
// 1.09, 700² (1.1 of 64) 1.43 / 1.28, 800² (1.5) 1.45 / 1.59.  (Thirty-two warps
// instead of sixteen: 256² 1.55 -> 1.91.)
// What the lines were drawn from, before the odd taps were scalar (compute), us
// per step, one step per launch -> 16 warps / 8 warps / whole panels, 128 rows
// (FP16 halo 8 / 4 / 4; FP32 4):
//   FP16 star2d1r  700² 6.09 -> 1.56 / 1.95 / 3.38, 2048² 6.76 -> 3.48 / 3.32
//        / 4.00, 4096² 12.7 -> 11.7 / 8.66 / 7.90, 8196² 47.6 -> 46.6 / 32.0 / 29.7
//   FP16 star2d2r  700² 6.51 -> 2.11 / 2.66 / 4.61, 8196² 51.3 -> - / 51.9 /
//        45.4 (44.6 with halo 8); box2d1r 8196² 51.4 -> - / 48.1 / 40.2
//   FP16 box2d2r   700² 8.04 -> 3.59 / 4.15 / 7.3, 3000² 14.9 -> - / 13.6 / 18,
//        8196² 81 -> - / 97 / 106
//   FP32 star2d1r  1026² 4.81 -> 1.54 / 1.69 / 2.06, 1800² 5.93 -> 3.95 / 2.42 /
//        2.90, 8196² 85.8 -> - / 44.3 / 37.9; star2d2r 87.6 -> - / 77.4 / 64.9;
//        box2d1r 87.2 -> - / 68.6 / 57.8
//   FP32 box2d2r   1026² 7.28 -> 4.10 / 5.68 / 6.20, 2500² 17.6 -> - / 16.4 /
//        14.9, 4096² 37.0 -> - / 44.7 / 38.9
// With scalar odd taps, the chosen form in calls of 50 steps (one step per launch
// -> visits):
//   FP16 star2d1r  256² 5.68 -> 0.79, 1026² 5.79 -> 1.36, 2048² 6.62 -> 2.54, 4096²
//        12.5 -> 7.24, 8196² 47.2 -> 28.0
//   FP16 star2d2r  6.12 -> 1.12, 6.24 -> 1.98, 7.27 -> 3.80, 14.1 -> 10.4, 48.5 -> 42.2
//   FP16 box2d1r   5.99 -> 0.95, 6.12 -> 1.65, 7.35 -> 3.36, 13.9 -> 9.85, 48.8 -> 37.8
//   FP16 box2d2r   7.42 -> 1.50, 7.55 -> 3.17, 9.27 -> 6.86, 3000² 14.3 -> 13.1, then
//        single steps: 4096² 21.6, 8196² 73.1
//   FP32 star2d1r  4.56 -> 0.91, 4.64 -> 1.57, 6.69 -> 2.88, 22.5 -> 9.34, 85.7 -> 36.3
//   FP32 star2d2r  5.09 -> 1.44, 5.25 -> 2.55, 7.77 -> 4.82, 24.1 -> 17.5, 87.2 -> 67.0
//   FP32 box2d1r   5.05 -> 1.03, 5.18 -> 2.02, 7.72 -> 4.72, 24.1 -> 14.6, 87.1 -> 55.3
//   FP32 box2d2r   6.44 -> 1.87, 7.08 -> 4.19, 12.5 -> 11.1, then single steps: 3000²
//        20.9, 4096² 34.9, 8196² 122
// One plan at a time, that is: plans in several streams fill the SMs in single
// steps too, and do not compute a visit's overlap.  us per step of one of 4 / 8
// plans in as many streams, single steps -> visits: FP16 star2d1r 1026² 1.73 ->
// 1.56 / 1.02 -> 1.56, box2d2r 2.69 -> 3.21 / 1.81 -> 3.21, FP32 box2d2r 512² 1.70
// -> 2.40 / 1.10 -> 2.40, 2048² 7.79 -> 11.3 / 7.80 -> 11.3.  (Forms of 64
// registers for two launches to an SM: one plan 10 to 25 % slower.)
CcVisitShape cc_visit_shape(const GridGeom &g, int stencil, bool f32, int steps, int sms) {
    CcVisitShape v{};
    const int r = stencil_r(stencil);
    const bool box2 = stencil == TCS_BOX2D2R;
    const int cpp = f32 ? 4 : 8, nchunks = (g.nx + cpp - 1) / cpp;
    auto shape = [&](int ppl, int warps, int halo, int tile_rows = kCcTileRows) {
        const int panels = 16 * ppl, rows = tile_rows - 2 * halo;
        v.rows = tile_rows;
        v.ppl = ppl;
        v.warps = warps;
        v.halo = halo;
        v.tiles_x = nchunks <= panels ? 1 : (nchunks - 2 + panels - 3) / (panels - 2);
        v.tiles_y = g.ny <= tile_rows ? 1 : (g.ny - 2 * halo + rows - 1) / rows;
        v.depth = halo / r + 1;
        v.visits = steps > 0 ? (steps - 1) / v.depth + 1 : 0;
        return (double)v.tiles_x * v.tiles_y / sms;
    };
    if (shape(1, 16, f32 ? 4 : 8, 32) <= (f32 ? 1.25 : 1.05)) return v;
    if (shape(1, 16, f32 ? 4 : 8, 64) <= (f32 ? 1.2 : 1.5)) return v;
    if (f32) {
        const double n = shape(1, 8, 4);
        if (n <= 1.4) {
            if (n > 1.0 || box2) shape(1, 16, 4);
        } else if (n > (box2 ? 5.0 : 3.6)) {
            shape(2, 8, 4);
            if (box2 && n > 8.0) v.visits = 0;
        }
    } else {
        const double n = shape(1, 16, 8);
        if (n > 1.7) {
            if (n <= 6.0 || box2) shape(1, 8, 4);
            else shape(2, 8, r == 2 ? 8 : 4);
            if (box2 && n > 7.0) v.visits = 0;
        }
    }
    return v;
}

// Configures the stencil's visit kernels ahead of any capture.
cudaError_t cc_visit_prepare(int stencil, bool f32) {
    CvParams p{};
    const TapCoeffs c{};
    for (const CcVisitShape &v : {CcVisitShape{1, 8, 128}, CcVisitShape{1, 16, 128}, CcVisitShape{1, 16, 64}, CcVisitShape{1, 16, 32}, CcVisitShape{2, 8, 128}}) {
        const cudaError_t e = f32 ? dispatch_cv<true>(stencil, v, p, c, 1, nullptr)
                                  : dispatch_cv<false>(stencil, v, p, c, 1, nullptr);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_cc_visits(const GridGeom &g, int stencil, bool f32, const TapCoeffs &c, void *in,
                             void *out, int steps, const CcVisitShape &v, unsigned *counters,
                             cudaStream_t s, int sms) {
    CvParams p;
    p.g = g;
    p.p = f32 ? g.p32 : g.p16;
    p.nchunks = (g.nx + p.p.cpp - 1) / p.p.cpp;
    p.tiles_x = v.tiles_x;
    p.tiles_y = v.tiles_y;
    p.halo = v.halo;
    p.neg_zero = -0.0f;
    p.visits = v.visits;
    p.base = steps / v.visits;
    p.extra = steps % v.visits;
    p.plane[0] = in;
    p.plane[1] = out;
    p.ended = counters;
    p.done = counters + kRowCounterStride;
    return f32 ? dispatch_cv<true>(stencil, v, p, c, sms, s)
               : dispatch_cv<false>(stencil, v, p, c, sms, s);
}

cudaError_t cc_error_word(int **word) {
    return cudaGetSymbolAddress(reinterpret_cast<void **>(word), g_cc_error);
}

}  // namespace tcs
