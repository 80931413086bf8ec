// Device layout transforms.
//
//  - The reference's host-side layout16 helpers, padding_2D, brick_layout_2D
//    and reverse_layout_2D (layout16/host_star2d1r.cu:63-101), as bit-exact
//    device kernels (16 x 16 bricks, row-major inside a brick).
//  - pack / unpack between FP32 row-major grids and the engine's panel
//    planes: array_float2half (common/common.hpp:146-160) + padding_2D +
//    layout change in one pass, and the inverse, by blocks of 32 rows by 32
//    panels through shared memory.
#include "tcs_device.cuh"
#include "tcs_internal.h"

namespace tcs {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ uint16_t f2h_bits(float v) {
    __half h = __float2half_rn(v);
    return *reinterpret_cast<uint16_t *>(&h);
}

__device__ __forceinline__ float h2f_bits(uint16_t b) {
    __half h = *reinterpret_cast<__half *>(&b);
    return __half2float(h);
}

// pack and unpack move a block of kBlkRows plane rows by kBlkPans panels
// through shared memory, so that both sides are contiguous: a warp's accesses
// of the FP32 grid are runs of 32 cells of one row, its accesses of a plane
// 32 rows of one panel (512 bytes).  (With one 16-byte panel row per thread
// straight to the plane, each was half a 32-byte sector, a plane row apart:
// 16386² split up- and download took 2.25 ms of a 50-step solve's 19.9 ms,
// 0.8 ms at the memory rate.)  The grid side uses 4-byte accesses, so a grid
// and its rows may start at any float.
constexpr int kBlkRows = 32, kBlkPans = 32;
constexpr int kBlkPitch = kBlkPans * 16 + 16;  // bytes of a staged plane row (16: no bank conflicts)
enum PackMode { kPackF16, kPackF32, kPackSplit };

struct BlockPos {
    int row, pan;  // first plane row and panel
};
__device__ __forceinline__ BlockPos block_pos(const PlaneGeom &p, int q0) {
    const int npb = (p.npan + kBlkPans - 1) / kBlkPans;
    const int rb = (int)(blockIdx.x / npb);
    return BlockPos{q0 + rb * kBlkRows, (int)(blockIdx.x - (unsigned)rb * npb) * kBlkPans};
}

// Split storage of x: x' = x 2^-E, hi = fp16(rint(x' 2^11) 2^-11) (fixed
// point), lo = fp16((x' - hi) 2^11).  Every step before the final rounding
// of lo is exact in FP32.
__device__ __forceinline__ void split_value(float x, float scale, uint16_t &h, uint16_t &l) {
    const float xs = x * scale;
    h = f2h_bits(rintf(xs * 2048.0f) * (1.0f / 2048.0f));
    l = f2h_bits((xs - h2f_bits(h)) * 2048.0f);
}

// Plane rows [q0, q1) of the padded grid.  Split: scaled by 2^-E, E from
// `sc` when given (and the largest |x'| of the cells outside the update
// rectangle [y0, y1) x [x0, x1) added to its border maximum), else `scale`.
struct PackArgs {
    const float *in;
    int ny, nx, pad;
    float pad_value;
    void *out, *out_lo;
    PlaneGeom p;
    int q0, q1;
    float scale;
    SplitScale *sc;
    int y0, y1, x0, x1;
    // launched right behind max_abs_scale_kernel on the same cells, which lets
    // it start only once all work before both has completed: the cells are
    // loaded beside that pass (past L1), before the wait for its scale (256
    // split grids of a mixed batch: 12.0 -> 9.2 us per upload)
    bool behind_max;
    bool early;  // EARLY of the kernel
};

// EARLY: lets the next kernel's launch start beside it (tcs_internal.h), as its
// first instruction (behind the load of an argument that says so it came late:
// 803 x 219 star2d1r, 2 steps 11.3 -> 12.1 us a solve).
template <int MODE, bool EARLY>
__global__ void __launch_bounds__(kThreads) pack_kernel(const PackArgs a) {
    constexpr int CPP = MODE == kPackF32 ? 4 : 8;
    constexpr int CELLS = kBlkPans * CPP;  // of a block's row
    constexpr int N = CELLS / 32, K = kBlkRows / 8;
    __shared__ __align__(16) uint8_t buf[MODE == kPackSplit ? 2 : 1][kBlkRows][kBlkPitch];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const BlockPos b = block_pos(a.p, a.q0);
    const int X = (b.pan - 1) * CPP + lane;  // this lane's first cell: X, X + 32, ...
    if (EARLY) pdl_launch_dependents();
    if (MODE != kPackSplit || !a.behind_max) pdl_wait();
    float v[K][N];
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int Y = b.row + warp + 8 * k - kPadTop;
        const int iy = Y - a.pad, ix = X - lane - a.pad;
        // (rows from q1 on belong to a later range: not read)
        const bool row_in = iy >= 0 && iy < a.ny && b.row + warp + 8 * k < a.q1;
        const float *src = a.in + (size_t)(row_in ? iy : 0) * a.nx;
        if (row_in && ix >= 0 && ix + CELLS <= a.nx) {
#pragma unroll
            for (int i = 0; i < N; i++) v[k][i] = __ldcg(src + ix + lane + 32 * i);
        } else {
            // border and padding cells: the loads clamped to the row and the
            // values selected, so that they all are in flight at once
            const bool row_pad = Y >= 0 && Y < a.ny + 2 * a.pad;
#pragma unroll
            for (int i = 0; i < N; i++) {
                const int x = ix + lane + 32 * i;
                const float c = row_in ? __ldcg(src + min(max(x, 0), a.nx - 1)) : 0.0f;
                const bool pad_in = row_pad && x >= -a.pad && x < a.nx + a.pad;
                v[k][i] = row_in && x >= 0 && x < a.nx ? c : pad_in ? a.pad_value : 0.0f;
            }
        }
    }
    if (MODE == kPackSplit && a.behind_max) pdl_wait();
    float scale = a.scale;
    bool border = false;  // the block may hold cells outside the update rectangle
    if (MODE == kPackSplit && a.sc) {
        scale = ldexpf(1.0f, -a.sc->bexp);
        const int ya = b.row - kPadTop, xa = X - lane;
        border = ya < a.y0 || ya + kBlkRows > a.y1 || xa < a.x0 || xa + CELLS > a.x1;
    }
    float m = 0.0f;
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int r = warp + 8 * k;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int c = lane + 32 * i;
            if (MODE == kPackF32) {
                reinterpret_cast<float *>(buf[0][r])[c] = v[k][i];
            } else if (MODE == kPackF16) {
                reinterpret_cast<uint16_t *>(buf[0][r])[c] = f2h_bits(v[k][i]);
            } else {
                uint16_t h, l;
                split_value(v[k][i], scale, h, l);
                reinterpret_cast<uint16_t *>(buf[0][r])[c] = h;
                reinterpret_cast<uint16_t *>(buf[MODE == kPackSplit][r])[c] = l;
                if (border) {
                    const int y = b.row + r - kPadTop, x = X + 32 * i;
                    const bool in_grid = y >= 0 && y < a.ny && x >= 0 && x < a.nx && b.row + r < a.q1;
                    if (in_grid && !(y >= a.y0 && y < a.y1 && x >= a.x0 && x < a.x1))
                        m = fmaxf(m, fabsf(fmaf(h2f_bits(h), 2048.0f, h2f_bits(l))));
                }
            }
        }
    }
    if (border) {  // |x'| 2^11 = |hi 2^11 + lo|, rounded once to FP32
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0 && m > 0.0f) atomicMax(&a.sc->bmax, __float_as_uint(m * (1.0f / 2048.0f)));
    }
    __syncthreads();
    const int row = b.row + lane;
    if (row >= a.q1) return;
#pragma unroll
    for (int k = 0; k < kBlkPans / 8; k++) {
        const int j = warp + 8 * k, pan = b.pan + j;
        if (pan >= a.p.npan) continue;
        const size_t q = (size_t)pan * a.p.nyp + row;
        static_cast<uint4 *>(a.out)[q] = *reinterpret_cast<const uint4 *>(&buf[0][lane][16 * j]);
        if (MODE == kPackSplit)
            static_cast<uint4 *>(a.out_lo)[q] = *reinterpret_cast<const uint4 *>(&buf[MODE == kPackSplit][lane][16 * j]);
    }
}

// The grid cells of plane rows [q0, q1), as FP32.  Split: scaled by 2^E, E
// from *exp when given, else `scale`.
struct UnpackArgs {
    const void *in, *in_lo;
    int ny, nx, pad;
    float *out;
    PlaneGeom p;
    int q0, q1;
    float scale;
    const int *exp;
    bool early;  // as PackArgs
};

template <int MODE, bool EARLY>
__global__ void __launch_bounds__(kThreads) unpack_kernel(const UnpackArgs a) {
    constexpr int CPP = MODE == kPackF32 ? 4 : 8;
    constexpr int CELLS = kBlkPans * CPP;
    constexpr int N = CELLS / 32, K = kBlkPans / 8;
    __shared__ __align__(16) uint8_t buf[MODE == kPackSplit ? 2 : 1][kBlkRows][kBlkPitch];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const BlockPos b = block_pos(a.p, a.q0);
    const int row = min(b.row + lane, a.q1 - 1);
    if (EARLY) pdl_launch_dependents();
    pdl_wait();
    uint4 v[K], l[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int pan = min(b.pan + warp + 8 * k, a.p.npan - 1);
        const size_t q = (size_t)pan * a.p.nyp + row;
        v[k] = static_cast<const uint4 *>(a.in)[q];
        if (MODE == kPackSplit) l[k] = static_cast<const uint4 *>(a.in_lo)[q];
    }
    float scale = a.scale;
    if (MODE == kPackSplit && a.exp) scale = ldexpf(1.0f, *a.exp);
#pragma unroll
    for (int k = 0; k < K; k++) {
        *reinterpret_cast<uint4 *>(&buf[0][lane][16 * (warp + 8 * k)]) = v[k];
        if (MODE == kPackSplit) *reinterpret_cast<uint4 *>(&buf[MODE == kPackSplit][lane][16 * (warp + 8 * k)]) = l[k];
    }
    __syncthreads();
    const int ix0 = (b.pan - 1) * CPP - a.pad;
#pragma unroll
    for (int k = 0; k < kBlkRows / 8; k++) {
        const int r = warp + 8 * k, iy = b.row + r - kPadTop - a.pad;
        if (b.row + r >= a.q1 || iy < 0 || iy >= a.ny) continue;
        float *dst = a.out + (size_t)iy * a.nx;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int c = lane + 32 * i, ix = ix0 + c;
            float x;
            if (MODE == kPackF32) x = reinterpret_cast<const float *>(buf[0][r])[c];
            else if (MODE == kPackF16) x = h2f_bits(reinterpret_cast<const uint16_t *>(buf[0][r])[c]);
            else
                x = fmaf(h2f_bits(reinterpret_cast<const uint16_t *>(buf[MODE == kPackSplit][r])[c]), 1.0f / 2048.0f,
                         h2f_bits(reinterpret_cast<const uint16_t *>(buf[0][r])[c])) * scale;
            if (ix >= 0 && ix < a.nx) dst[ix] = x;
        }
    }
}

// Scale exponent E of a grid whose max |x| has float bits `bits`: the
// smallest E with max |x| < 2^E (frexp's exponent), 0 for an all-zero grid.
__device__ __forceinline__ int scale_exp_of(unsigned bits) {
    const float m = __uint_as_float(bits);
    if (!(m > 0.0f) || !isfinite(m)) return 0;
    int e = 0;
    frexpf(m, &e);
    return e;
}

// The largest |x| of this block's share of n floats, as FP32 bits in every
// thread of warp 0: 16-byte loads from the first aligned element on, four in
// flight (one 4-byte load at a time ran at a third of the memory rate).
__device__ __forceinline__ unsigned block_max_abs(const float *__restrict__ in, size_t n) {
    const size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    size_t head = ((16 - (reinterpret_cast<uintptr_t>(in) & 15)) & 15) / sizeof(float);
    if (head > n) head = n;
    const size_t n4 = (n - head) / 4;
    const float4 *v = reinterpret_cast<const float4 *>(in + head);
    float m = 0.0f;
    auto take = [&](const float4 &x) {
        m = fmaxf(fmaxf(fmaxf(m, fabsf(x.x)), fmaxf(fabsf(x.y), fabsf(x.z))), fabsf(x.w));
    };
    size_t i = id;
    for (; i + 3 * stride < n4; i += 4 * stride) {
        const float4 a = v[i], b = v[i + stride], c = v[i + 2 * stride], d = v[i + 3 * stride];
        take(a);
        take(b);
        take(c);
        take(d);
    }
    for (; i < n4; i += stride) take(v[i]);
    if (id < head) m = fmaxf(m, fabsf(in[id]));
    for (size_t j = head + 4 * n4 + id; j < n; j += stride) m = fmaxf(m, fabsf(in[j]));
    __shared__ unsigned part[kThreads / 32];
    // (non-negative floats order like their bit patterns)
    unsigned u = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = u;
    __syncthreads();
    u = threadIdx.x < kThreads / 32 ? part[threadIdx.x] : 0u;
    return __reduce_max_sync(0xffffffffu, u);
}

// max |x| into *out_bits (which starts at 0).
__global__ void __launch_bounds__(kThreads) max_abs_kernel(const float *__restrict__ in, size_t n,
                                                           unsigned *out_bits) {
    const unsigned u = block_max_abs(in, n);
    if (threadIdx.x == 0) atomicMax(out_bits, u);
}

// The same for a split grid's upload: the last block to finish starts the
// grid's scale record from the maximum (E_0 = E_B = its exponent, steps -1
// and 0 unmeasured, no border yet) and leaves scratch[0] (the maximum) and
// scratch[1] (blocks done) zero for the next use.
__global__ void __launch_bounds__(kThreads) max_abs_scale_kernel(const float *__restrict__ in, size_t n,
                                                                 unsigned *scratch, SplitScale *sc) {
    pdl_wait();
    pdl_launch_dependents();  // (after the wait: see PackArgs::behind_max)
    const unsigned u = block_max_abs(in, n);
    if (threadIdx.x != 0) return;
    atomicMax(&scratch[0], u);
    __threadfence();
    if (atomicAdd(&scratch[1], 1u) != gridDim.x - 1) return;
    __threadfence();
    const int e = scale_exp_of(atomicExch(&scratch[0], 0u));
    scratch[1] = 0u;
    for (int i = 0; i < kScaleRing; i++) {
        sc->maxbits[i] = 0;
        sc->exp[i] = e;
    }
    sc->maxbits[0] = sc->maxbits[kScaleRing - 1] = kScaleNoMax;
    sc->bmax = 0u;
    sc->bexp = e;
}

// ------------------------------------------- reference layout16 helpers ---
// 16 x 16 bricks: brick (i, j) at (i*nbx + j)*256, cell (y, x) at y*16 + x.
struct Slice {
    int brick, row, col;
};
__device__ __forceinline__ Slice slice_of(size_t id) {
    Slice s;
    s.brick = static_cast<int>(id / 32);
    const int rem = static_cast<int>(id % 32);
    s.row = rem / 2;
    s.col = (rem % 2) * 8;
    return s;
}

// padding_2D: one thread per output cell.
__global__ void padding_2d_kernel(const uint16_t *__restrict__ in, uint16_t *__restrict__ out,
                                  int size, int halo, uint16_t value) {
    const int p = size + 2 * halo;
    const size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (size_t)p * p) return;
    const int i = static_cast<int>(id / p), j = static_cast<int>(id % p);
    const bool inside = i >= halo && i < size + halo && j >= halo && j < size + halo;
    out[id] = inside ? in[(size_t)(i - halo) * size + (j - halo)] : value;
}

// brick_layout_2D: one thread per 8-cell slice of the brick output.
__global__ void brick_2d_kernel(const uint16_t *__restrict__ in, uint16_t *__restrict__ out,
                                int ny, int nx, int nbx, size_t n_slices) {
    const size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n_slices) return;
    const Slice s = slice_of(id);
    const int Y = (s.brick / nbx) * 16 + s.row;
    const int X0 = (s.brick % nbx) * 16 + s.col;
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        uint32_t h[2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int X = X0 + 2 * i + j;
            h[j] = (Y < ny && X < nx) ? in[(size_t)Y * nx + X] : 0u;
        }
        w[i] = h[0] | (h[1] << 16);
    }
    reinterpret_cast<uint4 *>(out)[id] = make_uint4(w[0], w[1], w[2], w[3]);
}

// reverse_layout_2D: one thread per 8-cell slice of the brick input.
__global__ void unbrick_2d_kernel(const uint16_t *__restrict__ in, uint16_t *__restrict__ out,
                                  int ny, int nx, int nbx, size_t n_slices) {
    const size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n_slices) return;
    const Slice s = slice_of(id);
    const int Y = (s.brick / nbx) * 16 + s.row;
    if (Y >= ny) return;
    const uint4 v = reinterpret_cast<const uint4 *>(in)[id];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    const int X0 = (s.brick % nbx) * 16 + s.col;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int X = X0 + i;
        if (X < nx) out[(size_t)Y * nx + X] = (uint16_t)(w[i >> 1] >> (16 * (i & 1)));
    }
}

inline unsigned blocks_for(size_t n) { return static_cast<unsigned>((n + kThreads - 1) / kThreads); }
inline int nb(int n) { return (n + 15) / 16; }

}  // namespace

namespace {

using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                   const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                   const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's cuTensorMapEncodeTiled, found through the runtime (no link
// against the driver library).
EncodeTiledFn encode_tiled() {
    static const EncodeTiledFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                             &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

}  // namespace

cudaError_t encode_panel_map(const uint16_t *plane, const PlaneGeom &pg, CUtensorMap *map,
                             int panels, int rows) {
    const EncodeTiledFn enc = encode_tiled();
    if (!enc) return cudaErrorNotSupported;
    if (reinterpret_cast<uintptr_t>(plane) % 16 || pg.nyp % 8 || pg.cpp != 8)
        return cudaErrorInvalidValue;
    const cuuint64_t dims[3] = {(cuuint64_t)(2 * rows), (cuuint64_t)(pg.nyp / rows), (cuuint64_t)pg.npan};
    const cuuint64_t strides[2] = {(cuuint64_t)(16 * rows), (cuuint64_t)pg.nyp * 16};  // bytes, dims 1 and 2
    const cuuint32_t box[3] = {(cuuint32_t)(2 * rows), (cuuint32_t)((kTile + 8) / rows), (cuuint32_t)panels};
    const cuuint32_t es[3] = {1, 1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, const_cast<uint16_t *>(plane),
                           dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

namespace {

// Layout kernels launch with programmatic stream serialization (pdl_enabled):
// a kernel's launch overlaps its predecessor's run, and it waits for it
// before its first access.  A batch's or a small grid's transfers are a row
// of such launches of a few microseconds each.
template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kernel)(P...), unsigned blocks, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <int MODE>
cudaError_t launch_pack(PackArgs a, cudaStream_t s) {
    const unsigned blocks = (unsigned)((a.q1 - a.q0 + kBlkRows - 1) / kBlkRows) *
                            (unsigned)((a.p.npan + kBlkPans - 1) / kBlkPans);
    return a.early ? launch_pdl(pack_kernel<MODE, true>, blocks, s, a) : launch_pdl(pack_kernel<MODE, false>, blocks, s, a);
}
template <int MODE>
cudaError_t launch_unpack(UnpackArgs a, cudaStream_t s) {
    const unsigned blocks = (unsigned)((a.q1 - a.q0 + kBlkRows - 1) / kBlkRows) *
                            (unsigned)((a.p.npan + kBlkPans - 1) / kBlkPans);
    return a.early ? launch_pdl(unpack_kernel<MODE, true>, blocks, s, a)
                   : launch_pdl(unpack_kernel<MODE, false>, blocks, s, a);
}

PackArgs pack_args(const float *in, int ny, int nx, int pad, float pad_value, void *out, int cpp) {
    PackArgs a{};
    a.in = in;
    a.ny = ny;
    a.nx = nx;
    a.pad = pad;
    a.pad_value = pad_value;
    a.out = out;
    a.p = plane_geom(ny + 2 * pad, nx + 2 * pad, cpp);
    a.q1 = a.p.nyp;
    a.scale = 1.0f;
    a.early = true;
    return a;
}
UnpackArgs unpack_args(const void *in, int ny, int nx, int pad, float *out, int cpp) {
    UnpackArgs a{};
    a.in = in;
    a.ny = ny;
    a.nx = nx;
    a.pad = pad;
    a.out = out;
    a.p = plane_geom(ny + 2 * pad, nx + 2 * pad, cpp);
    // only the plane rows that hold the grid's
    a.q0 = kPadTop + pad;
    a.q1 = a.q0 + ny;
    a.scale = 1.0f;
    return a;
}

unsigned max_abs_blocks(size_t n) {
    const size_t want = (n + 16 * kThreads - 1) / (16 * kThreads);
    return static_cast<unsigned>(want < 1216 ? (want ? want : 1) : 1216);  // eight per SM
}

}  // namespace

cudaError_t launch_pack_f16(const float *in, int ny, int nx, int pad, float pad_value,
                            uint16_t *plane, cudaStream_t s, bool early) {
    PackArgs a = pack_args(in, ny, nx, pad, pad_value, plane, 8);
    a.early = early;
    return launch_pack<kPackF16>(a, s);
}

cudaError_t launch_unpack_f16(const uint16_t *plane, int ny, int nx, int pad, float *out,
                              cudaStream_t s, bool early) {
    UnpackArgs a = unpack_args(plane, ny, nx, pad, out, 8);
    a.early = early;
    return launch_unpack<kPackF16>(a, s);
}

__global__ void split_scale_end_run_kernel(SplitScale *sc, int steps) {
    const unsigned m1 = sc->maxbits[(steps - 1) & (kScaleRing - 1)];
    const unsigned m0 = sc->maxbits[steps & (kScaleRing - 1)];
    const int e1 = sc->exp[(steps - 1) & (kScaleRing - 1)];
    const int e0 = sc->exp[steps & (kScaleRing - 1)];
    for (int i = 1; i < kScaleRing - 1; i++) sc->maxbits[i] = 0;
    sc->maxbits[kScaleRing - 1] = m1;
    sc->exp[kScaleRing - 1] = e1;
    sc->maxbits[0] = m0;
    sc->exp[0] = e0;
}

cudaError_t launch_split_scale_end_run(SplitScale *sc, int steps, cudaStream_t s) {
    if (steps <= 0) return cudaSuccess;
    split_scale_end_run_kernel<<<1, 1, 0, s>>>(sc, steps);
    return cudaGetLastError();
}

cudaError_t launch_pack_f32(const float *in, int ny, int nx, int pad, float pad_value,
                            float *plane, cudaStream_t s, bool early) {
    PackArgs a = pack_args(in, ny, nx, pad, pad_value, plane, 4);
    a.early = early;
    return launch_pack<kPackF32>(a, s);
}

cudaError_t launch_unpack_f32(const float *plane, int ny, int nx, int pad, float *out,
                              cudaStream_t s, bool early) {
    UnpackArgs a = unpack_args(plane, ny, nx, pad, out, 4);
    a.early = early;
    return launch_unpack<kPackF32>(a, s);
}

// Plane rows [q0, q1) only (every panel), pad 0: the grid rows they hold are
// [q0 - 4, q1 - 4) clipped to the grid; the pad rows above and below belong
// to the first and last ranges.
cudaError_t launch_pack_rows(const float *in, int ny, int nx, bool f32, void *plane, int q0,
                             int q1, cudaStream_t s, bool early) {
    PackArgs a = pack_args(in, ny, nx, 0, 0.0f, plane, f32 ? 4 : 8);
    a.early = early;
    if (q0 < 0 || q1 > a.p.nyp || q0 >= q1) return cudaErrorInvalidValue;
    a.q0 = q0;
    a.q1 = q1;
    return f32 ? launch_pack<kPackF32>(a, s) : launch_pack<kPackF16>(a, s);
}

cudaError_t launch_unpack_rows(const void *plane, int ny, int nx, bool f32, float *out, int q0,
                               int q1, cudaStream_t s) {
    UnpackArgs a = unpack_args(plane, ny, nx, 0, out, f32 ? 4 : 8);
    if (q0 < 0 || q1 > a.p.nyp || q0 >= q1) return cudaErrorInvalidValue;
    a.q0 = q0;
    a.q1 = q1;
    return f32 ? launch_unpack<kPackF32>(a, s) : launch_unpack<kPackF16>(a, s);
}

cudaError_t launch_pack_split(const float *in, int ny, int nx, int pad, float pad_value,
                              int scale_exp, uint16_t *hi, uint16_t *lo, cudaStream_t s) {
    PackArgs a = pack_args(in, ny, nx, pad, pad_value, hi, 8);
    a.out_lo = lo;
    a.scale = ldexpf(1.0f, -scale_exp);
    return launch_pack<kPackSplit>(a, s);
}

cudaError_t launch_split_upload(const float *in, const GridGeom &g, unsigned *scratch,
                                SplitScale *sc, uint16_t *hi, uint16_t *lo, cudaStream_t s) {
    const size_t n = (size_t)g.ny * g.nx;
    cudaError_t e = launch_pdl(max_abs_scale_kernel, max_abs_blocks(n), s, in, n, scratch, sc);
    if (e != cudaSuccess) return e;
    PackArgs a = pack_args(in, g.ny, g.nx, 0, 0.0f, hi, 8);
    a.out_lo = lo;
    a.sc = sc;
    a.behind_max = true;
    a.y0 = g.y0; a.y1 = g.y1; a.x0 = g.x0; a.x1 = g.x1;
    return launch_pack<kPackSplit>(a, s);
}

cudaError_t launch_unpack_split(const uint16_t *hi, const uint16_t *lo, int ny, int nx, int pad,
                                int scale_exp, float *out, cudaStream_t s) {
    UnpackArgs a = unpack_args(hi, ny, nx, pad, out, 8);
    a.in_lo = lo;
    a.scale = ldexpf(1.0f, scale_exp);
    return launch_unpack<kPackSplit>(a, s);
}

cudaError_t launch_unpack_split_dev(const uint16_t *hi, const uint16_t *lo, int ny, int nx,
                                    const int *exp_in, float *out, cudaStream_t s, bool early) {
    UnpackArgs a = unpack_args(hi, ny, nx, 0, out, 8);
    a.early = early;
    a.in_lo = lo;
    a.exp = exp_in;
    return launch_unpack<kPackSplit>(a, s);
}

cudaError_t launch_max_abs(const float *in, size_t n, unsigned *out_bits, cudaStream_t s) {
    max_abs_kernel<<<max_abs_blocks(n), kThreads, 0, s>>>(in, n, out_bits);
    return cudaGetLastError();
}

cudaError_t launch_padding_2d(const uint16_t *in, uint16_t *out, int size, int halo,
                              uint16_t value, cudaStream_t s) {
    const size_t p = (size_t)(size + 2 * halo);
    padding_2d_kernel<<<blocks_for(p * p), kThreads, 0, s>>>(in, out, size, halo, value);
    return cudaGetLastError();
}

cudaError_t launch_brick_2d(const uint16_t *in, uint16_t *out, int ny, int nx, cudaStream_t s) {
    const size_t n = (size_t)nb(ny) * nb(nx) * 32;
    brick_2d_kernel<<<blocks_for(n), kThreads, 0, s>>>(in, out, ny, nx, nb(nx), n);
    return cudaGetLastError();
}

cudaError_t launch_unbrick_2d(const uint16_t *in, uint16_t *out, int ny, int nx, cudaStream_t s) {
    const size_t n = (size_t)nb(ny) * nb(nx) * 32;
    unbrick_2d_kernel<<<blocks_for(n), kThreads, 0, s>>>(in, out, ny, nx, nb(nx), n);
    return cudaGetLastError();
}

}  // namespace tcs
