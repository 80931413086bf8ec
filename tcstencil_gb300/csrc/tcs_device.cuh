// Device helpers shared by the sweep kernels: shared-memory barriers, TMA
// tensor copies, tcgen05 (UMMA / TMEM) wrappers and bounded waits.  All PTX
// here targets sm_103a.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <stdint.h>

namespace tcs {

enum DeviceError : int {
    kErrNone = 0,
    kErrWaitFull = 1,     // consumer waited too long for a TMA stage
    kErrWaitEmpty = 2,    // producer waited too long for a free stage
    kErrWaitAccum = 3,    // MMA issuer waited too long for a free accumulator
    kErrWaitResult = 4,   // epilogue waited too long for an accumulator
    kErrWaitDrain = 5,    // final drain of in-flight copies / MMAs timed out
    kErrWaitDep = 6,      // a step waited too long for its previous step (batch, multi-step)
};

// Upper bound on any single in-kernel wait: the hardware finishes each awaited
// copy or MMA in microseconds, so one second means something is wrong.
constexpr uint64_t kWaitLimitNs = 1000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t global_timer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Error words are per translation unit (static __device__ ints): a bounded
// wait that gives up writes its code there (first error wins); the host reads
// and clears every unit's word in tcs_device_error().
__device__ __forceinline__ void record_error(int *word, int code) { atomicCAS(word, 0, code); }

// -------------------------------------------- cross-CTA completion counts ---
__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Completion count with release semantics: the stores ordered before it (this
// thread's, and its warp's or CTA's through the barrier that precedes it) are
// visible at GPU scope before the count, for the consumer's acquire load.
__device__ __forceinline__ void red_release_add(unsigned *p, unsigned v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Per-warp progress words in shared memory: the writer's earlier stores
// (its warp's, ordered by a preceding __syncwarp) happen before a reader's
// acquire that sees the value.
__device__ __forceinline__ void st_release_cta(uint32_t *p, uint32_t v) {
    asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}

__device__ __forceinline__ uint32_t ld_acquire_cta(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
    return v;
}

// Counts in shared memory whose last adder has seen the earlier adders'
// stores.
__device__ __forceinline__ unsigned add_acq_rel_cta(unsigned *p, unsigned v) {
    unsigned old;
    asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], %2;"
                 : "=r"(old) : "r"(smem_u32(p)), "r"(v) : "memory");
    return old;
}

// Relaxed read of a count; a following fence_acq_rel_gpu makes it an acquire.
__device__ __forceinline__ unsigned ld_relaxed(const unsigned *p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Relaxed count, published by a preceding fence_acq_rel_gpu (release pattern).
__device__ __forceinline__ void red_relaxed_add(unsigned *p, unsigned v) {
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void fence_acq_rel_gpu() {
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
}

// ------------------------------------------ programmatic dependent launch ---
// A step kernel launched with programmatic stream serialization may start
// while the previous step is still running.  launch_dependents lets the next
// launch in the stream begin once every CTA of this grid has passed it; wait
// returns when the previous grid has completed and its stores are visible.
// With no programmatic predecessor, wait returns at once.
__device__ __forceinline__ void pdl_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ------------------------------------------------------------- mbarrier ---
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_n(uint64_t *bar, uint32_t n) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(n) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// The next 1024-byte boundary of the dynamic shared memory.  As an offset to
// the array, not a rounded integer: the compiler then knows that accesses
// through the result are to shared memory, and emits no generic ones (with
// them: 8196² box2d2r FP16 41.8 us per step, 40.0 without; two-step split
// 1026² 5.3, 5.1).
__device__ __forceinline__ uint8_t *align_smem(uint8_t *raw) { return raw + (-smem_u32(raw) & 1023u); }

// Waits for the phase of `parity` to complete.  Gives up (returns false) when
// *abort becomes non-zero or after kWaitLimitNs; the caller then records the
// error and leaves its loop.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity,
                                          const volatile int *abort,
                                          uint64_t limit_ns = kWaitLimitNs) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_timer_ns();
    while (true) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort) return false;
        if (global_timer_ns() - t0 > limit_ns) return false;
        __nanosleep(32);
    }
}

// 16-byte shared-memory accesses by address.
__device__ __forceinline__ void sts128(uint32_t addr, const uint4 &v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y),
                 "r"(v.z), "r"(v.w)
                 : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(addr)
                 : "memory");
    return v;
}

// ------------------------------------------------------------------ TMA ---
__device__ __forceinline__ void tma_prefetch_map(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// 3-D tiled load into shared memory, completion counted on `bar` in bytes.
// The innermost coordinate c0 is always 0 here (16-byte aligned).
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, uint64_t *bar,
                                            int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
        : "memory");
}

// 1-D bulk copy of `bytes` (a multiple of 16) from global to shared memory,
// both addresses 16-byte aligned; completion counted on `bar` in bytes.
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes,
                                          uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// Orders this thread's earlier generic-proxy accesses of global memory (and
// those it has observed) before its later async-proxy (bulk copy) accesses.
__device__ __forceinline__ void fence_proxy_async_global() {
    asm volatile("fence.proxy.async.global;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// -------------------------------------------------------------- tcgen05 ---
__device__ __forceinline__ void tmem_alloc(uint32_t *dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(dst)),
                 "r"(ncols)
                 : "memory");
}

__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// D[tmem] (+)= A[smem desc] * B[smem desc], kind::f16 (FP16 x FP16 -> FP32).
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                         uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Arrives once on `bar` when every tcgen05.mma issued so far by this thread
// has completed.
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}

// 32 lanes x 32 bits, 16 consecutive columns: thread t of the warp receives
// row (lane base + t), columns col .. col+15.
__device__ __forceinline__ void tmem_ld_x16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
          "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
          "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld_x8(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
          "=r"(v[7])
        : "r"(taddr));
}

// Waits for this thread's tcgen05.ld's.  The words they loaded pass through an
// empty asm that depends on the wait, so that no use of one can be moved
// before it (the loads return at once, and to the compiler their results are
// there).
__device__ __forceinline__ void tmem_loaded(uint32_t &v, uint32_t waited) { asm("" : "+r"(v) : "r"(waited)); }
template <typename T, int N>
__device__ __forceinline__ void tmem_loaded(T (&v)[N], uint32_t waited) {
#pragma unroll
    for (int i = 0; i < N; i++) tmem_loaded(v[i], waited);
}
template <typename... V>
__device__ __forceinline__ void tmem_ld_wait(V &...v) {
    uint32_t waited;
    asm volatile("tcgen05.wait::ld.sync.aligned;\n\tmov.u32 %0, 0;" : "=r"(waited)::"memory");
    (tmem_loaded(v, waited), ...);
}

// Shared-memory matrix descriptor, no swizzle.  The operand is made of
// 8-row x 16-byte core matrices stored as 128 contiguous bytes; `lbo` is the
// byte distance between core matrices adjacent along K, `sbo` along M/N.
// Bits 46-47 hold the descriptor version (1) that tcgen05 requires.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((saddr >> 4) & 0x3FFFu);
    d |= static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16;
    d |= static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    return d;
}

// Instruction descriptor, kind::f16: FP32 accumulator, FP16 A and B, both
// K-major, N = n, M = m.
__host__ __device__ constexpr uint32_t idesc_f16_f32(int m, int n) {
    return (1u << 4)                                   // D format: F32
           | (0u << 7) | (0u << 10)                    // A, B format: F16
           | (0u << 15) | (0u << 16)                   // A, B K-major
           | (static_cast<uint32_t>(n >> 3) << 17)     // N / 8
           | (static_cast<uint32_t>(m >> 4) << 24);    // M / 16
}

// --------------------------------------------------------------- misc ---
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&h);
}

__device__ __forceinline__ float2 unpack_half2(uint32_t w) {
    __half2 h = *reinterpret_cast<__half2 *>(&w);
    return __half22float2(h);
}

}  // namespace tcs
