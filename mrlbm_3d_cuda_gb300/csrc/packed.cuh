// Packed FP32 arithmetic (sm_100+ add / sub / mul / fma .rn.f32x2) and bulk-copy pipeline
// primitives of the step kernel.
#pragma once

#include <cstdint>

#include "kernels.h"

namespace mrlbm {

// Two floats in one 64-bit register pair.  Each lane of a packed operation rounds like the scalar
// instruction, so code written once for `float` and `V2` gives the same bits in both.
struct V2 {
    unsigned long long v;
};
__device__ __forceinline__ V2 v2(float a, float b) {
    V2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float lo(V2 a) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    return x;
}
__device__ __forceinline__ float hi(V2 a) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    return y;
}
__device__ __forceinline__ V2 add(V2 a, V2 b) {
    V2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ V2 sub(V2 a, V2 b) {
    V2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ V2 mul(V2 a, V2 b) {
    V2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ V2 fma(V2 a, V2 b, V2 c) {
    V2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
template <typename T>
__device__ __forceinline__ T bc(float c);
template <>
__device__ __forceinline__ float bc<float>(float c) { return c; }
template <>
__device__ __forceinline__ V2 bc<V2>(float c) { return v2(c, c); }

// ---- mbarriers and bulk copies (CTA-local) ---------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
// Waits for the phase of the given parity.  They give up after 1 + `limit` polls and return false: kWaitLimit polls
// that find nothing take 16 s (3.8 us each), far beyond any copy or plane of work.  (A suspend-time hint
// on the polls made them sleep: up to 2.5 times slower steps.)
__device__ __forceinline__ bool mbar_try(uint32_t a, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    return done != 0;
}
// The wait of a whole warp: its lanes poll each by itself and leave together, all with the same answer, so
// that what follows (shuffles, the release of a stage by lane 0) finds the warp whole.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, int limit) {
    const uint32_t a = smem_addr(bar);
    bool done = mbar_try(a, parity);
#pragma unroll 1
    for (int i = 0; !done && i < limit; ++i) done = mbar_try(a, parity);
    return __all_sync(0xffffffffu, done);
}
// The wait of one lane for what is on its way into shared memory, whatever limit the other waits have.
__device__ __forceinline__ bool mbar_wait_lane(uint64_t *bar, uint32_t parity) {
    const uint32_t a = smem_addr(bar);
#pragma unroll 1
    for (int i = 0; i < kWaitLimit; ++i)
        if (mbar_try(a, parity)) return true;
    return false;
}

// Hand-off between two warps at a named barrier (hardware: the waiting warp does not poll).
__device__ __forceinline__ void token_wait(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void token_pass(int id) { asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory"); }

// Copy `bytes` (a multiple of 16; both addresses 16-byte aligned) into shared memory; completes on `bar`.
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

// Words that are not kept in L1.
__device__ __forceinline__ uint32_t load_uncached(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.global.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ void store_uncached(uint32_t *p, uint32_t a) {
    asm volatile("st.global.L1::no_allocate.b32 [%0], %1;" ::"l"(p), "r"(a) : "memory");
}
__device__ __forceinline__ void store_uncached(uint32_t *p, uint32_t a, uint32_t b) {
    asm volatile("st.global.L1::no_allocate.v2.b32 [%0], {%1, %2};" ::"l"(p), "r"(a), "r"(b) : "memory");
}

// Cluster launch control: a running CTA takes over a CTA of its grid that has not started yet.
// request: asynchronously into the 16-byte `slot`, completing 16 bytes on `bar`; result: the index of the
// CTA taken over, or -1 when none is left (no further request is made then).
__device__ __forceinline__ void takeover_request(void *slot, uint64_t *bar) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.relaxed.cta.shared::cta.b64 _, [%0], 16;" ::"r"(smem_addr(bar)) : "memory");
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
                     smem_addr(slot)),
                 "r"(smem_addr(bar))
                 : "memory");
}
__device__ __forceinline__ int takeover_result(const void *slot) {
    int x;
    asm volatile(
        "{\n\t.reg .b128 h;\n\t.reg .pred p;\n\t.reg .b32 y, z, w;\n\t"
        "ld.shared.b128 h, [%1];\n\t"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
        "mov.b32 %0, -1;\n\t"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%0, y, z, w}, h;\n\t}"
        : "=r"(x)
        : "r"(smem_addr(slot))
        : "memory");
    return x;
}

}  // namespace mrlbm
