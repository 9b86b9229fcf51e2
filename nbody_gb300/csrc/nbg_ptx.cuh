// nbg_ptx.cuh -- inline-PTX building blocks for sm_103a kernels: mbarriers
// with bounded waits, 1-D bulk async copies (TMA) global -> shared, packed
// FP32x2 arithmetic and the MUFU reciprocal square root.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace nbg {

// ---- launch order -----------------------------------------------------------
// Waits until the kernels queued before this one have finished and their
// writes are visible; the first statement of every kernel launched with
// queued() (a no-op in any other launch).  No kernel lets its successor in
// earlier (griddepcontrol.launch_dependents): waiting CTAs take the slots that
// let the last ones run alone, and an Euler step of 2^17 bodies took 566 us
// with it instead of 466.  Always true: the test, whose
// outcome the compiler does not know, keeps loads through the read-only path,
// which it may move across a mere memory clobber, behind the wait.
__device__ __forceinline__ bool after_previous() {
    unsigned sms;
    asm volatile("griddepcontrol.wait;\n\tmov.u32 %0, %%nsmid;" : "=r"(sms)::"memory");
    return sms != 0;
}

// ---- time ------------------------------------------------------------------
__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Wall-clock limit of every device-side wait (ns).  A healthy wait in these
// kernels lasts microseconds; on expiry the kernel records an error bit and
// leaves the loop instead of spinning forever.
constexpr uint64_t kWaitLimitNs = 2000000000ull;

// ---- mbarrier --------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
                 : "memory");
}

// Make initialised barriers visible to the async (bulk copy) proxy.
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Wait for the phase with the given parity to complete.  Returns false (and
// sets kDevErrTimeout in *err) if it does not complete within kWaitLimitNs.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, unsigned* err) {
#pragma unroll 1
    for (int i = 0; i < 128; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    uint64_t t0 = globaltimer_ns();
#pragma unroll 1
    while (true) {
        if (mbar_try_wait(bar, parity)) return true;
        if (globaltimer_ns() - t0 > kWaitLimitNs) {
            atomicOr(err, 1u /* kDevErrTimeout */);
            return false;
        }
    }
}

// ---- 1-D bulk async copy (TMA engine), completion via mbarrier tx count ----
// dst, src 16-byte aligned; bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst_smem, const void* src_gmem, uint32_t bytes,
                                         uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(smem_addr(dst_smem)),
        "l"(src_gmem), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}

// ---- shared-memory vector load (forces LDS.128 on a 32-bit shared address) ----
__device__ __forceinline__ float4 lds128(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(addr));
    return v;
}

// ---- packed FP32x2 arithmetic (sm_100+) -------------------------------------
typedef unsigned long long f2_t;  // two floats in one 64-bit register pair

__device__ __forceinline__ f2_t f2_pack(float lo, float hi) {
    f2_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(f2_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2_t f2_add(f2_t a, f2_t b) {
    f2_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2_t f2_sub(f2_t a, f2_t b) {
    f2_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2_t f2_mul(f2_t a, f2_t b) {
    f2_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2_t f2_fma(f2_t a, f2_t b, f2_t c) {
    f2_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// MUFU reciprocal square root (approximate, flush-to-zero).
__device__ __forceinline__ float rsqrt_mufu(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// MUFU reciprocal (approximate, flush-to-zero).
__device__ __forceinline__ float rcp_mufu(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The value of a two-word sum.  One that is not finite is in its high word (the
// low word's error terms are then inf - inf).
__device__ __forceinline__ double two_word_value(float hi, float lo) {
    return fabsf(hi) <= 3.402823466e38f ? (double)hi + (double)lo : (double)hi;
}

// Knuth two-sum in packed form: (hi, lo) += p with the rounding error of the
// high-part addition carried into lo.
__device__ __forceinline__ void f2_two_sum(f2_t& hi, f2_t& lo, f2_t p) {
    f2_t s = f2_add(hi, p);
    f2_t bp = f2_sub(s, hi);
    f2_t ap = f2_sub(s, bp);
    f2_t e = f2_add(f2_sub(hi, ap), f2_sub(p, bp));
    hi = s;
    lo = f2_add(lo, e);
}

}  // namespace nbg
