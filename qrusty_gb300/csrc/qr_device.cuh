// qr_device.cuh -- device helpers shared by the apply kernels: mbarriers and
// 1-D TMA bulk copies in inline PTX, and FP64 bit tricks on the integer pipe.
#pragma once

#include <cstdint>

namespace qr {

__device__ __forceinline__ uint32_t saddr(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes,
                                         uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(saddr(dst)),
        "l"(src), "r"(bytes), "r"(saddr(bar))
        : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(saddr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t gtimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait: gives up after ~limit_ns and reports false.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity,
                                                  uint64_t limit_ns) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = gtimer_ns();
    while (!mbar_try_wait(bar, parity)) {
        if (gtimer_ns() - t0 > limit_ns) return false;
    }
    return true;
}

constexpr uint64_t kWaitLimitNs = 2000000000ull;  // 2 s per stage

// Error-free addition on (re, im) at once with packed FP32
// operations; x - y is formed as fma(y, -1, x) (y * -1 is exact, so the one
// rounding is that of x - y).
__device__ __forceinline__ float2 sub2_rn(float2 x, float2 y) {
    return __ffma2_rn(y, make_float2(-1.f, -1.f), x);
}
// hi += b with an error-free transformation; returns the error term
// instead of accumulating it
__device__ __forceinline__ float2 two_sum_carry2(float2 &hi, float2 b) {
    const float2 s = __fadd2_rn(hi, b);
    const float2 bb = sub2_rn(s, hi);
    const float2 e = __fadd2_rn(sub2_rn(hi, sub2_rn(s, bb)), sub2_rn(b, bb));
    hi = s;
    return e;
}
__device__ __forceinline__ float flip(float d, uint32_t s) {
    return __uint_as_float(__float_as_uint(d) ^ (s << 31));
}
// d with the sign bit flipped when s == 1; bits that are zero iff d is +0 or
// -0; the exponent bits (all ones: infinite or NaN).  Integer pipe.
__device__ __forceinline__ double flip(double d, uint32_t s) {
    return __hiloint2double(__double2hiint(d) ^ (int)(s << 31), __double2loint(d));
}
__device__ __forceinline__ uint32_t mag_bits(double d) {
    return ((uint32_t)__double2hiint(d) << 1) | (uint32_t)__double2loint(d);
}
__device__ __forceinline__ uint32_t exp_bits(double d) {
    return (uint32_t)__double2hiint(d) & 0x7ff00000u;
}

}  // namespace qr
