// TMA bulk copies from global to shared memory, completing on mbarriers, and the bounded
// waits for them.
#pragma once

#include <cstdint>

namespace awg {

__device__ __forceinline__ unsigned smem_u32(const void *p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
// Global -> shared bulk copy: both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t *bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
constexpr int WAIT_TRIES = 1 << 22;  // try_wait rounds before a wait gives up
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity) {
    for (int it = 0; it < WAIT_TRIES; it++)
        if (mbar_test(bar, parity)) return true;
    return false;
}

// count elements of ESZ bytes at p, copied from the 16-byte boundary below p: the bytes to
// copy (a multiple of 16) and the element offset of p inside the copy.
template <int ESZ>
struct Rounded {
    const char *a16;
    unsigned bytes;
    int off;
    __device__ __forceinline__ Rounded(const void *p, long long count) {
        a16 = (const char *)((uintptr_t)p & ~(uintptr_t)15);
        off = (int)(((uintptr_t)p & 15) / ESZ);
        bytes = count > 0 ? (unsigned)(((const char *)p + ESZ * count - a16 + 15) & ~(long long)15) : 0u;
    }
};

}  // namespace awg
