// Tensor memory as per-thread storage (sm_100a), for the step kernels.
#pragma once
#include <cstdint>

namespace mb {

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- tensor memory: warp w of a CTA owns lanes 32 (w % 4) .. + 31 and its
// share of the columns; thread t of the warp holds one word per column
template <int N>
__device__ __forceinline__ void tm_ld(uint32_t addr, uint32_t (&r)[N]) {
    static_assert(N == 1 || N == 2 || N == 4, "");
    if constexpr (N == 1)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r[0]) : "r"(addr));
    else if constexpr (N == 2)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
    else  // (the wait before the first use names the registers)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(addr));
}
__device__ __forceinline__ void tm_st(uint32_t addr, uint32_t v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void tm_st2(uint32_t addr, uint32_t a, uint32_t b) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void tm_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Allocates `cols` columns (a power of two >= 32) for the CTA; returns the base
// address to every thread.  `slot`: a shared word, free again on return.  All
// threads call it.
__device__ __forceinline__ uint32_t tm_alloc(uint32_t* slot, uint32_t cols) {
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)), "r"(cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t base = *reinterpret_cast<volatile uint32_t*>(slot);
    __syncthreads();  // the word is free again
    return base;
}
__device__ __forceinline__ void tm_free(uint32_t base, uint32_t cols) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols));
    }
}

}  // namespace mb
