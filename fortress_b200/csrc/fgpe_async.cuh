// fgpe_async.cuh -- asynchronous copies from global to shared memory.
#pragma once
#include "fgpe_device.cuh"

namespace fgpe {

#ifdef FGPE_CHECK_ALIGN
// Diagnostic build only: record the first misaligned copy and skip it.
static __device__ unsigned long long g_align_fault[4];
__device__ __forceinline__ bool align_bad(const void* s, const void* g, unsigned bytes, int site) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(s);
    if ((d % bytes) == 0 && ((unsigned long long)g % bytes) == 0) return false;
    if (atomicCAS(&g_align_fault[0], 0ull, 1ull) == 0ull) {
        g_align_fault[1] = (unsigned long long)site;
        g_align_fault[2] = d;
        g_align_fault[3] = (unsigned long long)g;
    }
    return true;
}
#define FGPE_ALIGN_GUARD(s, g, b, site) if (align_bad(s, g, b, site)) return
#else
#define FGPE_ALIGN_GUARD(s, g, b, site)
#endif

__device__ __forceinline__ void cp16(void* smem_dst, const void* gsrc) {
    FGPE_ALIGN_GUARD(smem_dst, gsrc, 16, 16);
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp8(void* smem_dst, const void* gsrc) {
    FGPE_ALIGN_GUARD(smem_dst, gsrc, 8, 8);
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(gsrc) : "memory");
}
// One complex element: 16-byte copy for complex128, 8-byte for complex64 (the
// padded row layout puts complex64 elements on 8-byte boundaries only).
template <typename T> __device__ __forceinline__ void cp_elem(cx<T>* smem_dst, const cx<T>* gsrc) {
    if constexpr (sizeof(cx<T>) == 16) cp16(smem_dst, gsrc);
    else cp8(smem_dst, gsrc);
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

}  // namespace fgpe
