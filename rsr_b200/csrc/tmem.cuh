// tmem.cuh -- tensor memory (TMEM) as per-lane storage: allocation, and
// 32-bit loads and stores of P consecutive columns of a thread's own lane
// (shape 32x32b: a warp reaches the 32 lanes of its quadrant, warp w of a
// block lanes 32 (w % 4) .. +31).  The register adjoint keeps its tape
// here.  Stores are asynchronous (tm_wait_st before a load reads them);
// tm_ld waits for its own load, and the wait names the loaded registers so
// that no use of them is scheduled before it.  A block allocates with
// tm_alloc (one warp, which also gives up the right to allocate again),
// fences around the barrier that publishes the address, and frees with
// tm_dealloc before it exits.
#pragma once
#include <stdint.h>

#include "vm_ops.cuh"

namespace rsr {

__device__ __forceinline__ void tm_alloc(uint32_t *dst_smem, uint32_t ncols) {
    const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(dst_smem));
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tm_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tm_fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tm_fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tm_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

template <int P>
__device__ __forceinline__ void tm_st(uint32_t addr, const Vf<P> &v) {
    if constexpr (P == 2) {
        asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(__float_as_uint(v.v[0])),
                     "r"(__float_as_uint(v.v[1])) : "memory");
    } else if constexpr (P == 4) {
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr),
                     "r"(__float_as_uint(v.v[0])), "r"(__float_as_uint(v.v[1])), "r"(__float_as_uint(v.v[2])),
                     "r"(__float_as_uint(v.v[3])) : "memory");
    } else {
        static_assert(P == 8, "tape slots of 2, 4 or 8 columns");
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(addr),
                     "r"(__float_as_uint(v.v[0])), "r"(__float_as_uint(v.v[1])), "r"(__float_as_uint(v.v[2])),
                     "r"(__float_as_uint(v.v[3])), "r"(__float_as_uint(v.v[4])), "r"(__float_as_uint(v.v[5])),
                     "r"(__float_as_uint(v.v[6])), "r"(__float_as_uint(v.v[7])) : "memory");
    }
}

template <int P>
__device__ __forceinline__ void tm_ld_issue(Vf<P> &v, uint32_t addr) {
    if constexpr (P == 2) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=f"(v.v[0]), "=f"(v.v[1]) : "r"(addr) : "memory");
    } else if constexpr (P == 4) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v.v[0]), "=f"(v.v[1]), "=f"(v.v[2]), "=f"(v.v[3]) : "r"(addr) : "memory");
    } else {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=f"(v.v[0]), "=f"(v.v[1]), "=f"(v.v[2]), "=f"(v.v[3]), "=f"(v.v[4]), "=f"(v.v[5]), "=f"(v.v[6]), "=f"(v.v[7])
                     : "r"(addr) : "memory");
    }
}
// Names v's registers: no use of them is scheduled before the asm
// statements above this one.
template <int P>
__device__ __forceinline__ void tm_pin(Vf<P> &v) {
#pragma unroll
    for (int j = 0; j < P; ++j) asm volatile("" : "+f"(v.v[j]));
}
// W slots of P columns each from addr on: the loads in flight together, one
// wait, and the registers named after it.
template <int P, int W>
__device__ __forceinline__ void tm_ld(Vf<P> *v, uint32_t addr) {
#pragma unroll
    for (int c = 0; c < W; ++c) tm_ld_issue<P>(v[c], addr + c * (uint32_t)P);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int c = 0; c < W; ++c) tm_pin<P>(v[c]);
}

}  // namespace rsr
