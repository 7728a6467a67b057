// kernels_common.cuh -- pieces shared by the evaluation kernels: launch
// arguments, per-tile data access, compensated accumulation and the warp
// reduction of partial sums.
#pragma once
#include <stdint.h>

#include <atomic>

#include <cuda_runtime.h>

#include "lane_layout.h"
#include "uops.h"
#include "vm_ops.cuh"

namespace rsr {

enum EvalMode : int { MODE_MSE = 0, MODE_POINTS = 1 };

struct LaunchArgs {
    const ProgDesc *progs;
    const DatasetDesc *datasets;
    const WorkItem *items;
    const uint32_t *code;     // code pool
    const float *consts;      // constant pool
    double *partials;         // per (program, chunk) sums; gradient: (1+32) per slot
    float *points_out;        // MODE_POINTS: predictions
    uint64_t points_stride;   // MODE_POINTS: floats between consecutive programs
    uint32_t *item_counter;   // persistent kernels: next work item; 0 before and after a launch
    float *mse_out;           // register kernels, when every program has one part: the epilogue's
    float *grad_out;          // results, written by the item's block (no finalize launch); else null
    const uint8_t *active;    // optional per-program mask (launch order): 0 = skip
    const uint32_t *run_if;   // optional: the launch does nothing when *run_if == 0 (device-side
                              // loops whose later rounds may have no work, e.g. line searches)
    uint32_t n_items;
    uint32_t mode;
    uint32_t smem_code_words; // per warp
    uint32_t smem_const_floats;
    uint32_t smem_slots;      // per warp (slot-file kernels; adjoint: value slots)
    uint32_t smem_adj_slots;  // per warp (adjoint: adjoint slots)
    uint32_t progs_per_warp;
    // register kernel: per-warp shared-memory layout (floats)
    uint32_t region_floats;   // per warp
    uint32_t block_hdr_floats;
    uint32_t acc_off;
    uint32_t stack_off[N_STACKS];
    uint32_t tmem_cols;       // register adjoint: tensor-memory columns of a block's tapes
};

// Opt-in dynamic shared-memory limit of one block on sm_100 (227 KB).  Every
// launcher raises its kernel's limit to this value rather than to the launch's
// own size: the limit is per-function state shared by all host threads, and a
// launch from one thread must not see it lowered by another thread.
constexpr int kMaxDynSmemOptin = 227 * 1024;

// Raises kernel k's dynamic shared-memory limit to kMaxDynSmemOptin once per
// device: `done` (a static of the caller's instance) holds one bit per
// device on which it is set, so later launches skip the driver call.
template <typename K>
__host__ inline cudaError_t raise_smem_limit(K k, std::atomic<uint64_t> &done) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmemOptin);
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return e;
}

// Kahan-compensated single-precision running sum (one per lane).
struct Kahan {
    float s = 0.0f, c = 0.0f;
    __device__ __forceinline__ void add(float v) {
        const float y = v - c;
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
    __device__ __forceinline__ double value() const { return (double)s - (double)c; }
};

// The epilogue of compute_mse (evaluator.rs:166-173): a sum that the
// reference's f32 accumulator would have overflowed, or a quotient that is not
// finite, gives f32::MAX (returns false).
__device__ __forceinline__ bool mse_of_sum(double s, uint64_t num_samples, float *mse) {
    const float m = (float)(s / (double)num_samples);
    const bool ok = s <= (double)3.402823466e38f && fabsf(m) <= 3.402823466e38f;
    *mse = ok ? m : 3.402823466e38f;
    return ok;
}

// The next work item of a persistent launch.  Every block ends on one number
// past the last item; the block that draws the last of those sets the counter
// back to 0 for the plan's next launch.
__device__ __forceinline__ uint32_t next_item(uint32_t *counter, uint32_t n_items) {
    const uint32_t id = atomicAdd(counter, 1u);
    if (id == n_items + gridDim.x - 1u) *counter = 0u;
    return id;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Loads P consecutive floats starting at a P-aligned index.
template <int P>
__device__ __forceinline__ Vf<P> load_pts(const float *__restrict__ p) {
    Vf<P> r;
    if constexpr (P == 1) {
        r.v[0] = __ldg(p);
    } else if constexpr (P == 2) {
        float2 a = __ldg(reinterpret_cast<const float2 *>(p));
        r.v[0] = a.x; r.v[1] = a.y;
    } else {
#pragma unroll
        for (int j = 0; j < P / 4; ++j) {
            float4 a = __ldg(reinterpret_cast<const float4 *>(p) + j);
            r.v[4 * j] = a.x; r.v[4 * j + 1] = a.y; r.v[4 * j + 2] = a.z; r.v[4 * j + 3] = a.w;
        }
    }
    return r;
}

template <int P>
__device__ __forceinline__ void store_pts(float *p, const Vf<P> &v, uint64_t first, uint64_t limit) {
#pragma unroll
    for (int k = 0; k < P; ++k)
        if (first + k < limit) p[k] = v.v[k];
}

// Loads a lane's P values; p points at its first (tile start + lane_point(lane, 0)).
template <int P>
__device__ __forceinline__ Vf<P> load_lane(const float *__restrict__ p) {
    if constexpr (P <= 4) {
        return load_pts<P>(p);
    } else {
        Vf<P> r;
#pragma unroll
        for (int j = 0; j < P / 4; ++j) {
            const float4 a = __ldg(reinterpret_cast<const float4 *>(p + j * 128));
            r.v[4 * j] = a.x; r.v[4 * j + 1] = a.y; r.v[4 * j + 2] = a.z; r.v[4 * j + 3] = a.w;
        }
        return r;
    }
}

// Shared memory by 32-bit address, for what an interpreter loop keeps in
// registers across its switch; opaque() so that the compiler holds such a value
// instead of building it again in the loop from what it came from (a lane's
// feature address from the thread index, a program's constants from the launch
// arguments).  Without opaque -> with it: 4096 vector programs x 100k points 2.35 ->
// 2.30 ms, their gradients 10.99 -> 10.67, 256 matrix programs x 1M points 2.13 ->
// 1.92, 8192 2x2 matrix programs over 16 data sets 8.57 -> 7.71.
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint32_t opaque(uint32_t v) {
    asm volatile("" : "+r"(v));
    return v;
}
template <typename T>
__device__ __forceinline__ T *opaque(T *p) {
    asm volatile("" : "+l"(p));
    return p;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
    uint32_t r;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r) : "r"(a));
    return r;
}
__device__ __forceinline__ uint2 lds_u32x2(uint32_t a) {
    uint2 r;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "r"(a));
    return r;
}
__device__ __forceinline__ void sts_f32(uint32_t a, float v) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ double lds_f64(uint32_t a) {
    double r;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(r) : "r"(a));
    return r;
}
__device__ __forceinline__ void sts_f64(uint32_t a, double v) {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ float2 lds_f32x2(uint32_t a) {
    float2 r;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(r.x), "=f"(r.y) : "r"(a));
    return r;
}
__device__ __forceinline__ void sts_f32x2(uint32_t a, float x, float y) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ float lds_f32(uint32_t a) { return __uint_as_float(lds_u32(a)); }

// Shared-memory image of a lane's P values in a block of 32*P floats; a is
// the address of the lane's first value (block start + lane_point(lane, 0)).
template <int P>
__device__ __forceinline__ Vf<P> lds_lane(uint32_t a) {
    Vf<P> r;
    if constexpr (P == 2) {
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(r.v[0]), "=f"(r.v[1]) : "r"(a));
    } else {
#pragma unroll
        for (int j = 0; j < P / 4; ++j)
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(r.v[4 * j]), "=f"(r.v[4 * j + 1]), "=f"(r.v[4 * j + 2]), "=f"(r.v[4 * j + 3])
                         : "r"(a + 512u * j));
    }
    return r;
}

template <int P>
__device__ __forceinline__ void sts_lane(uint32_t a, const Vf<P> &v) {
    if constexpr (P == 2) {
        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.v[0]), "f"(v.v[1]) : "memory");
    } else {
#pragma unroll
        for (int j = 0; j < P / 4; ++j)
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a + 512u * j), "f"(v.v[4 * j]),
                         "f"(v.v[4 * j + 1]), "f"(v.v[4 * j + 2]), "f"(v.v[4 * j + 3])
                         : "memory");
    }
}

// Stores the lane's values whose points lie below `limit`; `tile` is the
// tile's first point, p the output's value of point `tile`.
template <int P>
__device__ __forceinline__ void store_lane(float *p, int lane, const Vf<P> &v, uint64_t tile, uint64_t limit) {
#pragma unroll
    for (int q = 0; q < P; ++q) {
        const uint32_t o = lane_point<P>(lane, q);
        if (tile + o < limit) p[o] = v.v[q];
    }
}

}  // namespace rsr
