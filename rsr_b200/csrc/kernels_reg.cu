// kernels_reg.cu -- the batched register kernel: an accumulator machine.
//
// Each value type of the reference VM (state.rs:12-37) has one accumulator
// register set holding P data points per lane: A_F, A_V2[2], A_V3[3],
// A_M2[4], A_M3[9].  Micro-ops (uops.h, accumulator form) combine an
// accumulator with a feature, a constant, a value spilled to a per-type
// stack in shared memory (slot fixed by the encoder), or another type's
// accumulator, so dispatch is on the micro-op kind alone (about 140 cases,
// one code block each) and values never leave registers except for spills.
//
// The kernel is persistent: warps pull work items (up to 8 programs sharing a
// dataset, on a chunk of point tiles) from a global counter, so uneven
// program lengths and dataset sizes balance across the 148 SMs; all programs
// of an item run on each tile while its features are hot in L1.
#include <cuda_runtime.h>

#include "acc_ops.cuh"
#include "kernels.h"
#include "kernels_common.cuh"

namespace rsr {

#define RSR_C(K) case (K): acc_op<PROF, P, (K)>(a, io, arg); handler_end<(K)>(); break;
#define RSR_C4(K) RSR_C(K) RSR_C(K + 1) RSR_C(K + 2) RSR_C(K + 3)
#define RSR_C9(K) RSR_C4(K) RSR_C4(K + 4) RSR_C(K + 8)
#define RSR_C27(K) RSR_C9(K) RSR_C9(K + 9) RSR_C9(K + 18)
#define RSR_BLOCK_F RSR_C27(K_F)     // 0..26
#define RSR_BLOCK_F_NU RSR_C9(K_F) RSR_C9(K_F + 9) RSR_C(K_F + 18) RSR_C(K_F + 19) RSR_C(K_F + 20)  // 0..20
static_assert(K_F_UN == K_F + 21 && K_F_END == K_F + 27, "Float block: 21 kinds, then the 6 unary ones");
// Vec3 block without the mat-vec kinds whose matrix is a feature, a constant
// or a spilled value (64 + 30..32)
#define RSR_BLOCK_V3_NM RSR_C27(K_V3) RSR_C(K_V3 + 27) RSR_C(K_V3 + 28) RSR_C(K_V3 + 29) RSR_C(K_V3 + 33)
static_assert(kv_mulm(5, 3) == 29 && kv_make(5, 3) == 33, "Vec3 block: mat-vec kinds at 29..32");
// Vec3 block as the F+V3 profile can meet it: a mat-vec with a spilled matrix
// (64 + 32) needs a Mat3 accumulator, which that profile does not have
#define RSR_BLOCK_V3_F RSR_C27(K_V3) RSR_C4(K_V3 + 27) RSR_C(K_V3 + 31) RSR_C(K_V3 + 33)
#define RSR_BLOCK_V2 RSR_C27(K_V2)   // 32..58
#define RSR_BLOCK_V3 RSR_C27(K_V3) RSR_C4(K_V3 + 27) RSR_C(K_V3 + 31) RSR_C(K_V3 + 32) RSR_C(K_V3 + 33)  // 64..97
#define RSR_BLOCK_M2 RSR_C27(K_M2)   // 104..130
#define RSR_BLOCK_M3 RSR_C27(K_M3)   // 136..162

// A prologue's store (uops.h, hoisted constants): every lane holds the same
// value, and writes it.
template <int PROF, int P, int t>
__device__ __forceinline__ void store_const(Acc<PROF, P> &a, const AccIO<P> &io, uint32_t off) {
    if constexpr (((kProfileTypes[PROF] >> t) & 1u) != 0u) {
        constexpr int W = kStackWidth[t];
        const Vf<P> *A = acc_of<PROF, P, t>(a);
#pragma unroll
        for (int c = 0; c < W; ++c) sts_f32(io.consts + 4u * (off + c), A[c].v[0]);
    }
}

// Runs one program (accumulator form, ended by a K_STOP word) on this lane's
// P points; the result is left in A_F.  OMIT: handlers left out of the kernel
// because no program of the launch needs them -- bit 0: the unary Float ops
// (sin, cos, exp, sqr, sqrt, ln); bit 1 (F+V3 profile): mat-vec products whose
// matrix is a feature, a constant or a spilled value.
//
// What bounds it is the dispatch around the P x width FP32 instructions of a
// micro-op, so the loop holds nothing else: the switch is a jump table
// (built with --jump-table-density, build.py) over the kinds the encoder can
// emit for the profile, with no range check (the default is unreachable), and
// the program ends by a micro-op instead of a counter.
#define RSR_RUN(CASES)                                                   \
    switch (w & 0xFFu) {                                                 \
        CASES                                                            \
        RSR_STORES                                                       \
        case K_STOP: return;                                             \
        default: __builtin_unreachable();                                \
    }
#define RSR_S(T) case kTapeKind[T]: store_const<PROF, P, (T)>(a, io, arg); handler_end<kTapeKind[T]>(); break;
#define RSR_STORES RSR_S(SF) RSR_S(SV2) RSR_S(SV3) RSR_S(SM2) RSR_S(SM3)
template <int PROF, int P, int OMIT>
__device__ __forceinline__ void run_program(Acc<PROF, P> &a, const AccIO<P> &io, uint32_t code) {
    constexpr bool NU = (OMIT & 1) != 0, NM = (OMIT & 2) != 0;
    uint32_t w = lds_u32(code);
#pragma unroll 1
    for (;;) {
        code += 4u;
        const uint32_t wn = lds_u32(code);  // the word after K_STOP is read, not run
        const uint32_t arg = w >> 8;
        if constexpr (PROF == P_F && NU) { RSR_RUN(RSR_BLOCK_F_NU) }
        else if constexpr (PROF == P_F) { RSR_RUN(RSR_BLOCK_F) }
        else if constexpr (PROF == P_FV3 && NU && NM) { RSR_RUN(RSR_BLOCK_F_NU RSR_BLOCK_V3_NM) }
        else if constexpr (PROF == P_FV3 && NU) { RSR_RUN(RSR_BLOCK_F_NU RSR_BLOCK_V3_F) }
        else if constexpr (PROF == P_FV3 && NM) { RSR_RUN(RSR_BLOCK_F RSR_BLOCK_V3_NM) }
        else if constexpr (PROF == P_FV3) { RSR_RUN(RSR_BLOCK_F RSR_BLOCK_V3_F) }
        else if constexpr (PROF == P_FV2M2 && NU) { RSR_RUN(RSR_BLOCK_F_NU RSR_BLOCK_V2 RSR_BLOCK_M2) }
        else if constexpr (PROF == P_FV2M2) { RSR_RUN(RSR_BLOCK_F RSR_BLOCK_V2 RSR_BLOCK_M2) }
        else if constexpr (PROF == P_FV3M3) { RSR_RUN(RSR_BLOCK_F RSR_BLOCK_V3 RSR_BLOCK_M3) }
        else { RSR_RUN(RSR_BLOCK_F RSR_BLOCK_V2 RSR_BLOCK_V3 RSR_BLOCK_M2 RSR_BLOCK_M3) }
        w = wn;
    }
}

#undef RSR_RUN
#undef RSR_STORES
#undef RSR_S
#undef RSR_BLOCK_F
#undef RSR_BLOCK_F_NU
#undef RSR_BLOCK_V3_NM
#undef RSR_BLOCK_V3_F
#undef RSR_BLOCK_V2
#undef RSR_BLOCK_V3
#undef RSR_BLOCK_M2
#undef RSR_BLOCK_M3
#undef RSR_C27
#undef RSR_C9
#undef RSR_C4
#undef RSR_C

__host__ __device__ __forceinline__ uint32_t align4r(uint32_t v) { return (v + 3u) & ~3u; }

constexpr uint32_t kMaxProgsPerWarp = 8;
static_assert(kMaxProgsPerWarp <= kRegThreads / 32, "a warp for each program's prologue");
constexpr uint32_t kPrologue = 0xFFFFFFFFu;  // the tile that stands for an item's prologues
constexpr uint32_t kEnd = 0xFFFFFFFFu;       // no program at this address

// What a block keeps of its work item in shared memory (words).
enum RegMeta : uint32_t {
    M_PROGS = 0,       // [g][2] shared-memory addresses of each program's code and constants, kEnd behind the last
    M_Y_OFF = 18,      // targets' byte distance from the features
    M_N_EVAL = 20,     // points to count
    M_ITEM = 22, M_FULL_TILES, M_TILE_BEGIN, M_TILE_END, M_PROG_BEGIN, M_HOISTED,
    kMetaWords = 32,
    // [g] address of its prologue, kEnd if it has none: in the room of the
    // cross-warp sums, which are written when every prologue has run
    M_PROLOGUES = kMetaWords
};
static_assert(M_Y_OFF == M_PROGS + 2 * (kMaxProgsPerWarp + 1) && M_HOISTED < kMetaWords && kMetaWords % 4 == 0,
              "RegMeta layout");

// Block-cooperative item loop.  All warps of a block run the same programs
// (one work item) on different tiles of the item's chunk, so the SM's
// instruction cache holds one program's case bodies instead of one per warp.
// Per-warp Kahan sums are reduced across warps in a fixed order.
//
// Shared memory: block header (code | constants | meta | cross-warp sums)
// then one region per warp (spill stacks | Kahan state).
// Blocks per SM each instance is compiled for (the register cap follows): as
// many as its accumulators allow, with a few bytes of spill where one more block
// is worth them.  Device time against one block fewer: F and F+V3 at eight
// points, a third (80 registers, up to 32 bytes of spill stores), 4096 vector
// programs x 100k points 2.68 -> 2.30 ms, 256 matrix programs x 1M points 2.12 ->
// 1.92, 1024 scalar programs x 100k points 0.87 -> 0.79; F+V2+M2 would spill several
// accumulators there.  F+V2+M2 at four points, a fourth (64 registers, 12 bytes):
// 8192 programs over 16 data sets 7.73 -> 7.71, as much as that measurement can tell.
template <int PROF, int P, int OMIT>
constexpr int reg_min_blocks() {
    if constexpr (PROF == P_ALL) return P >= 4 ? 1 : 2;
    else if constexpr (PROF == P_FV3M3) return P >= 4 ? 2 : 3;
    else if constexpr (PROF == P_FV2M2) return P >= 8 ? 2 : 4;
    else return P >= 8 ? 3 : 4;
}

template <int PROF, int P, int OMIT>
__global__ void __launch_bounds__(kRegThreads, reg_min_blocks<PROF, P, OMIT>()) reg_eval_kernel(const LaunchArgs a) {
    extern __shared__ __align__(16) float smem[];
    if (a.run_if && *a.run_if == 0u) return;  // the same for every thread of the launch
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nw = blockDim.x >> 5;
    uint32_t *scode = reinterpret_cast<uint32_t *>(smem);
    float *sconst = smem + align4r(a.smem_code_words);
    uint32_t *meta = reinterpret_cast<uint32_t *>(sconst + align4r(a.smem_const_floats));  // RegMeta
    double *red = reinterpret_cast<double *>(meta + kMetaWords);  // [warp][g]
    float *wbase = smem + a.block_hdr_floats + (size_t)warp * a.region_floats;
    // Kahan state of this warp: (sum, compensation) of each lane, 256 bytes a program
    const uint32_t kahan = smem_addr(wbase + a.acc_off) + 8u * lane;

    AccIO<P> io;
#pragma unroll
    for (int t = 0; t < N_STACKS; ++t) io.stk[t] = opaque(smem_addr(wbase + a.stack_off[t] + lane_point<P>(lane, 0)));

    for (;;) {
        if (threadIdx.x == 0) meta[M_ITEM] = next_item(a.item_counter, a.n_items);
        __syncthreads();
        const uint32_t item_id = meta[M_ITEM];
        if (item_id >= a.n_items) break;
        const WorkItem it = a.items[item_id];
        const uint32_t G = it.n_progs;
        if (a.active) {
            // an item whose programs have all finished (fits) is skipped whole;
            // the flags are the same for every thread of the block
            bool any = false;
            for (uint32_t g = 0; g < G; ++g) any |= a.active[it.prog_begin + g] != 0;
            if (!any) {
                __syncthreads();  // M_ITEM is rewritten by the next item fetch
                continue;
            }
        }
        // The item's programs lie one after another in the code and constant
        // pools, as they do here (every program ended by its K_STOP, followed
        // by room for its hoisted constants), so one copy each stages them,
        // while warp 0's lanes lay down where each begins.
        const DatasetDesc ds = a.datasets[it.dataset];
        const uint32_t code0 = a.progs[it.prog_begin].uop_off, const0 = a.progs[it.prog_begin].const_off;
        const ProgDesc &last = a.progs[it.prog_begin + G - 1];
        const uint32_t n_code = last.uop_off + last.uop_len + 1u - code0;
        const uint32_t n_const = last.const_off + last.n_consts + last.n_tape - const0;
        for (uint32_t i = threadIdx.x; i < n_code; i += blockDim.x) scode[i] = __ldg(a.code + code0 + i);
        for (uint32_t i = threadIdx.x; i < n_const; i += blockDim.x) sconst[i] = __ldg(a.consts + const0 + i);
        for (uint32_t g = 0; g < G; ++g) sts_f32x2(kahan + 256u * g, 0.0f, 0.0f);
        if (warp == 0) {
            bool hoisted = false;
            if (lane < (int)G) {
                const ProgDesc &pd = a.progs[it.prog_begin + lane];
                const uint32_t code = smem_addr(scode + (pd.uop_off - code0));
                hoisted = pd.n_slots != 0u;
                meta[M_PROGS + 2 * lane] = code + 4u * pd.n_slots;
                meta[M_PROGS + 2 * lane + 1] = smem_addr(sconst + (pd.const_off - const0));
                meta[M_PROLOGUES + lane] = hoisted ? code : kEnd;
            } else if (lane <= (int)kMaxProgsPerWarp) {
                meta[M_PROGS + 2 * lane] = kEnd;
                if (lane < (int)kMaxProgsPerWarp) meta[M_PROLOGUES + lane] = kEnd;
            }
            hoisted = __any_sync(0xffffffffu, hoisted);
            if (lane == 0) {
                *reinterpret_cast<int64_t *>(meta + M_Y_OFF) =
                    reinterpret_cast<const char *>(ds.y) - reinterpret_cast<const char *>(ds.x);
                *reinterpret_cast<uint64_t *>(meta + M_N_EVAL) = ds.n_eval;
                meta[M_FULL_TILES] = (uint32_t)(ds.n_eval / (32u * P));
                meta[M_TILE_END] = it.tile_end;
                meta[M_TILE_BEGIN] = it.tile_begin;
                meta[M_PROG_BEGIN] = it.prog_begin;
                meta[M_HOISTED] = hoisted;
            }
        }
        __syncthreads();
        io.stride = opaque((uint32_t)ds.stride);
        Acc<PROF, P> acc;
        // What the loops need beside the program itself -- their bounds, the
        // targets, the dataset's end -- is read again for every program
        // (shared memory and L1): held in registers it would be live across
        // the interpreter, which has none to spare at three blocks an SM.
        const volatile uint32_t *vmeta = meta;
        // The item's prologues come first, as tile kPrologue: warp g runs
        // program g's (one call of the interpreter in the kernel), then the
        // block goes on to the tiles.
        uint32_t tile = vmeta[M_HOISTED] ? kPrologue : it.tile_begin + warp;
        for (;;) {
            if (tile != kPrologue && tile >= vmeta[M_TILE_END]) break;
            io.xl = opaque(ds.x + ((uint64_t)tile * (32u * P) + lane_point<P>(lane, 0)));
            for (uint32_t g = tile == kPrologue ? (uint32_t)warp : 0u;; ++g) {
                uint2 at = lds_u32x2(smem_addr(meta) + 4u * M_PROGS + 8u * g);  // code, constants
                if (tile == kPrologue) at.x = vmeta[M_PROLOGUES + warp];
                if (at.x == kEnd) break;  // no further program, or no prologue
                if (a.active && !a.active[vmeta[M_PROG_BEGIN] + g]) {
                    if (tile == kPrologue) break;
                    continue;
                }
                io.consts = opaque(at.y);
                run_program<PROF, P, OMIT>(acc, io, opaque(at.x));
                if (tile == kPrologue) break;
                const Vf<P> pred = acc.F[0];
                if (a.mode == MODE_POINTS) {
                    const uint64_t t0 = (uint64_t)tile * (32u * P);
                    store_lane<P>(a.points_out + (uint64_t)(vmeta[M_PROG_BEGIN] + g) * a.points_stride + t0, lane,
                                  pred, t0, *reinterpret_cast<const volatile uint64_t *>(vmeta + M_N_EVAL));
                    continue;
                }
                const int64_t y_off = *reinterpret_cast<const volatile int64_t *>(vmeta + M_Y_OFF);
                const Vf<P> y = load_lane<P>(
                    reinterpret_cast<const float *>(reinterpret_cast<const char *>(io.xl) + y_off));
                const float2 sc = lds_f32x2(kahan + 256u * g);
                Kahan k;
                k.s = sc.x;
                k.c = sc.y;
                bool full = tile < vmeta[M_FULL_TILES];
                if (!full) {  // the dataset's last tile: lanes whose points all lie inside
                    const uint64_t n_eval = *reinterpret_cast<const volatile uint64_t *>(vmeta + M_N_EVAL);
                    const uint64_t t0 = (uint64_t)tile * (32u * P);
                    full = t0 + lane_point<P>(lane, P - 1) < n_eval;
                    if (!full) {
#pragma unroll
                        for (int q = 0; q < P; ++q) {
                            if (t0 + lane_point<P>(lane, q) < n_eval) {
                                const float d = pred.v[q] - y.v[q];
                                k.add(d * d);
                            }
                        }
                    }
                }
                if (full) {
                    // the lane's P squared errors summed pairwise, then one
                    // compensated add per tile
                    float sq[P];
#pragma unroll
                    for (int q = 0; q < P; ++q) {
                        const float d = pred.v[q] - y.v[q];
                        sq[q] = d * d;
                    }
#pragma unroll
                    for (int h = P / 2; h > 0; h /= 2)
#pragma unroll
                        for (int q = 0; q < h; ++q) sq[q] = sq[q] + sq[q + h];
                    k.add(sq[0]);
                }
                sts_f32x2(kahan + 256u * g, k.s, k.c);
            }
            if (tile == kPrologue) {
                __syncthreads();
                tile = vmeta[M_TILE_BEGIN] + warp;
            } else {
                tile += nw;
            }
        }
        if (a.mode == MODE_MSE) {
            for (uint32_t g = 0; g < G; ++g) {
                const float2 sc = lds_f32x2(kahan + 256u * g);
                Kahan k;
                k.s = sc.x;
                k.c = sc.y;
                const double s = warp_sum(k.value());
                if (lane == 0) red[warp * kMaxProgsPerWarp + g] = s;
            }
            __syncthreads();
            if (threadIdx.x < G) {
                double s = 0.0;
                for (int w = 0; w < nw; ++w) s += red[w * kMaxProgsPerWarp + threadIdx.x];
                const uint32_t p = it.prog_begin + threadIdx.x;
                if (a.mse_out)
                    mse_of_sum(s, ds.num_samples, a.mse_out + p);
                else
                    a.partials[a.progs[p].part_off + it.chunk] = s;
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------- launchers
// Shared-memory layout (floats).  Block header: code | constants | RegMeta |
// cross-warp sums (kRegThreads/32 x 8 doubles).  Per warp: stacks
// (per type) | Kahan state.
void reg_layout(uint32_t code_words, uint32_t const_floats, const uint32_t *stack_depth, int P, int G,
                uint32_t *stack_off, uint32_t *acc_off, uint32_t *region_floats, uint32_t *block_hdr_floats) {
    *block_hdr_floats = align4r(code_words) + align4r(const_floats) + kMetaWords + 2u * (kRegThreads / 32) * kMaxProgsPerWarp;
    uint32_t off = 0;
    for (int t = 0; t < N_STACKS; ++t) {
        stack_off[t] = off;
        off += stack_depth[t] * (uint32_t)kStackWidth[t] * 32u * (uint32_t)P;
    }
    *acc_off = off;
    off += 2u * 32u * (uint32_t)G;  // Kahan state of the item's programs
    *region_floats = align4r(off);
}

size_t reg_smem_bytes(uint32_t code_words, uint32_t const_floats, const uint32_t *stack_depth, int P, int G) {
    uint32_t so[N_STACKS], ao, rf, hf;
    reg_layout(code_words, const_floats, stack_depth, P, G, so, &ao, &rf, &hf);
    return ((size_t)hf + (size_t)rf * (kRegThreads / 32)) * 4u;
}

template <int PROF, int P, int OMIT>
static cudaError_t launch_reg_pp(const LaunchArgs &a, uint32_t grid, cudaStream_t st) {
    auto k = reg_eval_kernel<PROF, P, OMIT>;
    const size_t smem = ((size_t)a.block_hdr_floats + (size_t)a.region_floats * (kRegThreads / 32)) * 4u;
    static std::atomic<uint64_t> limit_raised{0};
    cudaError_t e = raise_smem_limit(k, limit_raised);
    if (e != cudaSuccess) return e;
    k<<<grid, kRegThreads, smem, st>>>(a);
    return cudaGetLastError();
}

// Instantiated points-per-thread values: {2, 4, 8} for the F, F+V3 and
// F+V2+M2 profiles, {2, 4} for the others.
int reg_max_p(int profile) { return profile == P_F || profile == P_FV3 || profile == P_FV2M2 ? 8 : 4; }

// Handler sets a profile has kernels without (the OMIT mask of run_program).
unsigned reg_omittable(int profile) {
    return profile == P_FV3 ? 3u : profile == P_F || profile == P_FV2M2 ? 1u : 0u;
}

template <int PROF, int OMIT>
static cudaError_t launch_reg_p3(const LaunchArgs &a, int P, uint32_t grid, cudaStream_t st) {
    return P >= 8 ? launch_reg_pp<PROF, 8, OMIT>(a, grid, st)
         : P >= 4 ? launch_reg_pp<PROF, 4, OMIT>(a, grid, st) : launch_reg_pp<PROF, 2, OMIT>(a, grid, st);
}

cudaError_t launch_reg(const LaunchArgs &a, int profile, int P, unsigned omit, uint32_t grid, cudaStream_t st) {
    switch (profile) {
        case P_F: return omit & 1u ? launch_reg_p3<P_F, 1>(a, P, grid, st) : launch_reg_p3<P_F, 0>(a, P, grid, st);
        case P_FV3:
            switch (omit & 3u) {
                case 3: return launch_reg_p3<P_FV3, 3>(a, P, grid, st);
                case 2: return launch_reg_p3<P_FV3, 2>(a, P, grid, st);
                case 1: return launch_reg_p3<P_FV3, 1>(a, P, grid, st);
                default: return launch_reg_p3<P_FV3, 0>(a, P, grid, st);
            }
        case P_FV2M2: return omit & 1u ? launch_reg_p3<P_FV2M2, 1>(a, P, grid, st)
                                       : launch_reg_p3<P_FV2M2, 0>(a, P, grid, st);
        case P_FV3M3: return P >= 4 ? launch_reg_pp<P_FV3M3, 4, 0>(a, grid, st)
                                    : launch_reg_pp<P_FV3M3, 2, 0>(a, grid, st);
        default: return P >= 4 ? launch_reg_pp<P_ALL, 4, 0>(a, grid, st) : launch_reg_pp<P_ALL, 2, 0>(a, grid, st);
    }
}

// Loads one instance ahead of its first real launch: an empty launch (run_if
// points at a zero word, so every thread returns at its first check) also
// sizes the context's local memory for the instance's spills.
template <int PROF, int P, int OMIT>
static cudaError_t preload_pp(const uint32_t *zero, cudaStream_t st) {
    auto k = reg_eval_kernel<PROF, P, OMIT>;
    static std::atomic<uint64_t> limit_raised{0};
    cudaError_t e = raise_smem_limit(k, limit_raised);
    if (e != cudaSuccess) return e;
    LaunchArgs none{};
    none.run_if = zero;
    k<<<1, kRegThreads, 0, st>>>(none);
    return cudaGetLastError();
}

template <int PROF, int OMIT>
static cudaError_t preload_p3(const uint32_t *zero, cudaStream_t st) {
    cudaError_t e;
    if ((e = preload_pp<PROF, 2, OMIT>(zero, st)) != cudaSuccess) return e;
    if ((e = preload_pp<PROF, 4, OMIT>(zero, st)) != cudaSuccess) return e;
    return preload_pp<PROF, 8, OMIT>(zero, st);
}

cudaError_t preload_reg(const uint32_t *zero, cudaStream_t st) {
    const cudaError_t r[] = {
        preload_p3<P_F, 0>(zero, st),     preload_p3<P_F, 1>(zero, st),
        preload_p3<P_FV3, 0>(zero, st),   preload_p3<P_FV3, 1>(zero, st),
        preload_p3<P_FV3, 2>(zero, st),   preload_p3<P_FV3, 3>(zero, st),
        preload_p3<P_FV2M2, 0>(zero, st), preload_p3<P_FV2M2, 1>(zero, st),
        preload_pp<P_FV3M3, 2, 0>(zero, st), preload_pp<P_FV3M3, 4, 0>(zero, st),
        preload_pp<P_ALL, 2, 0>(zero, st),   preload_pp<P_ALL, 4, 0>(zero, st)};
    for (cudaError_t e : r)
        if (e != cudaSuccess) return e;
    return cudaSuccess;
}

template <int PROF, int P, int OMIT>
static int occ(size_t smem) {
    // the occupancy query counts a block above 48 KB of dynamic shared memory
    // as unlaunchable until the kernel's limit has been raised
    auto k = reg_eval_kernel<PROF, P, OMIT>;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmemOptin) != cudaSuccess) return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, kRegThreads, smem) != cudaSuccess) return 0;
    return n;
}

template <int PROF, int OMIT>
static int occ3(int P, size_t smem) {
    return P >= 8 ? occ<PROF, 8, OMIT>(smem) : P >= 4 ? occ<PROF, 4, OMIT>(smem) : occ<PROF, 2, OMIT>(smem);
}

int reg_max_blocks_per_sm(int profile, int P, unsigned omit, size_t smem) {
    switch (profile) {
        case P_F: return omit & 1u ? occ3<P_F, 1>(P, smem) : occ3<P_F, 0>(P, smem);
        case P_FV3:
            switch (omit & 3u) {
                case 3: return occ3<P_FV3, 3>(P, smem);
                case 2: return occ3<P_FV3, 2>(P, smem);
                case 1: return occ3<P_FV3, 1>(P, smem);
                default: return occ3<P_FV3, 0>(P, smem);
            }
        case P_FV2M2: return omit & 1u ? occ3<P_FV2M2, 1>(P, smem) : occ3<P_FV2M2, 0>(P, smem);
        case P_FV3M3: return P >= 4 ? occ<P_FV3M3, 4, 0>(smem) : occ<P_FV3M3, 2, 0>(smem);
        default: return P >= 4 ? occ<P_ALL, 4, 0>(smem) : occ<P_ALL, 2, 0>(smem);
    }
}

}  // namespace rsr
