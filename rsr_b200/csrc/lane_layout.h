// lane_layout.h -- which points of a tile a lane of the register kernels holds.
#pragma once
#include <stdint.h>

#include "uops.h"

namespace rsr {

// ------------------------------------------------ interleaved lane layout
// The register kernels give lane l of a warp the points of a 32*P-point
// tile in runs of at most four: P <= 4, points l*P .. l*P+P-1; P = 8, points
// 4l .. 4l+3 and 128+4l .. 128+4l+3.  Each 16-byte access of the warp then
// covers 512 contiguous bytes -- four L1 wavefronts for a global load, no
// bank conflict for shared memory -- where eight consecutive points a lane
// would take eight (two lanes 32 bytes apart share a 128-byte line or a bank).
// Per-lane values in shared memory use the same layout in blocks of 32*P
// floats: [P/4 runs][32 lanes][4] (P >= 4), [32 lanes][P] below.
template <int P>
constexpr int kLaneRun = P < 4 ? P : 4;

// Offset of value q of `lane` from the start of its tile (or block).
template <int P>
RSR_HD constexpr uint32_t lane_point(int lane, int q) {
    return (uint32_t)((q / kLaneRun<P>) * 32 * kLaneRun<P> + lane * kLaneRun<P> + q % kLaneRun<P>);
}

// The points of a lane that count, those below n_eval: bit q for value q.  In a
// tile that the data set's end cuts off bit P is set too, in all lanes, also in
// those whose points all count: "mask > (1 << P) - 1" then answers the same for
// the whole warp, so that a branch on it leaves no lane behind (the reverse
// sweep reads tensor memory with instructions that the whole warp has to issue
// together).
template <int P>
RSR_HD constexpr uint32_t counted_points(int lane, uint64_t tile, uint64_t n_eval) {
    if (tile + 32u * P <= n_eval) return (1u << P) - 1u;
    uint32_t mask = 1u << P;
    for (int q = 0; q < P; ++q) mask |= (tile + lane_point<P>(lane, q) < n_eval ? 1u : 0u) << q;
    return mask;
}

}  // namespace rsr
