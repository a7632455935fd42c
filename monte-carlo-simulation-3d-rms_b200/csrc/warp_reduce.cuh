// warp_reduce.cuh -- cross-walker FP64 sums inside one warp.
//
// The reference adds every walker's record into the same global addresses
// with an FP64 compare-and-swap loop (hpc_code/lib/main.cu:40-56, 344-378):
// 23+Nbvec contended atomics per walker per record.  Here a warp first sums its
// walkers: a final sum by register shuffles in a fixed order, records and signals
// by lanes that each add up a column, b-value or gradient over the walkers
// (signal_lanes), and one lane per value passes the warp's sum on.
#pragma once
#include <cuda_runtime.h>

namespace rms {

constexpr unsigned kFullMask = 0xffffffffu;

// Sum over the warp; every lane receives the total (butterfly, fixed order).
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(kFullMask, v, off);
    return v;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(kFullMask, v, off);
    return v;
}

// The lanes of a warp over `items` (at most 32: b-values, gradients) and a
// tile's nw walkers: lane -> (item, share of the walkers), with as many shares
// as the items leave lanes for -- twelve b-values over 32 walkers are two shares
// of 16, not 20 idle lanes.
struct SignalLanes {
    int item, share, shares, per;   // per: lanes of a share, a power of two
};
__device__ __forceinline__ SignalLanes signal_lanes(int lane, int items, int nw) {
    int per = 32, shares = 1;
    while (per / 2 >= items && 2 * shares <= nw) {
        per >>= 1;
        shares <<= 1;
    }
    return SignalLanes{lane & (per - 1), lane / per, shares, per};
}
// Sum over an item's shares (every lane of the warp calls it).
__device__ __forceinline__ double share_sum(double s, const SignalLanes& l) {
    for (int off = l.per; off < 32; off <<= 1) s += __shfl_xor_sync(kFullMask, s, off);
    return s;
}

}  // namespace rms
