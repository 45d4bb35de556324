// The box of points [n,3] by one cluster of eight blocks, which can wait for one
// another without a word in memory that somebody would have to clear first.
#pragma once

#include <cooperative_groups.h>

#include "mo_common.cuh"

namespace mo {

// The thread count is a multiple of three, so a thread keeps one coordinate and
// the reads are consecutive; a warp reduces each coordinate by itself and its
// leaders put it into the first block's shared memory.  Eight SMs read ~0.25
// TB/s: past BBOX_CLUSTER_MAX points the whole chip and more launches are faster (box
// and parameters, us, inputs not in L2: 400k 23 against 30, 600k 31 against 32, 800k 39
// against 32).
constexpr int BBOX_BLOCKS = 8, BBOX_THREADS = 960, BBOX_UNROLL = 16;
constexpr int64_t BBOX_CLUSTER_MAX = 600000;

// Called by all threads of the cluster; box: six ints of shared memory.  True in
// one thread, where box then holds the extremes (ordered ints: min x, y, z, max
// x, y, z) of the coordinates that are not NaN, or with FINITE that are finite.
template <bool FINITE>
__device__ bool bbox_cluster(const float* __restrict__ V, int64_t n, int* box) {
    static_assert(BBOX_THREADS % 96 == 0, "whole warps, and a coordinate a thread");
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int tid = (int)threadIdx.x, c = tid % 3;
    if (tid < 6) box[tid] = tid < 3 ? INT_MAX : INT_MIN;
    cluster.sync();
    int lo = INT_MAX, hi = INT_MIN;
    constexpr int64_t STRIDE = (int64_t)BBOX_BLOCKS * BBOX_THREADS;
    const int64_t total = 3 * n;
    for (int64_t i = (int64_t)blockIdx.x * BBOX_THREADS + tid; i < total; i += STRIDE * BBOX_UNROLL) {
        float f[BBOX_UNROLL];
#pragma unroll
        for (int k = 0; k < BBOX_UNROLL; ++k)
            f[k] = i + k * STRIDE < total ? __ldg(V + i + k * STRIDE) : __int_as_float(0x7fc00000);
#pragma unroll
        for (int k = 0; k < BBOX_UNROLL; ++k) {
            if (FINITE ? !isfinite(f[k]) : f[k] != f[k]) continue;  // NaN never wins a comparison in the reference
            const int o = float_to_ordered(f[k]);
            lo = min(lo, o);
            hi = max(hi, o);
        }
    }
    int* first = cluster.map_shared_rank(box, 0);
    for (int k = 0; k < 3; ++k) {  // lanes of coordinate k
        const unsigned lanes = __ballot_sync(0xffffffffu, c == k);
        if (c != k) continue;
        lo = __reduce_min_sync(lanes, lo);
        hi = __reduce_max_sync(lanes, hi);
        if ((tid & 31) == __ffs(lanes) - 1) {
            atomicMin(&first[k], lo);
            atomicMax(&first[3 + k], hi);
        }
    }
    cluster.sync();
    return blockIdx.x == 0 && tid == 0;
}

}  // namespace mo
