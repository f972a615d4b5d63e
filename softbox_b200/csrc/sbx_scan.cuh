// sbx_scan.cuh — block-wide scans of the counting sorts and of the wide step.
#pragma once
#include "sbx_internal.cuh"

namespace {

// block-wide exclusive scan of one int per thread; returns the exclusive prefix, *total = sum
template <int NT>
__device__ __forceinline__ int block_exclusive_scan(int v, int* total) {
    __shared__ int warp_sums[NT / 32];
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = (lane < NT / 32) ? warp_sums[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < NT / 32) warp_sums[lane] = w;
    }
    __syncthreads();
    int warp_prefix = warp > 0 ? warp_sums[warp - 1] : 0;
    *total = warp_sums[NT / 32 - 1];
    __syncthreads();
    return warp_prefix + x - v;
}

// a scan tile: 256 threads, 16 rows each
constexpr int SCAN_TILE_ROWS = 8 * SCAN_CHUNK;
constexpr int TILE_PER_THREAD = SCAN_TILE_ROWS / 256;

__device__ __forceinline__ int tile_slot(int r) { return r + (r >> 5); }     // padded: no bank conflicts

}  // namespace
