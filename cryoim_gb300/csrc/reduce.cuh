// reduce.cuh — FP64 sums across a warp and a block in few FP64 operations: the SM's FP64 pipe
// takes a warp's add or conversion every 16 cycles (FP32: every quarter cycle), so sums of
// several values, or one sum that every thread repeats, can outweigh the FP32 work that they
// close.
#pragma once

#include <cuda_runtime.h>

namespace cryoim {

// N (a power of two up to 32) values of each lane summed over the warp: lanes exchange halves of
// the values until each has one, so N - 1 + log2(32 / N) adds instead of 5 N.  v[0] becomes the
// sum of value warp_sum_index<N>(lane), in the order of the butterfly.
template <int N>
__device__ __forceinline__ void warp_sums(double (&v)[N], int lane) {
    int o = 16;
#pragma unroll
    for (int n = N / 2; n >= 1; n >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const double send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (; o >= 1; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
}
template <int N>
__device__ __forceinline__ int warp_sum_index(int lane) {
    return lane / (32 / N);
}

// The same over a block of up to 32 warps: sh[N][32]; the sums are in sh[i][0] for warp 0 when it
// returns (the other warps may still be inside).
template <int N>
__device__ __forceinline__ void block_sums(double (&v)[N], double (*sh)[32]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    warp_sums<N>(v, lane);
    if (lane % (32 / N) == 0) sh[warp_sum_index<N>(lane)][warp] = v[0];
    __syncthreads();
    if (warp) return;
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = lane < nw ? sh[i][lane] : 0.0;
    __syncwarp();
    warp_sums<N>(v, lane);
    if (lane % (32 / N) == 0) sh[warp_sum_index<N>(lane)][0] = v[0];
    __syncwarp();
}

}  // namespace cryoim
