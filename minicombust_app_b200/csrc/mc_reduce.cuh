// Deterministic grid reductions without atomics on data: each block writes
// its partial sums, the last block to arrive (one atomicAdd on a counter, no
// waiting) reduces the partials in a fixed order and publishes the result.
// Block size is fixed at MCB_THREADS.
#pragma once

#include <cuda_runtime.h>

#define MCB_THREADS 256

namespace mcb {

// Sum, or maximum, of one value per thread across the block of MCB_THREADS;
// result in every thread.  By shuffles: two barriers, where a tree in shared
// memory takes ten; every reduction kernel runs it twice in a row (the block's
// partial, then the last block's total), which bounds the small ones (a
// refined pass on 305,000 cells 4.59 -> 4.53 ms).
template <int K, bool MAX = false>
__device__ inline void block_reduce(double (&v)[K], double (*sh)[MCB_THREADS])
{
    constexpr int WARPS = MCB_THREADS / 32;
    static_assert((WARPS & (WARPS - 1)) == 0, "the second stage halves the warps");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto join = [](double a, double b) { return MAX ? fmax(a, b) : a + b; };
    __syncthreads();  // sh may still be read from a previous reduction
#pragma unroll
    for (int k = 0; k < K; k++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] = join(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
        if (lane == 0) sh[k][warp] = v[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; k++) {
        v[k] = sh[k][lane & (WARPS - 1)];
#pragma unroll
        for (int o = WARPS / 2; o > 0; o >>= 1) v[k] = join(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
    }
}

// Reduce the threads' values across the block, publish the block's K
// partials and report whether this block is the last to arrive.
// partials: [gridDim.x][K]; counter must be zero before the launch and is
// reset by the last block.
template <int K, bool MAX = false>
__device__ inline bool publish_partials(const double (&v)[K], double *partials, unsigned int *counter,
                                        double (*sh)[MCB_THREADS])
{
    __shared__ bool am_last;
    double b[K];
#pragma unroll
    for (int k = 0; k < K; k++) b[k] = v[k];
    block_reduce<K, MAX>(b, sh);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < K; k++) partials[(size_t)blockIdx.x * K + k] = b[k];
        __threadfence();
        const unsigned int prev = atomicAdd(counter, 1u);
        am_last = (prev == gridDim.x - 1);
    }
    __syncthreads();
    return am_last;
}

// In the last block: reduce the partials of all blocks (fixed order: thread
// t takes blocks t, t+256, ..., then a fixed tree).  Result in every thread.
template <int K, bool MAX = false>
__device__ inline void reduce_partials(double (&out)[K], const double *partials, unsigned int *counter,
                                       double (*sh)[MCB_THREADS])
{
    double acc[K];
#pragma unroll
    for (int k = 0; k < K; k++) acc[k] = MAX ? -1.0e308 : 0.0;
    for (unsigned int b = threadIdx.x; b < gridDim.x; b += MCB_THREADS) {
#pragma unroll
        for (int k = 0; k < K; k++) {
            const double p = __ldcg(partials + (size_t)b * K + k);
            acc[k] = MAX ? fmax(acc[k], p) : acc[k] + p;
        }
    }
    block_reduce<K, MAX>(acc, sh);
#pragma unroll
    for (int k = 0; k < K; k++) out[k] = acc[k];
    if (threadIdx.x == 0) *counter = 0u;
}

__device__ __forceinline__ double warp_sum_all(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums of K values over a warp.  The first step of a pair is shared: half the
// warp keeps one value and sends the other, so two values take five exchanges
// each way and not ten.  Result k is valid in lane 0 (k even) or 16 (k odd).
template <int K>
__device__ __forceinline__ void warp_sums(double (&v)[K], int lane)
{
#pragma unroll
    for (int k = 0; k + 1 < K; k += 2) {
        const bool hi = lane & 16;
        const double keep = hi ? v[k + 1] : v[k], send = hi ? v[k] : v[k + 1];
        double t = keep + __shfl_xor_sync(0xffffffffu, send, 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        v[k] = v[k + 1] = t;
    }
    if (K & 1) v[K - 1] = warp_sum_all(v[K - 1]);
}

// Block sums of K values by warp shuffles (any block size that is a multiple
// of 32): two barriers whatever K is.  sw: [K][32] shared; result in every
// lane of warp 0.
template <int K>
__device__ __forceinline__ void block_sums(double (&v)[K], double (*sw)[32])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    __syncthreads();  // sw may still be read from a previous reduction
#pragma unroll
    for (int k = 0; k < K; k++) {
        v[k] = warp_sum_all(v[k]);
        if (lane == 0) sw[k][warp] = v[k];
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int k = 0; k < K; k++) v[k] = warp_sum_all(lane < nw ? sw[k][lane] : 0.0);
    }
}

// publish_partials / reduce_partials with shuffle sums.
template <int K>
__device__ __forceinline__ bool publish_sums(const double (&v)[K], double *partials, unsigned int *counter,
                                             double (*sw)[32], unsigned int block = blockIdx.x,
                                             unsigned int blocks = gridDim.x)
{
    __shared__ bool am_last;
    double b[K];
#pragma unroll
    for (int k = 0; k < K; k++) b[k] = v[k];
    block_sums<K>(b, sw);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < K; k++) partials[(size_t)block * K + k] = b[k];
        __threadfence();
        am_last = atomicAdd(counter, 1u) == blocks - 1;
    }
    __syncthreads();
    return am_last;
}

// In the last block: the partials of all blocks in a fixed order (thread t
// takes blocks t, t + blockDim, ...).  Result in thread 0.
template <int K>
__device__ __forceinline__ void reduce_sums(double (&out)[K], const double *partials, unsigned int *counter,
                                            double (*sw)[32], unsigned int blocks = gridDim.x)
{
#pragma unroll
    for (int k = 0; k < K; k++) out[k] = 0.0;
    for (unsigned int b = threadIdx.x; b < blocks; b += blockDim.x)
#pragma unroll
        for (int k = 0; k < K; k++) out[k] += __ldcg(partials + (size_t)b * K + k);
    block_sums<K>(out, sw);
    if (threadIdx.x == 0) *counter = 0u;
}

} // namespace mcb
