// Deterministic grid reductions: every block writes its partial sums, the
// last block to finish adds the partials in block order (fixed grid => fixed
// summation order => bit-reproducible results).
#pragma once
#include "b2s_internal.cuh"

namespace b2s
{
constexpr int RED_BLOCK = 256;

// block sum of NV doubles per thread; valid in thread 0
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double (*smem)[RED_BLOCK / 32])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for(int k = 0; k < NV; ++k)
    {
#pragma unroll
        for(int o = 16; o > 0; o >>= 1)
            v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    }
    if(lane == 0)
    {
#pragma unroll
        for(int k = 0; k < NV; ++k)
            smem[k][warp] = v[k];
    }
    __syncthreads();
    if(warp == 0)
    {
#pragma unroll
        for(int k = 0; k < NV; ++k)
        {
            double t = (lane < (int)(blockDim.x >> 5)) ? smem[k][lane] : 0.0;
#pragma unroll
            for(int o = 16; o > 0; o >>= 1)
                t += __shfl_xor_sync(0xffffffffu, t, o);
            v[k] = t;
        }
    }
}

// Publish this block's NV partial sums; returns true in thread 0 of the last
// block, which then finds the totals in `total`.
template <int NV>
__device__ __forceinline__ bool grid_sum(double (&v)[NV], double* partials, unsigned int* counter,
                                         double (&total)[NV])
{
    __shared__ double smem[NV][RED_BLOCK / 32];
    __shared__ bool   is_last;
    block_sum<NV>(v, smem);
    if(threadIdx.x == 0)
    {
#pragma unroll
        for(int k = 0; k < NV; ++k)
            partials[(size_t)k * gridDim.x + blockIdx.x] = v[k];
        __threadfence();
        unsigned int prev = atomicAdd(counter, 1u);
        is_last           = (prev == gridDim.x - 1);
    }
    __syncthreads();
    if(!is_last)
        return false;
    // last block: NV values side by side, G warps each (a fixed shape for a
    // given grid). Every lane adds a strided subset in order, then a fixed
    // tree; the loads go out 8 at a time, independent of one another. With one
    // warp per value the 1184 partials of a full grid took five dependent
    // rounds of loads at the end of every kernel with a sum.
    __threadfence();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int G = nw > NV ? nw / NV : 1;
    __shared__ double res[NV][RED_BLOCK / 32];
    for(int job = warp; job < NV * G; job += nw)
    {
        const int              k = job / G, part = job - k * G;
        const volatile double* pk   = (const volatile double*)partials + (size_t)k * gridDim.x;
        const unsigned int     step = 32u * G;
        double                 acc  = 0.0;
        for(unsigned int b = 32 * part + lane; b < gridDim.x; b += step * 8)
        {
            double t[8];
#pragma unroll
            for(int j = 0; j < 8; ++j)
                t[j] = b + step * j < gridDim.x ? pk[b + step * j] : 0.0;
#pragma unroll
            for(int j = 0; j < 8; ++j)
                if(b + step * j < gridDim.x)
                    acc += t[j];
        }
#pragma unroll
        for(int o = 16; o > 0; o >>= 1)
            acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if(lane == 0)
            res[k][part] = acc;
    }
    __syncthreads();
    if(threadIdx.x != 0)
        return false;
#pragma unroll
    for(int k = 0; k < NV; ++k)
    {
        double t = res[k][0];
        for(int g = 1; g < G; ++g)
            t += res[k][g];
        total[k] = t;
    }
    *counter = 0u;  // ready for the next launch
    return true;
}
}  // namespace b2s
