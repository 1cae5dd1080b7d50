// Bitonic compare-exchange steps of one block's tile, kept in registers.
//
// Thread t holds the PER consecutive elements PER t .. PER t + PER - 1 of the tile.  Strides below
// PER stay in the thread, strides up to 16 PER go through warp shuffles, and only the longer ones
// through shared memory (element e of thread t at e * threads + t: no bank conflicts either way).
// The steps and their directions are those of the plain network, so the order is too, ties and
// unordered keys included.  What bounded the shared-memory form was a barrier and two round trips
// per step: 2,048 64-bit keys 14.4 us, 11 levels of a 2,048-entry subtree 141 us.
#pragma once

#include <cstdint>

namespace vg
{
    __device__ __forceinline__ unsigned long long shuffle_xor(unsigned long long v, int lanes)
    {
        return __shfl_xor_sync(0xffffffffu, v, lanes);
    }

    // Steps of sizes k0 <= k <= k1 and strides below the tile's T elements (T a power of two, T <= PER *
    // blockDim.x; threads past T take part with any elements).  greater(a, b): a belongs after b;
    // up(i, k): element i's run of k elements ascends.  sm: PER * blockDim.x elements.  Every thread of
    // the block calls.
    template <int PER, typename E, typename Greater, typename Up>
    __device__ __forceinline__ void sort_steps(E (&v)[PER], E *sm, unsigned T, unsigned k0, unsigned k1, Greater greater, Up up)
    {
        const unsigned t = threadIdx.x, threads = blockDim.x;
        for (unsigned k = k0; k <= k1 && k; k <<= 1)
        {
            for (unsigned j = min(k, T) >> 1; j >= PER; j >>= 1)
            {
                const unsigned d = j / PER;  // the partner thread's distance
                E other[PER];
                if (d >= 32)
                {
                    __syncthreads();
#pragma unroll
                    for (int e = 0; e < PER; ++e)
                        sm[e * threads + t] = v[e];
                    __syncthreads();
#pragma unroll
                    for (int e = 0; e < PER; ++e)
                        other[e] = sm[e * threads + (t ^ d)];
                }
                else
                {
#pragma unroll
                    for (int e = 0; e < PER; ++e)
                        other[e] = shuffle_xor(v[e], static_cast<int>(d));
                }
                const bool lower = (t & d) == 0;
#pragma unroll
                for (int e = 0; e < PER; ++e)
                {
                    const bool rise = up(PER * t + e, k);
                    const bool swap = greater(lower ? v[e] : other[e], lower ? other[e] : v[e]) == rise;
                    v[e] = swap ? other[e] : v[e];
                }
            }
#pragma unroll
            for (unsigned j = PER / 2; j > 0; j >>= 1)
            {
                if (j < k && j < T)
                {
#pragma unroll
                    for (int e = 0; e < PER; ++e)
                    {
                        if ((e & j) == 0)
                        {
                            const bool swap = greater(v[e], v[e ^ j]) == up(PER * t + e, k);
                            const E a = v[e], b = v[e ^ j];
                            v[e] = swap ? b : a;
                            v[e ^ j] = swap ? a : b;
                        }
                    }
                }
            }
        }
    }
}  // namespace vg
