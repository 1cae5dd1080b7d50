// Device memory that comes and goes with calls and environments (the pointcloud filter's, tree
// builds' and debug reports' scratch, host calls' buffers, trees, environment images): a private
// stream-ordered pool per device, which keeps up to kPoolKeep bytes between calls (an allocation of
// tens of megabytes from the driver takes longer than the work in it) and returns the rest to the
// driver.  Safe with several threads and streams: allocations and releases are ordered on their
// streams, and the pool orders reuse across streams.
//
// Blocks of more than kPoolKeep, which the pool would return at every wait, come from the driver
// directly: taking and returning a gigabyte costs 0.5 ms there and 1.8 through the pool.  Their
// release waits for the stream.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <mutex>
#include <unordered_set>

namespace vg
{
    constexpr uint64_t kPoolKeep = uint64_t{256} << 20;

    // Blocks in use that did not come from the pool.
    struct DirectBlocks
    {
        std::mutex mu;
        std::unordered_set<void *> set;
    };

    inline DirectBlocks &direct_blocks()
    {
        static DirectBlocks *const blocks = new DirectBlocks;  // outlives what is destroyed at exit
        return *blocks;
    }

    // `bytes` of device memory for work on stream s.
    inline cudaError_t pool_take(void **p, size_t bytes, cudaStream_t s)
    {
        constexpr int kDevices = 64;
        static std::mutex mu;
        static cudaMemPool_t pools[kDevices] = {};
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess)
            return e;
        if (dev >= kDevices || bytes > kPoolKeep)
        {
            e = cudaMalloc(p, bytes);
            if (e != cudaSuccess)
                return e;
            try
            {
                DirectBlocks &direct = direct_blocks();
                std::lock_guard<std::mutex> lock(direct.mu);
                direct.set.insert(*p);
            }
            catch (...)
            {
                cudaFree(*p);
                *p = nullptr;
                return cudaErrorMemoryAllocation;
            }
            return cudaSuccess;
        }
        cudaMemPool_t pool = nullptr;
        {
            std::lock_guard<std::mutex> lock(mu);
            if (!pools[dev])
            {
                cudaMemPoolProps props{};
                props.allocType = cudaMemAllocationTypePinned;
                props.location.type = cudaMemLocationTypeDevice;
                props.location.id = dev;
                e = cudaMemPoolCreate(&pools[dev], &props);
                uint64_t keep = kPoolKeep;
                if (e == cudaSuccess)
                    e = cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold, &keep);
                if (e != cudaSuccess)
                    return e;
            }
            pool = pools[dev];
        }
        return cudaMallocFromPoolAsync(p, bytes, pool, s);
    }

    // Releases memory from pool_take once the work already on s is done.
    inline void pool_give(void *p, cudaStream_t s)
    {
        if (!p)
            return;
        bool direct = false;
        {
            DirectBlocks &blocks = direct_blocks();
            std::lock_guard<std::mutex> lock(blocks.mu);
            direct = blocks.set.erase(p) > 0;
        }
        if (direct)
        {
            cudaStreamSynchronize(s);
            cudaFree(p);
        }
        else if (cudaFreeAsync(p, s) != cudaSuccess)
        {
            cudaGetLastError();
            cudaFree(p);
        }
    }
}  // namespace vg
