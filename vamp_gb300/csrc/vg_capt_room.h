// Room for the affordance lists of a tree built level by level on the GPU (vg_capt_gpu.cu), in entries
// of each of its two list buffers: a guess before the build.  A level that runs out gets a buffer of what
// it needs and is done again (twice that, for the levels below, took as long: the waits it saves are
// short against the mapping of the memory).
#pragma once

#include <algorithm>

namespace vg
{
    class ListRoom
    {
    public:
        // 160 entries a leaf: a tree for the Panda's spheres needs 89 (50,000 points), one for larger
        // spheres more.  `leaves` is a power of two.
        explicit ListRoom(long long leaves)
          : floor_(2ull * static_cast<unsigned long long>(leaves)),
            entries_(std::min(std::max(80ull * floor_, 1ull << 18), std::max(1ull << 28, floor_)))
        {
        }

        unsigned long long entries() const
        {
            return entries_;
        }

        // The memory for the guess cannot be had.  False where it has come down to two entries a leaf.
        bool shrink()
        {
            if (entries_ <= floor_)
            {
                return false;
            }
            entries_ = std::max(entries_ / 4, floor_);
            return true;
        }

    private:
        unsigned long long floor_, entries_;
    };
}  // namespace vg
