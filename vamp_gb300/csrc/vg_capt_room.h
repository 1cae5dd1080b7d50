// Room for the affordance lists of a tree built level by level on the GPU (vg_capt_gpu.cu): entries of
// each of its two list buffers.  Guessed before the build, which starts again with more where a
// level runs out, and tries with less where the memory cannot be had.
#pragma once

#include <algorithm>

namespace vg
{
    class ListRoom
    {
    public:
        // 160 entries a leaf: a tree for the Panda's spheres needs 104 (50,000 points), one for larger
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

        // The memory for this room cannot be had.  False where no smaller room can do.
        bool shrink()
        {
            if (needed_ ? entries_ <= needed_ : entries_ <= floor_)
            {
                return false;
            }
            entries_ = needed_ ? needed_ : std::max(entries_ / 4, floor_);
            return true;
        }

        // A level ran out of room and needs `entries`: four times that for the levels below.
        void grow(unsigned long long entries)
        {
            needed_ = entries;
            entries_ = 4 * entries;
        }

    private:
        unsigned long long floor_, entries_;
        unsigned long long needed_ = 0;  // by the last level that ran out
    };
}  // namespace vg
