// A tree's build against a memory of `limit` entries for its two list buffers: per case, the number of
// leaves, the limit, the number of levels and what each needs; prints 1 (built) or 0 (no memory),
// the allocations tried, and the first guess.
#include "../vamp_gb300/csrc/vg_capt_room.h"

#include <cstdio>
#include <vector>

int main()
{
    long long leaves;
    unsigned long long limit;
    int levels;
    while (std::scanf("%lld %llu %d", &leaves, &limit, &levels) == 3)
    {
        std::vector<unsigned long long> needs(levels);
        for (auto &n : needs)
        {
            if (std::scanf("%llu", &n) != 1)
                return 1;
        }
        vg::ListRoom room(leaves);
        const unsigned long long guess = room.entries();
        int built = 1, tried = 1;
        while (built && 2 * room.entries() > limit)
        {
            built = room.shrink() ? 1 : 0;
            ++tried;
        }
        unsigned long long cap[2] = {room.entries(), room.entries()};
        for (int d = 0; built && d < levels; ++d)
        {
            const int c = 1 - (d & 1);
            if (needs[d] <= cap[c])
                continue;
            cap[c] = needs[d];
            ++tried;
            if (cap[c] + cap[1 - c] > limit)
                built = 0;
        }
        std::printf("%d %d %llu\n", built, tried, guess);
    }
    return 0;
}
