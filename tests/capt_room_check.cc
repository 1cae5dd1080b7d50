// A build's attempts against a memory of `limit` entries, for levels that need what is given: prints
// 1 (built) or 0 (no memory), the attempts, and the room it was built with, per case.
#include "../vamp_gb300/csrc/vg_capt_room.h"

#include <cstdio>

int main()
{
    long long leaves;
    unsigned long long limit, a, b, c;
    while (std::scanf("%lld %llu %llu %llu %llu", &leaves, &limit, &a, &b, &c) == 5)
    {
        const unsigned long long needs[3] = {a, b, c};
        vg::ListRoom room(leaves);
        int built = -1, attempts = 0;
        while (built < 0 && attempts < 200)
        {
            ++attempts;
            if (2 * room.entries() > limit)
            {
                if (!room.shrink())
                    built = 0;
                continue;
            }
            built = 1;
            for (unsigned long long need : needs)
            {
                if (need > room.entries())
                {
                    room.grow(need);
                    built = -1;
                    break;
                }
            }
        }
        std::printf("%d %d %llu\n", built, attempts, room.entries());
    }
    return 0;
}
