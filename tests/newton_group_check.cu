// Host check of chaos::newton_group (csrc/chaos_newton.cuh): the step loop of newton_compute, without its steps, from a
// few steps before `end`, ends at `end` for every end near 2^32 and near 0.  Prints "ok" or the failure.
#include <cstdio>

#include "chaos_newton.cuh"

int main()
{
    for (uint32_t k = 0; k < 80; k++) {
        const uint32_t end = k < 40 ? 0xffffffffu - k : k - 40;
        for (uint32_t back = 0; back <= 40 && back <= end; back++) {
            uint32_t i = end - back, rounds = 0;
            for (; chaos::newton_group(i, end); i += 4u)
                if (++rounds > 10u) return std::printf("end %u from %u: no end\n", end, end - back), 1;
            if (i > end || end - i > 4u || (i == end && back != 0)) return std::printf("end %u from %u: %u\n", end, end - back, i), 1;
        }
    }
    std::puts("ok");
    return 0;
}
