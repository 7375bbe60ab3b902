// Host check of chaos::SlotRing (csrc/chaos_slots.h) with the device's part, the
// clearing of a slot's word, played here.  Prints "ok" and exits 0, or the failure.
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>

#include "chaos_slots.h"

using chaos::SlotRing;

#define CHECK(c)                                              \
    do {                                                      \
        if (!(c)) {                                           \
            std::printf("line %d: %s\n", __LINE__, #c);       \
            std::exit(1);                                     \
        }                                                     \
    } while (0)

int main()
{
    {  // a launch that runs on while the ring comes round: its slot stays its own
        std::vector<uint32_t> busy(64, 0);
        SlotRing ring;
        ring.init(busy.data(), 64);
        const uint32_t held = ring.take();
        for (int k = 0; k < 1000; k++) {
            const uint32_t s = ring.take();
            CHECK(s < 64 && s != held && busy[s] == 1);
            busy[s] = 0;
        }
        busy[held] = 0;
        bool again = false;
        for (int k = 0; k < 64; k++) {
            const uint32_t s = ring.take();
            again = again || s == held;
            busy[s] = 0;
        }
        CHECK(again);
    }
    {  // every slot taken: none; one given back: that one
        std::vector<uint32_t> busy(7, 0);
        SlotRing ring;
        ring.init(busy.data(), 7);
        uint32_t seen = 0;
        for (int k = 0; k < 7; k++) seen |= 1u << ring.take();
        CHECK(seen == 127);
        CHECK(ring.take() == SlotRing::NONE);
        busy[3] = 0;
        CHECK(ring.take() == 3);
        CHECK(ring.take() == SlotRing::NONE);
    }
    {  // threads: no slot has two holders
        std::vector<uint32_t> busy(16, 0);
        std::vector<std::atomic<int>> holders(16);
        SlotRing ring;
        ring.init(busy.data(), 16);
        std::atomic<int> wrong{0};
        std::vector<std::thread> pool;
        for (int t = 0; t < 8; t++)
            pool.emplace_back([&] {
                for (int k = 0; k < 20000; k++) {
                    const uint32_t s = ring.take();
                    if (s == SlotRing::NONE) continue;
                    if (holders[s].fetch_add(1) != 0) wrong++;
                    holders[s].fetch_sub(1);
                    __atomic_store_n(&busy[s], 0u, __ATOMIC_RELEASE);
                }
            });
        for (auto &t : pool) t.join();
        CHECK(wrong == 0);
    }
    std::puts("ok");
    return 0;
}
