// chaos_slots.h -- which work-counter slot a launch may have.
//
// A slot's words are carried from one launch to the next (the kernels leave them
// at zero, see leave_counter), so a slot goes out again only after its last
// launch has ended.  The device says so itself: each slot has a word in mapped
// host memory, set here when the slot goes out and cleared by the launch's last
// warp, so no event or query is needed, and a stream capture elsewhere is not
// disturbed.  Going by the order of the launches instead would hand the slot of
// a frame of seconds to another stream's preview after 4096 previews (80 ms).
// A launch that the caller's own call waits for is given back here instead: the
// write to the host is the end of such a launch (200x110 pixels: 18.1 us with it,
// 17.2 without).  A launch that never ran keeps its slot.
#pragma once

#include <atomic>
#include <cstdint>

namespace chaos {

class SlotRing {
public:
    static constexpr uint32_t NONE = 0xffffffffu;

    // busy: one word a slot, all zero
    void init(uint32_t *busy, uint32_t slots)
    {
        busy_ = busy;
        slots_ = slots;
    }

    // A slot that no launch holds, or NONE.  Any number of threads.
    uint32_t take()
    {
        const uint32_t at = next_.fetch_add(1, std::memory_order_relaxed);
        for (uint32_t k = 0; k < slots_; k++) {
            const uint32_t slot = (at + k) % slots_;
            uint32_t free = 0;
            // (acquire: the launch that held it left the slot's words at zero before this one)
            if (__atomic_load_n(busy_ + slot, __ATOMIC_RELAXED) == 0 &&
                __atomic_compare_exchange_n(busy_ + slot, &free, 1u, false, __ATOMIC_ACQUIRE, __ATOMIC_RELAXED))
                return slot;
        }
        return NONE;
    }

    // A slot whose launch has been waited for.
    void give(uint32_t slot) { __atomic_store_n(busy_ + slot, 0u, __ATOMIC_RELEASE); }

private:
    uint32_t *busy_ = nullptr;
    uint32_t slots_ = 0;
    std::atomic<uint32_t> next_{0};
};

}  // namespace chaos
