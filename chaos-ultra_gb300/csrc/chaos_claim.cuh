// chaos_claim.cuh -- work claims of the persistent kernels, one global atomic
// per block-sized piece.
//
// One counter for a whole frame limits how small a warp's claim may be: claims
// of 4 tiles instead of 16 took a 7680x4320 reuse frame (260,000 claims) from
// 210 to 527 us.  So a block claims a piece for all its warps and they share it
// out by an atomic in shared memory.  The piece in hand is one 64-bit word
// (end << 32 | next), so a warp takes its part by adding to it, and a warp that
// finds it used up claims the next piece from the counter, keeps what it asked
// for and leaves the rest in the word.  One warp of the block does that at a
// time: another that finds the piece used up meanwhile claims just what it asked
// for.  Nothing waits.
#pragma once

#include <cstdint>

namespace chaos {

// A launch's work counter (`next`; zero when the launch starts) and its slot's
// other words: the number of blocks that have ended (zero between launches; null
// where the caller or a memset before the launch zeroes the counter) and the
// host's word that says the slot is taken (chaos_slots.h; null where the host
// gives the slot back).
struct WorkCounter {
    uint32_t *next, *done, *busy;
};

// The end of a persistent kernel: the launch's last warp leaves the work counter
// at zero for the launch that takes it next (a memset before every launch cost
// a small frame as much as its kernel) and gives the slot back.  Each warp's
// lane 0 calls it after the warp's last claim.  retired: shared, zero from before
// the block's first barrier.  No claim is still on its way when the words go back
// to zero: a warp gets here by the result of its last one.  (The host's word
// follows them at system scope; 20.2 -> 20.5 us for a 256x144 frame.  A fence in
// every block waited for the block's pixels: 166 -> 168 us at 1920x1080.)
__device__ __forceinline__ void leave_counter(const WorkCounter &w, uint32_t *retired)
{
    if (!w.done) return;
    if (atomicAdd(retired, 1u) + 1u != (blockDim.x >> 5)) return;
    if (atomicAdd(w.done, 1u) + 1u != gridDim.x) return;
    *w.next = 0u;
    *w.done = 0u;
    if (!w.busy) return;
    __threadfence_system();
    *(volatile uint32_t *)w.busy = 0u;
}

// Pieces of `size` items; the first of every block goes out without a claim
// (block b has [b size, (b + 1) size)).
struct ClaimPlan {
    uint32_t n, size;
};

struct ClaimShared {
    unsigned long long piece;  // end << 32 | next
    uint32_t busy;             // a warp is claiming the next piece
};

class Claims {
public:
    // All threads of the block; the caller synchronises it before the first take.
    __device__ __forceinline__ Claims(ClaimShared &shared, uint32_t *counter, const ClaimPlan &plan)
        : shared_(shared), counter_(counter), plan_(plan)
    {
        if (threadIdx.x == 0) {
            const uint32_t at = min(blockIdx.x * plan.size, plan.n);
            shared.piece = pack(at, min(at + plan.size, plan.n));
            shared.busy = 0;
        }
    }

    // Takes up to `want` consecutive items for the warp (uniform; all lanes
    // call it together): the first one's index, and how many in `got`, which is 0
    // only when no items are left.
    __device__ __forceinline__ uint32_t take(uint32_t want, uint32_t &got)
    {
        uint32_t at = 0, n = 0;
        if ((threadIdx.x & 31u) == 0u) take_one(want, at, n);
        got = __shfl_sync(0xffffffffu, n, 0);
        return __shfl_sync(0xffffffffu, at, 0);
    }

private:
    static __device__ __forceinline__ unsigned long long pack(uint32_t next, uint32_t end)
    {
        return ((unsigned long long)end << 32) | next;
    }

    __device__ __forceinline__ bool take_piece(uint32_t want, uint32_t &at, uint32_t &n)
    {
        const unsigned long long w = atomicAdd(&shared_.piece, (unsigned long long)want);
        const uint32_t end = (uint32_t)(w >> 32);
        at = (uint32_t)w;
        n = at < end ? min(want, end - at) : 0u;
        return n != 0u;
    }

    __device__ __forceinline__ uint32_t claim(uint32_t size)
    {
        return gridDim.x * plan_.size + atomicAdd(counter_, size);
    }

    // lane 0
    __device__ __forceinline__ void take_one(uint32_t want, uint32_t &at, uint32_t &n)
    {
        if (take_piece(want, at, n)) return;
        if (atomicExch(&shared_.busy, 1u) != 0u) {  // another warp is at the counter
            at = claim(want);
            n = at < plan_.n ? min(want, plan_.n - at) : 0u;
            return;
        }
        // a piece may have come since (only this warp puts one there now)
        if (!take_piece(want, at, n)) {
            at = claim(plan_.size);
            const uint32_t end = at < plan_.n ? min(plan_.size, plan_.n - at) + at : at;
            n = min(want, end - at);
            atomicExch(&shared_.piece, pack(at + n, end));
        }
        __threadfence_block();
        atomicExch(&shared_.busy, 0u);
    }

    ClaimShared &shared_;
    uint32_t *counter_;
    ClaimPlan plan_;
};

}  // namespace chaos
