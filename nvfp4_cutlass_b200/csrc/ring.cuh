// Cursor of a shared-memory ring and the producer's last walk around it.  Plain C++ apart from the qualifiers, so that the
// order of waits can be checked without a GPU.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define NVFP4_RING_FN __host__ __device__ __forceinline__
#else
#define NVFP4_RING_FN inline
#endif

namespace nvfp4::gemm {

// Cursor of a ring of `kDepth` slots; the phase bit flips on every wrap.
struct Ring {
    uint32_t slot = 0, phase = 0;
    template <uint32_t kDepth>
    NVFP4_RING_FN void advance()
    {
        if (++slot == kDepth) { slot = 0; phase ^= 1; }
    }
};

// The producer's waits after its last load.  Commits of the tensor core free the ring positions (kGroup of them at a time);
// the last ones find nobody who waits for them, and a block that left before they had arrived would be signalled when
// its shared memory, and the barriers in it, belong to another block already.  `next` is the position that the producer
// would fill next; wait(group, parity) -> bool waits for a group's barrier as the producer would before refilling it.  A
// group that has been filled in part only is never committed and not waited for.  Returns false when a wait gave up.
template <uint32_t kDepth, uint32_t kGroup = 1, typename Wait>
NVFP4_RING_FN bool drain_ring(Ring next, Wait&& wait)
{
    uint32_t groups = kDepth / kGroup;
    if (next.slot % kGroup != 0) --groups;
    while (next.slot % kGroup != 0) next.advance<kDepth>();
    for (uint32_t i = 0; i < groups; ++i) {
        if (!wait(next.slot / kGroup, next.phase ^ 1u)) return false;
        for (uint32_t j = 0; j < kGroup; ++j) next.advance<kDepth>();
    }
    return true;
}

// The waits of one of `kGroups` groups that take the blocks of a ring in turn, ahead of block `it`.  A barrier's parity tells
// a use from the one before it, no more: whoever waits for use u has to know that use u - 1 is over, or the parity of
// u - 2 passes for it.  A group that takes every block knows, having waited for u - 1 itself; one that takes every third has
// not, and a load that arrived later than its successors was enough to let it through early.  So it first waits
// for the end of the slot's last use, done(slot, parity), a barrier that its own work moves on and that therefore cannot be
// ahead; then for full(slot, parity).  Returns false when a wait gave up.
template <uint32_t kDepth, uint32_t kGroups, typename Done, typename Full>
NVFP4_RING_FN bool wait_turn(uint32_t it, Done&& done, Full&& full)
{
    const uint32_t slot = it % kDepth, phase = (it / kDepth) & 1u;
    if (kGroups > 1 && it >= kDepth && !done(slot, phase ^ 1u)) return false;
    return full(slot, phase);
}

}  // namespace nvfp4::gemm
