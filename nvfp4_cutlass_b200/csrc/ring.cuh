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

}  // namespace nvfp4::gemm
