// The order of waits and copies of a thread that feeds a ring of shared-memory
// stages by asynchronous copies, apart from the instructions themselves, so
// that the same code runs on the host.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define HG_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define HG_HOST_DEVICE inline
#endif

namespace hg {

// Copies `tiles` tiles through STAGES stages, tile k into stage k % STAGES once
// its readers are done with the tile before.  wait_empty(stage, parity) and
// wait_full(stage, parity) wait for a phase of the stage's barriers and return
// false when it did not complete in time; copy(stage, tile) starts a copy.
// Whatever a wait returned, every copy that was started has been waited for on
// return: a block that ended earlier would leave its shared memory to another
// block with the copy still under way.  True when nothing timed out.
template <uint32_t STAGES, class WaitEmpty, class Copy, class WaitFull>
HG_HOST_DEVICE bool feed_ring(uint32_t tiles, WaitEmpty wait_empty, Copy copy, WaitFull wait_full) {
    uint32_t started = 0;
    bool ok = true;
    for (; started < tiles; ++started) {
        const uint32_t s = started % STAGES, round = started / STAGES;
        if (round > 0 && !wait_empty(s, (round - 1u) & 1u)) {
            ok = false;
            break;
        }
        copy(s, started);
    }
    // a stage's earlier copies landed before its readers let it go
    for (uint32_t s = 0; s < STAGES && s < started; ++s) ok = wait_full(s, ((started - 1u - s) / STAGES) & 1u) && ok;
    return ok;
}

}  // namespace hg
