// ring.cuh -- shared-memory ring of the persistent ring kernels (f64_ring.cu,
// h16_ring.cu): copying warps put chunks into a byte ring, computing warps
// take them in order.  Chunk j of a CTA uses record j % kRecs with the
// barriers full[] (its bytes and record are there) and empty[] (every
// computing warp is done with it).  Where a chunk goes, and what has to come
// before it, is worked out beforehand, so copying warps share no state.
#pragma once

#include <cstdint>

#include "ring_place.cuh"
#include "tc05_ptx.cuh"

namespace kami {
namespace ring {

__host__ __device__ constexpr int up128(int bytes) { return (bytes + 127) & ~127; }

// Copying warp: waits until chunk `dep` is done with; `gone`: the last chunk
// known to be.  The computing warps pass the chunks in order, so a chunk's
// barrier answers for the older ones too.  A wait on parity cannot tell a
// phase from the one two ahead: never further than RECS past what is known.
template <int RECS = kRecs>
__device__ __forceinline__ bool wait_gone(uint64_t *empty, int dep, int &gone, uint64_t limit)
{
    bool ok = true;
    while (gone < dep && ok)
    {
        const int to = min(dep, gone + RECS);
        ok = __all_sync(0xffffffffu, tc::mbar_wait_bounded(&empty[to % RECS], (to / RECS) & 1, limit));
        gone = to;
    }
    return ok;
}

// ... until chunk `land` (negative: none) has landed.  A warp that is slow may
// come here when the chunk is done with and other warps have put another one
// into its record, so that full[] is a phase further; empty[] cannot be, that
// chunk being behind this warp's own.
__device__ __forceinline__ bool wait_landed(uint64_t *full, uint64_t *empty, int land, int gone, uint64_t limit)
{
    if (land <= gone)
        return true;
    const int s = land % kRecs, parity = (land / kRecs) & 1;
    uint64_t t0 = 0;
    while (!__all_sync(0xffffffffu, tc::mbar_try_wait(&full[s], parity) || tc::mbar_test(&empty[s], parity)))
    {
        const uint64_t now = tc::globaltimer_ns();
        t0 = t0 ? t0 : now;
        if (__any_sync(0xffffffffu, now - t0 > limit))
            return false;
    }
    return true;
}

} // namespace ring
} // namespace kami
