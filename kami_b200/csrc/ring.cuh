// ring.cuh -- shared-memory ring of the persistent ring kernels (f64_ring.cu,
// h16_ring.cu): copying warps put chunks into a byte ring, computing warps
// take them in order.  Chunk j of a CTA uses record j % kRecs with the
// barriers full[] (its bytes and record are there) and empty[] (every
// computing warp is done with it).  Where a chunk goes, and what has to come
// before it, is worked out beforehand, so copying warps share no state.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#include "tc05_ptx.cuh"

namespace kami {
namespace ring {

constexpr int kRecs = 32;                   // chunks in flight at most
constexpr int kAhead = 64 * 1024;           // bytes in flight, the chunk that passes it included

__host__ __device__ constexpr int up128(int bytes) { return (bytes + 127) & ~127; }

// Host: places one CTA's chunks in order in a ring of `ring_bytes`, from its
// start again where the rest is too short.
class Placer
{
    struct Span
    {
        int from, to;
    };
    std::vector<Span> at_of; // ring bytes of the chunks so far
    int ring_bytes, recs, head = 0, gone = -1;

  public:
    explicit Placer(int ring_bytes, int recs = kRecs) : ring_bytes(ring_bytes), recs(recs) {}
    void clear()
    {
        at_of.clear();
        head = 0;
        gone = -1;
    }
    int count() const { return (int)at_of.size(); }
    // dep: the last chunk that must be done with before the bytes and the
    // record may be written.  land: the last one that must have landed.  Copies
    // in flight share the SM's bandwidth, so more of them than latency asks for
    // only delay the oldest: with the whole ring asked for at once the first
    // chunk lands with the last (FP64 64^3 x 610: 23.2 us, 20.0 with kAhead), and
    // FP64 32^3 x 65536 takes 290 us instead of 257.
    int place(int bytes, int *dep, int *land, int most = kAhead)
    {
        const int j = count(), at = head + bytes > ring_bytes ? 0 : head, end = at + bytes;
        // The chunks whose bytes this one takes: the oldest that are left, after
        // those behind the place where the ring starts again.  Never fewer than
        // for the previous chunk, which may have taken part of an older one's
        // bytes, and this the rest.
        gone = std::max(gone, j - recs);
        int q = gone + 1;
        while (q < j && at < head && at_of[q].from >= head)
            ++q;
        for (; q < j && at_of[q].from < end && at < at_of[q].to; ++q)
            gone = q;
        *dep = gone;
        head = end;
        at_of.push_back(Span{at, end});
        int fly = bytes;
        for (*land = j - 1; *land > gone && fly < most; --*land)
            fly += at_of[*land].to - at_of[*land].from;
        return at;
    }
};

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
