// ring_place.cuh -- where the chunks of a ring kernel go (host code, standard
// library only: the ring kernels' plans are worked out with it, ring.cuh).
#pragma once

#include <algorithm>
#include <vector>

namespace kami {
namespace ring {

constexpr int kRecs = 32;         // chunks in flight at most
constexpr int kAhead = 64 * 1024; // bytes in flight, the chunk that passes it included

// Places one CTA's chunks in order in a ring of `ring_bytes`, from its start
// again where the rest is too short.
class Placer
{
    struct Span
    {
        int from, to;
    };
    std::vector<Span> at_of; // ring bytes of the chunks so far
    int ring_bytes, recs, most;
    int head = 0, gone = -1;
    int window = 0, fly = 0; // the fewest last chunks of `most` bytes: their first, their bytes

  public:
    explicit Placer(int ring_bytes, int recs = kRecs, int most = kAhead) : ring_bytes(ring_bytes), recs(recs), most(most)
    {
    }
    void clear()
    {
        at_of.clear();
        head = window = fly = 0;
        gone = -1;
    }
    int count() const { return (int)at_of.size(); }
    // dep: the last chunk that must be done with before the bytes and the
    // record may be written.  land: the last one that must have landed.  Copies
    // in flight share the SM's bandwidth, so more of them than latency asks for
    // only delay the oldest: with the whole ring asked for at once the first
    // chunk lands with the last (FP64 64^3 x 610: 23.2 us, 20.0 with kAhead), and
    // FP64 32^3 x 65536 takes 290 us instead of 257.
    int place(int bytes, int *dep, int *land)
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
        // kept from chunk to chunk: counted back from each it is up to 32 steps for
        // small ones (plan of 20000 FP64 8^3: 2.23 ms to create, 2.05 so)
        auto size = [&](int c) { return at_of[c].to - at_of[c].from; };
        for (fly += bytes; window < j && fly - size(window) >= most; ++window)
            fly -= size(window);
        *land = std::max(gone, window - 1);
        return at;
    }
};

} // namespace ring
} // namespace kami
