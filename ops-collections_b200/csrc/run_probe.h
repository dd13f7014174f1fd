// run_probe.h -- where the probing of the multimap's index goes and where it
// ends (multi.cu).  Plain C++, so that the rules can be run on the CPU as well.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define B2CO_PROBE_HD __host__ __device__ __forceinline__
#else
#define B2CO_PROBE_HD inline
#endif

namespace b2co {
namespace multi {

// A key's probing goes round the region (a power of two of slots) that it
// starts in; `region` is the region's size - 1.
template <class Index>
B2CO_PROBE_HD Index next_in_region(Index s, Index region)
{
    return (s & ~region) | ((s + 1) & region);
}

// Whether a region with this many keys is too full to be asked: what a build
// that sized its table by an estimate, or dealt it out by the hash's leading
// bits, checks after the fact.  Keys taken at random fill a region of 512 slots
// to less than half, and this is eight standard deviations above half; but
// nothing else keeps keys made for it from filling one to the last slot.
B2CO_PROBE_HD bool region_crowded(uint64_t keys, uint64_t slots) { return keys > slots / 4 * 3; }

enum { kProbeOn = 0, kProbeHit = 1, kProbeMiss = 2 };

// Walks from slot s until look(s) says hit or miss, at most once round the
// region; whether it was a hit.
template <class Index, class Look>
B2CO_PROBE_HD bool walk_region(Index start, Index region, Look look)
{
    Index s = start;
    do {
        int const what = look(s);
        if (what != kProbeOn) return what == kProbeHit;
        s = next_in_region(s, region);
    } while (s != start);
    return false;
}

}  // namespace multi
}  // namespace b2co
