// The rules by which the multimap's index is probed and refused (csrc/run_probe.h), run on the CPU: a build that fills
// a region to the last slot is refused, and a lookup ends whatever the region holds.
#include <cstdio>
#include <vector>

#include "run_probe.h"

using namespace b2co::multi;

namespace {

constexpr uint64_t kSlots = 512, kMaxProbes = 128;  // as a block builds its region
constexpr uint64_t kEmpty = ~0ull;

struct Region {
    std::vector<uint64_t> keys = std::vector<uint64_t>(kSlots, kEmpty);
    uint64_t placed = 0;
    bool crowded = false;
    void place(uint64_t key, uint64_t start)
    {
        uint64_t s = start;
        for (uint64_t probes = 0; probes < kMaxProbes; ++probes, s = next_in_region(s, kSlots - 1)) {
            if (keys[s] == key) return;
            if (keys[s] == kEmpty) {
                keys[s] = key;
                ++placed;
                return;
            }
        }
        crowded = true;
    }
    bool refused() const { return crowded || region_crowded(placed, kSlots); }
    // hit, and the slots looked at (walk_region ends on its own; the count shows where)
    bool find(uint64_t key, uint64_t start, uint64_t& looks) const
    {
        looks = 0;
        return walk_region(start, kSlots - 1, [&](uint64_t s) {
            ++looks;
            return int(keys[s] == key ? kProbeHit : keys[s] == kEmpty ? kProbeMiss : kProbeOn);
        });
    }
};

int failures = 0;
void check(bool ok, char const* what)
{
    if (!ok) std::printf("FAILED: %s\n", what), ++failures;
}

}  // namespace

int main()
{
    uint64_t looks;
    // a key for every start: no key probes at all, and no slot is left
    Region full;
    for (uint64_t i = 0; i < kSlots; ++i) full.place(1000 + i, i);
    check(!full.crowded && full.placed == kSlots, "512 starts fill the region without a probe");
    check(full.refused(), "a full region is refused");
    for (uint64_t start : {uint64_t(0), uint64_t(77), kSlots - 1}) {
        check(!full.find(5, start, looks) && looks == kSlots, "an absent key's walk ends after one round");
        check(full.find(1000 + start, start, looks) && looks == 1, "a present key is found");
    }
    // the other starts of the same region number stay in the region
    check(next_in_region(3 * kSlots + kSlots - 1, kSlots - 1) == 3 * kSlots, "probing goes round the region");
    // around the line, and what random keys reach
    for (uint64_t n : {uint64_t(0), uint64_t(1), kSlots / 2, kSlots / 4 * 3}) check(!region_crowded(n, kSlots), "not crowded");
    for (uint64_t n : {kSlots / 4 * 3 + 1, kSlots}) check(region_crowded(n, kSlots), "crowded");
    check(!region_crowded(uint64_t(1) << 31, uint64_t(1) << 32), "a table of full size is half full");
    // one start for all: refused by the probes
    Region one;
    for (uint64_t i = 0; i < 300; ++i) one.place(1000 + i, 7);
    check(one.crowded && one.refused(), "300 keys of one start are refused");
    // a region that is not refused has an empty slot, where every absent key's walk ends
    Region ok;
    for (uint64_t i = 0; i < kSlots / 4 * 3; ++i) ok.place(1000 + i, i);
    check(!ok.refused() && !ok.find(5, 0, looks) && looks == kSlots / 4 * 3 + 1, "three quarters");
    if (!failures) std::printf("run probe test ok\n");
    return failures != 0;
}
