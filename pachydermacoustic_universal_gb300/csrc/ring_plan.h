// ring_plan.h -- the ring queues a run may use (host only).
#pragma once
#include <algorithm>
#include <vector>

namespace pach {

constexpr int kPipes = 3;    // device loops that a run is shared out to
constexpr int kRingLeast = 22;
constexpr int kRingMost = 28;
// Default ring of small scenes' runs and of batches that keep one device loop, at least (log2): 1 GB.  2^22 leaves a
// 1003-primary shoebox room for one or two interactions a wave (96 waves, 12.9 ms; 30 waves, 9.6 ms with 2^24; three
// loops of a third of the primaries and 2^22 rays each take 8.7 ms).
constexpr int kRingMin = 24;

struct RingPlan {
    int loops, log2;         // `loops` rings of 2^log2 octave rays
};

// Room for the run's rays at up to 2048 live octave rays per primary, 2^22..2^28 (17 GB).
inline int ring_log2_for(long long primaries) {
    int l = kRingLeast;
    while (l < kRingMost && (1ull << l) < (unsigned long long)primaries * 2048ull) ++l;
    return l;
}

// The rings a run may use, the one to try first at the front; the next ones for when the memory cannot be had.
// given: the caller's ring_log2 (0: none); share: the primaries may be shared out to several loops; roomy: several
// rooms, or a small scene whose rays leave several children a wave; bound: ring slots that one primary's phase A
// can fill (a ring holds at least four).
// A loop's ring is a quarter of the whole one, but no less than what keeps its waves full (a batch's pilots run
// several rooms at a time: 8 rooms of 500 primaries 258 ms with 2^22 rays, 248 with 2^23, 257 with 2^24).  The last
// resort of batches and small scenes is the size by primaries alone: a small run then takes 0.34 GB with its hits,
// where three loops take 1.0 and the roomy ring 1.2.
inline std::vector<RingPlan> ring_plans(int given, long long primaries, int rooms, bool share, bool roomy,
                                        unsigned long long bound) {
    std::vector<RingPlan> all, fit;
    if (given > 0) {
        all.push_back({1, std::min(32, std::max(16, given))});
    } else {
        const int least = ring_log2_for(primaries), one = roomy ? std::max(kRingMin, least) : least;
        if (share) all.push_back({kPipes, std::max(rooms > 1 ? 23 : kRingLeast, one - 2)});
        all.push_back({1, one});
        if (least < one) all.push_back({1, least});
    }
    for (const RingPlan &p : all)
        if (bound * 4 <= (1ull << p.log2)) fit.push_back(p);
    return fit;
}

}  // namespace pach
