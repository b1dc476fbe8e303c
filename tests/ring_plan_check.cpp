// Host check of the rings a run may use (csrc/ring_plan.h): where the memory of the first cannot be had, each next
// one asks for less, down to the size by the primaries alone (2^22..2^28 rays, 2048 a primary); a given size is taken
// alone; no ring is too small for four primaries' phase A.  Exit status 0 when all hold.  Built and run by
// tests/test_ring_plan.py (CPU only).
#include <cstdio>

#include "../pachydermacoustic_universal_gb300/csrc/ring_plan.h"

using namespace pach;

// ring and hits of a run, bytes (64 a ring slot, 16 a wave item; waves of 2^22 in several loops, 2^23 in one)
static double bytes(const RingPlan &p) {
    const double cap = (double)(1ull << p.log2), wave = p.loops > 1 ? 4194304.0 : 8388608.0;
    return p.loops * (64.0 * cap + 16.0 * std::min(cap, wave));
}

int main() {
    int bad = 0;
    auto wrong = [&](const char *what, long long n, int rooms, int flags) {
        if (++bad < 20) std::printf("%s: %lld primaries, %d rooms, flags %d\n", what, n, rooms, flags);
    };
    for (long long n : {1ll, 40ll, 256ll, 257ll, 1003ll, 2048ll, 2049ll, 20000ll, 60000ll, 131073ll, 1000000ll, 10000000ll})
        for (int rooms : {1, 2, 64})
            for (int flags = 0; flags < 4; ++flags) {
                const bool share = flags & 1, roomy = rooms > 1 || (flags & 2);
                const std::vector<RingPlan> v = ring_plans(0, n, rooms, share, roomy, 1000);
                int least = 22;
                while (least < 28 && (1ll << least) < n * 2048) ++least;
                if (v.empty()) { wrong("none", n, rooms, flags); continue; }
                if (v[0].loops != (share ? 3 : 1)) wrong("first", n, rooms, flags);
                if (v.back().loops != 1 || v.back().log2 != least) wrong("last", n, rooms, flags);
                for (size_t k = share ? 2 : 1; k < v.size(); ++k)  // after the loops' rings: one ring, ever smaller
                    if (bytes(v[k]) >= bytes(v[k - 1])) wrong("not smaller", n, rooms, flags);
                // large runs' primaries alone ask for the whole ring; every other run's last resort is smaller than the
                // three rings that could not be had
                const bool large = share && v[1].log2 == least;
                if (share && !large && bytes(v.back()) > bytes(v[0])) wrong("fallback larger than what failed", n, rooms, flags);
                // four primaries' phase A has to fit
                for (unsigned long long bound : {1ull << 20, (1ull << 20) + 1, 1ull << 22, 1ull << 26, (1ull << 26) + 1})
                    for (const RingPlan &p : ring_plans(0, n, rooms, share, roomy, bound))
                        if (4 * bound > (1ull << p.log2)) wrong("too small", n, rooms, flags);
            }
    for (int given : {1, 16, 19, 28, 32, 40}) {
        const std::vector<RingPlan> v = ring_plans(given, 5000, 1, false, true, 16);
        if (v.size() != 1 || v[0].loops != 1 || v[0].log2 != std::min(32, std::max(16, given))) wrong("given", given, 1, 0);
    }
    std::printf("%d faults\n", bad);
    return bad != 0;
}
