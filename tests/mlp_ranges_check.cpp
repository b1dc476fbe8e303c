// Host check of the weight gradients' row ranges (csrc/mlp_plan.h): a network made for up to Mp_max rows holds as
// many partial products as training on any fewer rows writes, and the ranges cover the rows exactly once.  Exit
// status 0 when all hold.  Built and run by tests/test_mlp_ranges.py (CPU only).
#include <cstdio>

#include "../pachydermacoustic_universal_gb300/csrc/mlp_plan.h"

using namespace pach::mlp;

int main() {
    int bad = 0, most = 0;
    for (int Mp = 128; Mp <= 65536; Mp += 128) {  // rows are padded to whole tiles of 128
        const int per = wgrad_rows_per(Mp), n = wgrad_splits(Mp);
        if (per % 128 || n < 1 || (long long)(n - 1) * per >= Mp || (long long)n * per < Mp) {
            if (++bad < 20) std::printf("rows %d: %d ranges of %d\n", Mp, n, per);
        }
        most = n > most ? n : most;
        // `most`: what some row count up to Mp takes; the buffer of a network of Mp rows holds wgrad_splits_max(Mp)
        if (most > wgrad_splits_max(Mp) || wgrad_splits_max(Mp) > kMaxSplits) {
            if (++bad < 20) std::printf("up to %d rows: %d ranges, room for %d\n", Mp, most, wgrad_splits_max(Mp));
        }
    }
    std::printf("%d faults\n", bad);
    return bad != 0;
}
