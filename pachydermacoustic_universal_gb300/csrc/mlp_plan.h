// mlp_plan.h -- how the proposal network's weight gradients are split over training rows (mlp.cu; host only).
#pragma once
#include <algorithm>

namespace pach {
namespace mlp {

constexpr int kRowChunk = 128;   // rows of one operand copy: ranges are whole chunks
constexpr int kMaxSplits = 16;   // row ranges of the weight-gradient products

// Row ranges of the weight gradients for Mp rows: at least 256 rows each (two chunks in flight), at most
// kMaxSplits, whose sums the optimiser reads.  1200 rows: k_wgrad 14.4 us in one range, 7 us in five and 1 us more
// in k_adam.
inline int wgrad_ranges_wanted(int Mp) { return std::max(1, std::min(kMaxSplits, Mp / 256)); }
inline int wgrad_rows_per(int Mp) {
    const int s = wgrad_ranges_wanted(Mp);
    return ((Mp + s - 1) / s + kRowChunk - 1) / kRowChunk * kRowChunk;
}
inline int wgrad_splits(int Mp) { return (Mp + wgrad_rows_per(Mp) - 1) / wgrad_rows_per(Mp); }

// Most ranges of any row count up to Mp.  Rounding the ranges to whole chunks makes their number fall again as the
// rows grow (1024 rows 4, 1152 rows 3), so what the largest count takes is not enough; the number wanted only rises.
inline int wgrad_splits_max(int Mp) { return wgrad_ranges_wanted(Mp); }

}  // namespace mlp
}  // namespace pach
