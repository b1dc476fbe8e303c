// filters.h -- shared by the receiver-filter translation units (filters.cu, filters_ntt.cu).
#pragma once
#include "engine.h"

namespace pach {

constexpr int kCarrierLen = 16384;

// The histograms and per-call values that the envelopes of filters job0 .. are formed from.
struct FilterJob {
    const double *E, *P, *Dp, *Dn, *scale;
    const double *att;       // [T] 16 kHz ramp
    const double *car;       // [9][16384] carriers (carrier mode: the envelopes are these)
    double pmod[kBands];
    int T, kinds, job0;
};

// filters_ntt.cu: integer transforms, for T + 16383 <= 65536.  add: dB/m by which the 16 kHz band decays faster
// than the 8 kHz one.
bool ntt_supported(int T);
size_t ntt_workspace_bytes(int n_filters, int T);
cudaError_t ntt_filters(FilterJob J, int n, int fs, double add, int L, double *out, void *ws, size_t ws_bytes,
                        cudaStream_t st);

}  // namespace pach
