// Host check of the quotient of csrc/quotient.h against the division: equal for x = 0 and x from 2^-96 to 1 with
// q from 1 to 32 (random mantissas, and the ends of q's and x's mantissas where a rounded reciprocal is worst), and
// one of the two floats next to it below.  Exit status 0 when both hold.  Built and run by tests/test_quotient.py (CPU only).
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>

#include "../pachydermacoustic_universal_gb300/csrc/quotient.h"

int main() {
    std::mt19937_64 rng(1);
    long wrong = 0, far = 0, below = 0;
    for (long i = 0; i < 20000000; ++i) {
        const uint64_t v = rng();
        uint32_t qm = (uint32_t)v & 0x7FFFFF, xm = (uint32_t)(v >> 32) & 0x7FFFFF;
        if (i % 16 == 0) qm = 0x7FFFFF - (qm & 7);
        if (i % 16 == 1) qm &= 7;
        if (i % 16 == 2) xm = 0x7FFFFF - (xm & 7);
        if (i % 16 == 3) xm &= 7;
        const float q = std::fmin(32.f, std::ldexp(1.f + qm * 0x1p-23f, (int)((v >> 23) % 6)));
        const float x = i % 1000 == 0 ? 0.f : std::fmin(1.f, std::ldexp(1.f + xm * 0x1p-23f, -(int)((v >> 55) % 151)));
        const float got = pach::mlp::quotient(x, q, 1.f / q), ref = x / q;
        if (x == 0.f || x >= pach::mlp::kQuotientExact) {
            if (got != ref && wrong++ < 10) std::printf("%a / %a: %a, not %a\n", x, q, got, ref);
        } else {
            ++below;
            if (got != ref && got != std::nextafterf(ref, 1.f) && got != std::nextafterf(ref, 0.f) && far++ < 10) std::printf("%a / %a: %a, far from %a\n", x, q, got, ref);
        }
    }
    std::printf("%ld not the division's, %ld of %ld far below\n", wrong, far, below);
    return wrong || far || !below;
}
