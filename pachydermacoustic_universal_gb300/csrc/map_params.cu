// map_params.cu -- room-acoustic parameters of many energy-time curves at once, on the device.
//
// A map of 10^3..10^5 receivers x 8 bands is 10^4..10^6 curves that already sit in HBM after the
// trace; the reference derives its parameter maps one curve at a time on the host
// (Pach_Map_Receiver.cs:925-1270 calling AcousticalMath, Classes_Math.cs:282-586, 934-962).  Here one
// warp takes one curve, FP64 throughout: k_curve_params holds it in shared memory and needs about four FP64
// instructions a bin (GB300 issues one FP64 warp instruction per SM in 16 cycles, so those are the time);
// curve_general streams it in three passes with a logarithm a bin.
#include <algorithm>
#include <cmath>

#include "engine.h"

namespace pach {
namespace {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    return v;
}

// inclusive prefix sum over the warp
__device__ __forceinline__ double warp_scan(double v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(FULL, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

// Log10Data (Classes_Math.cs:392-408) of the Schroeder curve at bin i: 10 log10(S) floored at -60 dB,
// bin 0 left at 0.
__device__ __forceinline__ double level(double S, int i) {
    if (i == 0) return 0.0;
    return S >= 1e-6 ? 10.0 * log10(S) : -60.0;
}

// first index >= from (and >= 1) of a warp chunk whose flag is set, or -1
__device__ __forceinline__ int first_set(unsigned ballot, int base, int from) {
    const int skip = from - base;
    if (skip >= 32) return -1;
    if (skip > 0) ballot &= ~((1u << skip) - 1u);
    return ballot ? base + __ffs(ballot) - 1 : -1;
}

struct Out {
    double *t_x, *edt, *clar, *defi, *sum;
};

// Curve w = x [T] for any values and length.  All 32 lanes call.
__device__ __noinline__ void curve_general(const double *x, int w, int T, double fs, double scale, int depth,
                                           double clar_s, Out o) {
    const int lane = threadIdx.x & 31;
    // pass 1: total, and the early sums of Clarity (start 0: bins [0, ei)) and Definition
    const int ei_c = (int)floor((clar_s + 0.0) * fs), ei_d = (int)floor(0.05 * fs);
    double tot = 0, ec = 0, lc = 0, ed = 0;
    for (int i = lane; i < T; i += 32) {
        const double v = x[i] * scale;
        tot += v;
        if (i < ei_c) ec += v;
        if (i > ei_c) lc += v;
        if (i < ei_d) ed += v;
    }
    tot = warp_sum(tot);
    ec = warp_sum(ec);
    lc = warp_sum(lc);
    ed = warp_sum(ed);
    // Clarity (559-586): the boundary bin is split between early and late
    const double bw = 1.0 / fs;
    if (ei_c >= 0 && ei_c < T) {
        const double split = (clar_s + 0.0 - ei_c * bw) / bw, v = x[ei_c] * scale;
        ec += split * v;
        lc += (1 - split) * v;
    }
    double edd = ed;
    if (ei_d >= 0 && ei_d < T) edd += (0.05 + 0.0 - ei_d * bw) / bw * x[ei_d] * scale;
    // pass 2: fit limits on the Schroeder curve S[i] = 1 - cumsum[i] / total (Schroeder_Limits, 417-438)
    const double first30 = -5.0, second30 = -5.0 - fabs((double)depth);
    const double first_e = -1.0, second_e = -10.0001;
    int a30 = -1, b30 = -1, ae = -1, be = -1;
    double carry = 0;
    for (int base = 0; base < T && (b30 < 0 || be < 0); base += 32) {
        const int i = base + lane;
        const double v = i < T ? x[i] * scale : 0.0;
        const double cum = carry + warp_scan(v, lane);
        carry = __shfl_sync(FULL, cum, 31);
        const double S = tot == 0 ? 0.0 : 1.0 - cum / tot;
        const double l = i < T ? level(S, i) : 0.0;
        const bool ok = i < T;
        if (a30 < 0) a30 = first_set(__ballot_sync(FULL, ok && i >= 1 && l < first30), base, 1);
        if (a30 >= 0 && b30 < 0) b30 = first_set(__ballot_sync(FULL, ok && l < second30), base, a30);
        if (ae < 0) ae = first_set(__ballot_sync(FULL, ok && i >= 1 && l < first_e), base, 1);
        if (ae >= 0 && be < 0) be = first_set(__ballot_sync(FULL, ok && l < second_e), base, ae);
    }
    // not found: index 0, as the reference's loops leave them
    if (a30 < 0) a30 = 0;
    if (ae < 0) ae = 0;
    if (b30 < 0) b30 = 0;
    if (be < 0) be = 0;
    // pass 3: least-squares slopes over [a, b] of each fit, time axis (i - a) / fs (Least_Square_Fit, 446-473)
    double s30[4] = {0, 0, 0, 0}, se[4] = {0, 0, 0, 0};  // sum q, sum y, sum q^2, sum q y
    const int end = max(b30, be);
    carry = 0;
    for (int base = 0; base <= end; base += 32) {
        const int i = base + lane;
        const double v = i < T ? x[i] * scale : 0.0;
        const double cum = carry + warp_scan(v, lane);
        carry = __shfl_sync(FULL, cum, 31);
        if (i >= T) continue;
        const double S = tot == 0 ? 0.0 : 1.0 - cum / tot;
        const double l = level(S, i);
        if (i >= a30 && i <= b30) {
            const double q = (i - a30) / fs;
            s30[0] += q; s30[1] += l; s30[2] += q * q; s30[3] += q * l;
        }
        if (i >= ae && i <= be) {
            const double q = (i - ae) / fs;
            se[0] += q; se[1] += l; se[2] += q * q; se[3] += q * l;
        }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        s30[k] = warp_sum(s30[k]);
        se[k] = warp_sum(se[k]);
    }
    if (lane) return;
    auto fit = [&](const double (&s)[4], int a, int b) -> double {
        const int len = b - a + 1;
        if (len < 1) return NAN;
        const double slope = (len * s[3] - s[0] * s[1]) / (len * s[2] - s[0] * s[0]);
        return -60.0 / slope;
    };
    if (o.t_x) o.t_x[w] = fit(s30, a30, b30);
    if (o.edt) o.edt[w] = fit(se, ae, be);
    if (o.clar) o.clar[w] = 10.0 * log10(ec / lc);
    if (o.defi) o.defi[w] = edd / tot * 100.0;
    if (o.sum) o.sum[w] = tot;
}

__global__ void __launch_bounds__(256) k_map_params(const double *etc, int n, int T, double fs, double scale,
                                                    int depth, double clar_s, Out o) {
    const int w = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
    if (w < n) curve_general(etc + (size_t)w * T, w, T, fs, scale, depth, clar_s, o);
}

// x = m 2^e with m in [1, 2), for normal positive x.
__device__ __forceinline__ double split2(double x, int &e) {
    const int hi = __double2hiint(x);
    e = (hi >> 20) - 1023;
    return __hiloint2double((hi & 0x000FFFFF) | 0x3FF00000, __double2loint(x));
}

__device__ __forceinline__ int warp_isum(int v) { return __reduce_add_sync(FULL, v); }

// The two sums of a least-squares fit over bins [a, b], in units of log2: sum l_i and sum (i - a) l_i with
// l_i = log2 of the Schroeder curve (not below 1e-6).  No logarithm a bin: lane t takes r consecutive bins
// and keeps P, the product of their curve values, and W, the product of P's successive values, as mantissas
// in [1, 2) with integer exponents; log2 P is the lane's sum and log2 W its sum weighted r - j.  Products over
// the lanes (and of their suffix products, for the lane offsets) leave three numbers per fit, whose
// logarithms the caller takes: lg[0] = sum l, lg[1] = sum (t + 1) (lane t's sum), lg[2] = sum log2 W.
struct FitSums {
    double m[3];
    int e[3];
    int r;
};

__device__ __forceinline__ FitSums fit_products(const double *cum, const double *base, int c, int a, int b, double rt) {
    const int lane = threadIdx.x & 31;
    FitSums f;
    f.r = (b - a + 32) / 32;
    double P = 1.0, W = 1.0;
    int eP = 0, eW = 0;
    const int i0 = a + lane * f.r;
    int ch = i0 / c, next = (ch + 1) * c;
    double bs = base[min(ch, 63)];
#pragma unroll 4
    for (int j = 0; j < f.r; ++j) {
        const int i = i0 + j;
        if (i <= b) {
            if (i == next) {
                bs = base[++ch];
                next += c;
            }
            const double S = fma(-(bs + cum[i]), rt, 1.0);
            int e, g;
            // S >= 1e-6, compared as bits (positive doubles order as integers; a negative S is below)
            const double m = split2(__double_as_longlong(S) >= __double_as_longlong(1e-6) ? S : 1e-6, e);
            P = split2(P * m, g);
            eP += e + g;
        }
        W *= P;  // at most 2^r, r <= T / 32
        eW += eP;
    }
    int g;
    W = split2(W, g);
    eW += g;
    // suffix products over the lanes
    double Q = P;
    int eQ = eP;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_down_sync(FULL, Q, o);
        const int v = __shfl_down_sync(FULL, eQ, o);
        if (lane + o < 32) {
            Q *= u;
            eQ += v;
        }
    }
    f.m[0] = __shfl_sync(FULL, Q, 0);
    f.e[0] = __shfl_sync(FULL, eQ, 0);
    Q = split2(Q, g);
    eQ += g;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        Q *= __shfl_xor_sync(FULL, Q, o);
        W *= __shfl_xor_sync(FULL, W, o);
    }
    f.m[1] = Q;
    f.e[1] = warp_isum(eQ);
    f.m[2] = W;
    f.e[2] = warp_isum(eW);
    return f;
}

// Curves of up to kSharedBins bins, one warp each, in shared memory.  The curve is read once; lane t sums
// chunks t and t + 32 of c = T / 64 bins (c odd: no bank conflicts; two chains in flight) and leaves their
// running sums, a scan makes them the Schroeder curve, the fit limits are binary searches on it (energies are not negative, so it falls monotonically; the
// limits in dB are compared as ratios) and the fits are products (fit_products).  608 receivers x 8 bands x
// 3000 bins: 160 us (FP64 pipe 64 % busy), where a logarithm a bin in two of three passes took 1155 us (85 %
// busy).  A curve with a negative, infinite or undefined value, or whose total is not above zero or has no finite
// reciprocal, goes to curve_general.
constexpr int kSharedBins = 6000;  // 48 KB: four curves an SM still keep the FP64 pipe half busy
constexpr int kFourBytes = 27 * 1024;  // curves up to this size go four to a block
// Most dynamic shared memory of a launch.  The kernel's limit is one value for the whole device and every call sets
// it to this, whatever its own curves need: a call with longer curves on another thread launches in between.
constexpr int kMaxSharedBytes = 4 * kFourBytes;
__host__ __device__ constexpr int chunk_bins(int T) { return ((T + 63) / 64) | 1; }

// what every curve of a launch shares
struct Curves {
    double limit[4];         // curve values at the fits' limits: T_X first and second, EDT first and second
    double db[4];            // the limits themselves
    double split_c, split_d; // shares of the boundary bins ei_c, ei_d that are early
    double inv_fs;
    int ei_c, ei_d;
};

__global__ void __launch_bounds__(128) k_curve_params(const double *etc, int n, int T, double fs, double scale, int depth,
                                                      double clar_s, Curves k, Out o) {
    extern __shared__ double s_curve[];
    __shared__ double s_base[4][64];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int w = (int)(blockIdx.x * (blockDim.x >> 5)) + wid;
    if (w >= n) return;
    const int c = chunk_bins(T);
    double *cum = s_curve + (size_t)wid * 64 * c, *base = s_base[wid];
    const double *x = etc + (size_t)w * T;
    int odd = 0;
    for (int i = lane; i < 64 * c; i += 32 * 8) {  // eight loads in flight a lane
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = i + 32 * q < T ? __ldcs(x + i + 32 * q) : 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int hi = __double2hiint(v[q]);
            odd |= hi < 0 || hi >= 0x7FF00000;
            if (i + 32 * q < 64 * c) cum[i + 32 * q] = v[q];
        }
    }
    __syncwarp();
    double run = 0.0, run2 = 0.0;
    {
        double *p = cum + lane * c, *q = cum + (lane + 32) * c;
#pragma unroll 4
        for (int j = 0; j < c; ++j) {
            run += p[j];
            run2 += q[j];
            p[j] = run;
            q[j] = run2;
        }
    }
    const double incl = warp_scan(run, lane), incl2 = warp_scan(run2, lane);
    const double half = __shfl_sync(FULL, incl, 31);
    const double before = __shfl_up_sync(FULL, incl, 1), before2 = __shfl_up_sync(FULL, incl2, 1);
    base[lane] = lane ? before : 0.0;
    base[lane + 32] = half + (lane ? before2 : 0.0);
    const double tot = half + __shfl_sync(FULL, incl2, 31);
    const double rt = 1.0 / tot;
    if (__any_sync(FULL, odd) || !(tot > 0.0) || isinf(tot) || isinf(rt)) {
        curve_general(x, w, T, fs, scale, depth, clar_s, o);
        return;
    }
    __syncwarp();
    auto sum_to = [&](int i) { return base[i / c] + cum[i]; };  // bins 0 .. i
    // fit limits: first bin >= 1 below each level (lanes 0-3: T_X first and second, EDT first and second)
    const double th = k.limit[lane & 3], db = k.db[lane & 3];
    auto first_where = [&](auto below) {
        int lo = 1, hi = T;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (below(mid)) hi = mid;
            else lo = mid + 1;
        }
        return lo;
    };
    auto curve = [&](int i) { return fma(-sum_to(i), rt, 1.0); };
    int lo = T;
    if (lane < 4) {
        lo = first_where([&](int i) { return curve(i) < th; });
        // A bin within rounding of the limit (steps of equal bins: 1 - 99 / 100 at -20 dB) is decided by the quotient
        // and the logarithm, as curve_general does.
        if ((lo < T && fabs(curve(lo) - th) < 1e-14) || (lo > 1 && fabs(curve(lo - 1) - th) < 1e-14))
            lo = first_where([&](int i) { return level(1.0 - sum_to(i) / tot, i) < db; });
    }
    // not found: index 0, as the reference's loops leave them; a fit of one bin or less has no slope
    const int f0 = __shfl_sync(FULL, lo, 0), f1 = __shfl_sync(FULL, lo, 1), f2 = __shfl_sync(FULL, lo, 2),
              f3 = __shfl_sync(FULL, lo, 3);
    const bool fit30 = f1 < T && f1 > f0, fite = f3 < T && f3 > f2;
    FitSums F[2] = {};
    if (fit30) F[0] = fit_products(cum, base, c, f0, f1, rt);
    if (fite) F[1] = fit_products(cum, base, c, f2, f3, rt);
    // late sum of Clarity, bins > ei: whole chunks, and the rest of the boundary's from the curve itself
    const int first_late = k.ei_c < 0 ? 0 : (k.ei_c >= T ? T : k.ei_c + 1);
    const int ch = (first_late + c - 1) / c;  // first chunk that is late throughout
    double late = (lane >= ch ? run : 0.0) + (lane + 32 >= ch ? run2 : 0.0);
    for (int i = first_late + lane; i < min(T, ch * c); i += 32) late += x[i];
    late = warp_sum(late);
    double early = k.ei_c <= 0 ? 0.0 : sum_to(min(k.ei_c, T) - 1);
    if (k.ei_c >= 0 && k.ei_c < T) {  // the boundary bin is split between early and late
        const double v = x[k.ei_c];
        early += k.split_c * v;
        late += (1 - k.split_c) * v;
    }
    double early_d = k.ei_d <= 0 ? 0.0 : sum_to(min(k.ei_d, T) - 1);
    if (k.ei_d >= 0 && k.ei_d < T) early_d += k.split_d * x[k.ei_d];
    // the logarithms of the six products and of early / late, one lane each: a scalar FP64 instruction takes
    // the pipe as long as a warp's
    double lg = early / late;
    int le = 0;
#pragma unroll
    for (int q = 0; q < 6; ++q)
        if (lane == q) {
            lg = F[q / 3].m[q % 3];
            le = F[q / 3].e[q % 3];
        }
    const double l2 = log2(lg) + (double)le;
    // Least-squares slope over len bins 0 .. len - 1 at fs (Least_Square_Fit, 446-473), its time sums in closed
    // form: T = -60 / slope = -5 len (len^2 - 1) / fs / (sum k l - (len - 1) / 2 sum l).  Lane 0: T_X, 1: EDT,
    // 2: definition.
    const int base_lane = lane == 1 ? 3 : 0;
    const double p0 = __shfl_sync(FULL, l2, base_lane), p1 = __shfl_sync(FULL, l2, base_lane + 1),
                 p2 = __shfl_sync(FULL, l2, base_lane + 2), cl = __shfl_sync(FULL, l2, 6);
    const double dB = 3.0102999566398119521;  // 10 log10(2)
    const int len = lane == 1 ? f3 - f2 + 1 : f1 - f0 + 1;
    const double dl = (double)len, fr = (double)(lane == 1 ? F[1].r : F[0].r);
    double num = -5.0 * dl * (dl * dl - 1.0) * k.inv_fs, den = dB * (fr * p1 - p2 - (dl - 1.0) * 0.5 * p0);
    if (lane == 2) {
        num = early_d * 100.0;
        den = tot;
    }
    const double v = num / den;
    if (lane == 0 && o.t_x) o.t_x[w] = fit30 ? v : NAN;
    if (lane == 1 && o.edt) o.edt[w] = fite ? v : NAN;
    if (lane == 2 && o.defi) o.defi[w] = v;
    if (lane == 3 && o.clar) o.clar[w] = dB * cl;
    if (lane == 4 && o.sum) o.sum[w] = tot * scale;
}

// Curve value below which the level is under `db`; levels stop at -60, so none is under that.
double level_ratio(double db) { return db > -60.0 ? std::pow(10.0, db / 10.0) : -HUGE_VAL; }

}  // namespace

cudaError_t launch_map_params(const double *etc, int n, int T, double fs, double scale, int decay_depth,
                              double clarity_s, double *t_x, double *edt, double *clarity, double *definition,
                              double *sum, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const Out o{t_x, edt, clarity, definition, sum};
    if (T <= kSharedBins) {
        const int per = 64 * chunk_bins(T) * (int)sizeof(double);
        const int warps = per <= kFourBytes ? 4 : 1;
        static_assert(64 * chunk_bins(kSharedBins) * sizeof(double) <= kMaxSharedBytes, "one curve a block");
        const cudaError_t e = cudaFuncSetAttribute(k_curve_params, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   kMaxSharedBytes);
        if (e != cudaSuccess) return e;
        const double bw = 1.0 / fs;
        Curves k;
        k.db[0] = -5.0;
        k.db[1] = -5.0 - std::fabs((double)decay_depth);
        k.db[2] = -1.0;
        k.db[3] = -10.0001;
        for (int i = 0; i < 4; ++i) k.limit[i] = level_ratio(k.db[i]);
        k.ei_c = (int)std::floor((clarity_s + 0.0) * fs);
        k.ei_d = (int)std::floor(0.05 * fs);
        k.split_c = (clarity_s + 0.0 - k.ei_c * bw) / bw;
        k.split_d = (0.05 + 0.0 - k.ei_d * bw) / bw;
        k.inv_fs = bw;
        k_curve_params<<<(n + warps - 1) / warps, 32 * warps, (size_t)warps * per, s>>>(
            etc, n, T, fs, scale, decay_depth, clarity_s, k, o);
    } else {
        const int blocks = (int)(((long long)n * 32 + 255) / 256);
        k_map_params<<<blocks, 256, 0, s>>>(etc, n, T, fs, scale, decay_depth, clarity_s, o);
    }
    return cudaGetLastError();
}

}  // namespace pach
