// filters_ntt.cu -- receiver filters in integer arithmetic: the convolutions of ETCToFilter (see
// filters.cu) by number-theoretic transforms.
//
// GB300 issues two FP64 lanes per SM and cycle against 64 integer ones, and the FP64 transforms of
// filters.cu keep that pipe 85 % busy.  Here envelopes and carriers are rounded once to integers of 60 to
// 62 bits (a common power of two per filter; one per carrier, taken off the envelopes of its band), the sum of
// the nine convolutions is formed exactly modulo five primes near 2^27, and the Chinese remainder theorem
// gives the exact integer sum.  Every carrier's L1 norm is 2 / 16384, which bounds the sum below half the
// primes' product at those widths whatever the length (k_ntt_scale).  So the rounding of the inputs is the
// only error: 2^-62 of a carrier's peak and of the largest envelope value at 1 kHz.  (Four primes near 2^30
// leave 55 bits each, which the 16384 small samples of a carrier turn into 2e-15 of the output, five times the
// floating-point transforms' error.)
//
// A transform of length W = R x 4096 of a shorter input splits into R residue classes of frequencies:
//   X[R k + r] = sum_t' z_r[t'] w_4096^(k t'),  z_r[t'] = w_W^(r t') sum_j x[t' + 4096 j] w_R^(r j),
// R independent 4096-point transforms that one CTA each does in registers (three passes of radix 16, two
// exchanges through shared memory).  The CTA of a (filter, prime, class) transforms the nine envelopes one
// after another, adds their products with the carriers' spectra, and transforms back:
//   out[t' + 4096 j] = 1 / W sum_r w_R^(-r j) (w_W^(-r t') y_r[t']),
// the last sum being R-point transforms that k_ntt_out does together with the remaindering.
// Multiplications by known factors carry the factor's quotient (Shoup): q = hi(x w'), x w - q p in [0, 2p) for
// any 32-bit x (Harvey, "Faster arithmetic for number-theoretic transforms", 2014).  With p < 2^27 the sums of a
// 16-point transform of such values stay below 32 p < 2^32, so nothing is reduced between the multiplications:
// an addition, a subtraction and at most one multiplication a butterfly (two of the seven instructions of a
// butterfly that keeps its sums below 2p, for one more prime).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>

#include "filters.h"

namespace pach {
namespace {

typedef unsigned u32;
typedef unsigned long long u64;

constexpr int kN = 4096;             // points per class
constexpr int kPrimes = 5;
constexpr int kRow = 272;            // exchange buffers: 16 rows of 256 (+16: no bank conflicts)
constexpr u32 kP[kPrimes] = {132710401u, 132120577u, 131923969u, 131530753u, 130809857u};  // 1 mod 2^16
constexpr u32 kG[kPrimes] = {7u, 5u, 13u, 5u, 3u};  // primitive roots
constexpr double kLog2M = 134.869;   // of the primes' product (rounded down)
constexpr size_t kChunkBytes = size_t(96) << 20;  // per-filter buffers at a time: within L2

// A constant factor with its quotient: x = w, y = floor(w 2^32 / p).
typedef uint2 Fac;

struct Prime {
    u32 p, np;                  // np = -p: products with it are added
    u32 one;                    // floor(2^32 / p)
    u64 inv;                    // floor(2^64 / p)
    Fac c32;                    // 2^32 mod p
    Fac iR[8];                  // w_R^-i, i < R / 2
};

struct Tables {                 // kernel argument
    Prime P[kPrimes];
    int W, R;
};

// Powers of w_W: hi[m >> 8], lo[m & 255] (host-made, 10 KB of kernel argument).
struct Powers {
    u32 hi[kPrimes][256], lo[kPrimes][256];
};

struct Bufs {
    Fac *twA, *itwA;            // [prime][class][k1][u]: w_W^+-(u (r + R k1))
    Fac *twB, *itwB;            // [prime][k2][v]: w_256^+-(v k2)
    Fac *pre, *post;            // [prime][class][16 R]: w_W^(256 r m); [prime][class][16]: w_W^-(256 r i) / W
    Fac *spec;                  // [prime][class][band][4096]: the carriers' spectra
    double *car, *part, *att;   // [9][16384], [9][64][2] partial L1 sums and maxima, [T]
    double *norm;               // [9] the carriers' normalisations
    int *ec;                    // [9] the carriers' exponents, then the bits of carriers and envelopes
    u32 *cres;                  // [prime][9][16384]
    double *env;                // [job][9][T]
    int *ef;                    // [job] the envelopes' largest exponent + kExpBias (0: no energy)
    u32 *res;                   // [job][prime][9][T]
    u32 *y;                     // [job][prime][class][4096]
};
constexpr int kExpBias = 1 << 16, kExpNan = 1 << 20;

constexpr u32 mulmod_h(u32 a, u32 b, u32 p) { return (u32)((u64)a * b % p); }
constexpr u32 powmod_h(u32 a, u64 e, u32 p) {
    u32 r = 1;
    for (; e; e >>= 1, a = mulmod_h(a, a, p))
        if (e & 1) r = mulmod_h(r, a, p);
    return r;
}
Fac fac_h(u32 w, u32 p) { return make_uint2(w, (u32)(((u64)w << 32) / p)); }

// Prime K and its 16th roots as immediates of the class kernels (read from constant memory they cost a
// quarter more instructions): w_16^I, or its inverse.
template <int K>
struct PC {
    static constexpr u32 p = kP[K], np = 0u - kP[K], one = (u32)((1ull << 32) / kP[K]);
};
template <int K, bool INV, int I>
struct W16 {
    static constexpr u32 x = powmod_h(powmod_h(kG[K], (kP[K] - 1) / 16, kP[K]), INV ? 16 - I : I, kP[K]);
    static constexpr u32 y = (u32)(((u64)x << 32) / kP[K]);
};
template <int K, bool INV>
__device__ __forceinline__ Fac w16(int i) {  // i known once the loops around it are unrolled
    switch (i) {
        case 1: return make_uint2(W16<K, INV, 1>::x, W16<K, INV, 1>::y);
        case 2: return make_uint2(W16<K, INV, 2>::x, W16<K, INV, 2>::y);
        case 3: return make_uint2(W16<K, INV, 3>::x, W16<K, INV, 3>::y);
        case 4: return make_uint2(W16<K, INV, 4>::x, W16<K, INV, 4>::y);
        case 5: return make_uint2(W16<K, INV, 5>::x, W16<K, INV, 5>::y);
        case 6: return make_uint2(W16<K, INV, 6>::x, W16<K, INV, 6>::y);
        default: return make_uint2(W16<K, INV, 7>::x, W16<K, INV, 7>::y);
    }
}

// w < p with its quotient, from the 64-bit reciprocal (one too small at most).
__device__ __forceinline__ Fac fac_d(u32 w, const Prime &P) {
    u32 q = (u32)((w * P.inv) >> 32);
    q += ((u64)w << 32) - (u64)q * P.p >= P.p;
    return make_uint2(w, q);
}
__device__ __forceinline__ u32 shoup(u32 x, Fac w, u32 np) { return x * w.x + __umulhi(x, w.y) * np; }

// v modulo p, in [0, 2p), for any 32-bit v.
__device__ __forceinline__ u32 reduce(u32 v, const Prime &P) { return v + __umulhi(v, P.one) * P.np; }
template <int K>
__device__ __forceinline__ u32 reduce(u32 v) { return v + __umulhi(v, PC<K>::one) * PC<K>::np; }

// 16-point transform (INV: with inverse roots) in registers: input natural, values in [0, 2p); output index bit-reversed, in [0, 32p).
__device__ __forceinline__ constexpr int br4(int i) { return ((i & 1) << 3) | ((i & 2) << 1) | ((i & 4) >> 1) | (i >> 3); }
template <int K, bool INV>
__device__ __forceinline__ void dft16(u32 (&x)[16]) {
#pragma unroll
    for (int h = 8; h >= 1; h >>= 1) {
        const u32 below = PC<K>::p * (u32)(16 / h);  // this stage's inputs are below it: 2p, 4p, 8p, 16p
#pragma unroll
        for (int g = 0; g < 16; g += 2 * h)
#pragma unroll
            for (int j = 0; j < h; ++j) {
                const u32 a = x[g + j], b = x[g + j + h], d = a - b + below;
                x[g + j] = a + b;
                x[g + j + h] = j == 0 ? d : shoup(d, w16<K, INV>(j * (8 / h)), PC<K>::np);
            }
    }
}

// 4096-point transform of the CTA's 256 threads: thread u starts with z[u + 256 i] in x[i] and ends, as
// (k1, k2) = (u >> 4, u & 15), with X[k1 + 16 k2 + 256 br4(i)] in [0, 32p).  twA includes the class's factor
// w_W^(r u).  The second exchange stays within a row of the buffer, which one half-warp reads and writes, so only
// the first needs the CTA's barrier; the caller's next write into buf needs another.
template <int K>
__device__ __forceinline__ void ntt4096(u32 (&x)[16], const Fac *s_twA, const Fac *s_twB, u32 *buf) {
    const int u = threadIdx.x, b = u & 15;
    u32 *row = buf + (u >> 4) * kRow;
    dft16<K, false>(x);
#pragma unroll
    for (int i = 0; i < 16; ++i) buf[br4(i) * kRow + u] = shoup(x[i], s_twA[br4(i) * 256 + u], PC<K>::np);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = row[b + 16 * i];
    dft16<K, false>(x);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 16; ++i) row[br4(i) * 17 + b] = shoup(x[i], s_twB[br4(i) * 16 + b], PC<K>::np);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = row[b * 17 + i];
    dft16<K, false>(x);
}

// Shared memory of a class CTA.
struct ClassSmem {
    Fac twA[16 * 256], twB[256], pre[256];
    u32 buf[16 * kRow];
};

__device__ __forceinline__ void load_class(ClassSmem &s, const Bufs &B, const Tables &t, int prime, int cls) {
    const size_t pc = (size_t)prime * t.R + cls;
    for (int i = threadIdx.x; i < 16 * 256; i += 256) s.twA[i] = B.twA[pc * 4096 + i];
    s.twB[threadIdx.x] = B.twB[prime * 256 + threadIdx.x];
    if ((int)threadIdx.x < 16 * t.R) s.pre[threadIdx.x] = B.pre[pc * 16 * t.R + threadIdx.x];
}

// z_r of T residues src (w_W^(r u) left to twA): x[i] = sum_j src[u + 256 (i + 16 j)] w_W^(256 r (i + 16 j)).
template <int K>
__device__ __forceinline__ void load_folded(u32 (&x)[16], const u32 *src, int T, const Fac *s_pre) {
    const int u = threadIdx.x;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int t = u + 256 * i;
        x[i] = t < T ? shoup(__ldg(src + t), s_pre[i], PC<K>::np) : 0u;
    }
    for (int j = 1; j * kN < T; ++j)
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int t = u + 256 * i + kN * j;
            if (t < T) x[i] = reduce<K>(x[i] + shoup(__ldg(src + t), s_pre[i + 16 * j], PC<K>::np));
        }
}

// ------------------------------------------------------------------------------------------ tables
// grid (W / 256 + 1, prime): the last block of a prime makes twB.
__global__ void __launch_bounds__(256) k_ntt_tables(__grid_constant__ const Powers pw, __grid_constant__ const Tables t,
                                                    Bufs B) {
    __shared__ u32 hi[256], lo[256];
    const int prime = blockIdx.y, tid = threadIdx.x;
    const Prime &P = t.P[prime];
    hi[tid] = pw.hi[prime][tid];
    lo[tid] = pw.lo[prime][tid];
    __syncthreads();
    auto mul = [&](u32 a, u32 b) {
        const u32 v = shoup(a, fac_d(b, P), P.np);
        return min(v, v - P.p);
    };
    auto power = [&](u32 m) { return mul(hi[(m & (t.W - 1)) >> 8], lo[m & 255]); };
    auto root = [&](u32 m) { return fac_d(power(m), P); };
    if ((int)blockIdx.x == t.W / 256) {
        const u32 e = (u32)(tid >> 4) * (tid & 15) * (t.W / 256);
        B.twB[prime * 256 + tid] = root(e);
        B.itwB[prime * 256 + tid] = root(t.W - e % t.W);
        return;
    }
    // block = (class, k1): 16 blocks a class
    const int cls = blockIdx.x >> 4, k1 = blockIdx.x & 15;
    const u32 e = (u32)tid * (u32)(cls + t.R * k1);
    const size_t at = ((size_t)prime * t.R + cls) * 4096 + k1 * 256 + tid;
    B.twA[at] = root(e);
    B.itwA[at] = root(t.W - e % t.W);
    if (k1 == 0) {
        if (tid < 16 * t.R) B.pre[((size_t)prime * t.R + cls) * 16 * t.R + tid] = root(256u * cls * tid);
        if (tid < 16) {
            // 1 / W = p - (p - 1) / W
            const u32 w = mul(power(t.W - (256u * cls * tid) % t.W), P.p - (P.p - 1) / t.W);
            B.post[((size_t)prime * t.R + cls) * 16 + tid] = fac_d(w, P);
        }
    }
}

// The carriers before their normalisation (GenerateBandLimitedSincPulse, the reference's expressions), whose
// second half mirrors the first, with the L1 sums by block: grid (64, 9).  Row 9 of the grid: the 16 kHz ramp.
__global__ void __launch_bounds__(128) k_ntt_carriers(Bufs B, int fs, int T, double add) {
    __shared__ double red[8];
    const int b = blockIdx.y, tid = threadIdx.x;
    if (b == 9) {
        for (int t = blockIdx.x * 128 + tid; t < T; t += gridDim.x * 128) {
            const double dist = (double)t * (1.0 / (double)fs) * 343.0;
            B.att[t] = pow(10.0, -add * dist / 20.0);
        }
        return;
    }
    const double rt2 = sqrt(2.0);
    const double fcb = b < 8 ? 62.5 * pow(2.0, (double)b) : 16000.0;
    const double fl = fcb / rt2, fu = fcb * rt2;
    const double fc = (fl + fu) / 2.0, bw = fu - fl, t0 = (kCarrierLen - 1) / 2.0;
    const double pi = 3.141592653589793;
    const int n = blockIdx.x * 128 + tid;  // < 8192
    const double t = ((double)n - t0) / (double)fs;
    const double sinc = bw == 0.0 ? 1.0 : sin(pi * bw * t) / (pi * bw * t);
    const double v = sinc * cos(2.0 * pi * fc * t);
    B.car[(size_t)b * kCarrierLen + n] = v;
    B.car[(size_t)b * kCarrierLen + kCarrierLen - 1 - n] = v;
    double part = fabs(v), top = part;
    for (int o = 16; o; o >>= 1) {
        part += __shfl_xor_sync(0xffffffffu, part, o);
        top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
    }
    if ((tid & 31) == 0) {
        red[tid >> 5] = part;
        red[4 + (tid >> 5)] = top;
    }
    __syncthreads();
    if (tid == 0) {
        B.part[2 * (b * 64 + blockIdx.x)] = red[0] + red[1] + red[2] + red[3];
        B.part[2 * (b * 64 + blockIdx.x) + 1] = fmax(fmax(red[4], red[5]), fmax(red[6], red[7]));
    }
}

// m 2^e = x for finite x (m the signed mantissa; denormals keep their exponent).
__device__ __forceinline__ long long mantissa(double x, int &e) {
    const long long bits = __double_as_longlong(x);
    const int f = (int)((bits >> 52) & 0x7FF);
    long long m = bits & 0xFFFFFFFFFFFFFll;
    if (f) m |= 1ll << 52;
    e = (f ? f : 1) - 1075;
    return bits < 0 ? -m : m;
}

// Normalisations, exponents (carrier b below 2^ec) and widths: with carriers of bc bits and envelopes of be
// bits the sum of products stays below sum_b 2^be (2^-13 2^(bc - ec_b)), as each carrier's L1 norm is 2^-13;
// bc + be is the most that keeps this below half the primes' product.  9 warps.
__global__ void __launch_bounds__(288) k_ntt_scale(Bufs B) {
    __shared__ double s_w[9];
    const int b = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double *part = B.part + 2 * b * 64;
    double l1 = part[2 * lane] + part[2 * lane + 64];
    double top = fmax(part[2 * lane + 1], part[2 * lane + 65]);
    for (int o = 16; o; o >>= 1) {
        l1 += __shfl_xor_sync(0xffffffffu, l1, o);
        top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
    }
    if (lane == 0) {
        double norm = 2.0 / (2.0 * l1 * (double)kCarrierLen);  // the parts hold half of a symmetric sum
        if (!(norm > 0.0)) norm = 1.0;
        int e;
        mantissa(top * norm, e);
        B.norm[b] = norm;
        B.ec[b] = e + 53;
        s_w[b] = scalbn(1.0, -(e + 53) - 13);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double w = 0.0;
        for (int k = 0; k < 9; ++k) w += s_w[k];
        // 2^-10: the rounding of 16384 samples and of the norms
        const int total = (int)floor(kLog2M - 1.0 - log2(w) - 0x1p-10);
        B.ec[9] = min(62, (total + 1) / 2);
        B.ec[10] = min(62, total - B.ec[9]);
    }
}

// |m| 2^s rounded to an integer, s <= 0 for every value that is not a rounding too large; zero when too small.
__device__ __forceinline__ u64 shift_round(u64 m, int s) {
    if (s >= 0) return m << s;
    s = -s;
    if (s > 54) return 0;
    return (m + (1ull << (s - 1))) >> s;
}

// v modulo p, in [0, 4p).
__device__ __forceinline__ u32 residue(u64 v, const Prime &P) {
    return shoup((u32)(v >> 32), P.c32, P.np) + reduce((u32)v, P);
}

// Normalised carriers as integers below 2^bc, modulo the primes: grid (64, 9).
__global__ void __launch_bounds__(256) k_ntt_carrier_res(__grid_constant__ const Tables t, Bufs B) {
    const int b = blockIdx.y, n = blockIdx.x * 256 + threadIdx.x;
    int e;
    const long long m = mantissa(B.car[(size_t)b * kCarrierLen + n] * B.norm[b], e);
    const u64 q = shift_round((u64)(m < 0 ? -m : m), e + B.ec[9] - B.ec[b]);
    for (int k = 0; k < kPrimes; ++k) {
        const Prime &P = t.P[k];
        const u32 r = residue(q, P);
        B.cres[((size_t)k * 9 + b) * kCarrierLen + n] = m < 0 ? 4 * P.p - r : r;
    }
}

// Spectrum of a carrier's class: grid (class, band, prime).
template <int K>
__device__ void carrier_spectrum(const Tables &t, const Bufs &B, int cls, int band) {
    extern __shared__ unsigned char smem[];
    ClassSmem &s = *reinterpret_cast<ClassSmem *>(smem);
    const Prime &P = t.P[K];
    load_class(s, B, t, K, cls);
    __syncthreads();
    u32 x[16];
    load_folded<K>(x, B.cres + ((size_t)K * 9 + band) * kCarrierLen, kCarrierLen, s.pre);
    ntt4096<K>(x, s.twA, s.twB, s.buf);
    Fac *dst = B.spec + (((size_t)K * t.R + cls) * 9 + band) * kN + threadIdx.x;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const u32 v = reduce<K>(x[i]);
        dst[i * 256] = fac_d(min(v, v - P.p), P);
    }
}

#define PACH_BY_PRIME(call)        \
    switch (blockIdx.z) {          \
        case 0: call(0); break;    \
        case 1: call(1); break;    \
        case 2: call(2); break;    \
        case 3: call(3); break;    \
        default: call(4); break;   \
    }

__global__ void __launch_bounds__(256) k_ntt_spec(__grid_constant__ const Tables t, Bufs B) {
#define PACH_CALL(K) carrier_spectrum<K>(t, B, blockIdx.x, blockIdx.y)
    PACH_BY_PRIME(PACH_CALL)
#undef PACH_CALL
}

// ------------------------------------------------------------------------------------------ per filter
// Envelopes of the chunk's filters (envelope() of filters.cu; a receiver's directional kinds share one
// division, P Dir / E = (P / E) Dir) and their largest exponents: grid (T / 256, receivers of the chunk x 8).
template <int KINDS>
__global__ void __launch_bounds__(256) k_ntt_env(FilterJob J, Bufs B, int nj) {
    __shared__ int s_top[KINDS];
    const int lane = threadIdx.x & 31;
    const int r = J.job0 / KINDS + blockIdx.y / 8, b = blockIdx.y & 7;
    const int t = blockIdx.x * 256 + threadIdx.x;
    const bool in = t < J.T;
    const size_t i = ((size_t)r * 8 + b) * J.T + t;
    if ((int)threadIdx.x < KINDS) s_top[threadIdx.x] = 0;
    const double p = in ? J.P[i] : 0.0, e = KINDS > 1 && in ? J.E[i] : 0.0;
    double D[KINDS];
#pragma unroll
    for (int kind = 1; kind < KINDS; ++kind)
        D[kind] = in ? ((kind & 1) ? J.Dn : J.Dp)[(((size_t)r * 3 + ((kind - 1) >> 1)) * 8 + b) * J.T + t] : 0.0;
    // factors of the band: P's, and P / E's for the directions (0 where E = 0)
    const double f = J.scale ? J.pmod[b] * J.scale[r] : J.pmod[b];
    const double q = e == 0.0 ? 0.0 : p / e * f;
    // P / E out of range or subnormal: P Dir / E may not be
    const int qh = __double2hiint(fabs(q));
    const bool direct = qh >= 0x7FF00000 || (qh < 0x00100000 && p != 0.0 && e != 0.0);
    const double pf = p * f, att = in && b == 7 ? B.att[t] : 0.0;
    const int ec = B.ec[b] + kExpBias, ec8 = B.ec[8] + kExpBias;
    // exponent of a value: v 2^ec < 2^(top - kExpBias)
    auto top_of = [](double v, int ec_) {
        if (__double_as_longlong(v) == 0) return 0;
        if (__double2hiint(v) >= 0x7FF00000) return kExpNan;
        int ex;
        const u64 m = (u64)mantissa(v, ex);
        return ex + 64 - __clzll((long long)m) + ec_;
    };
    __syncthreads();
#pragma unroll
    for (int kind = 0; kind < KINDS; ++kind) {
        const int job = r * KINDS + kind - J.job0;
        if (job < 0 || job >= nj) continue;
        double v = fabs(kind == 0 ? pf : (direct ? p * D[kind] / e * f : q * D[kind]));
        double *dst = B.env + ((size_t)job * 9 + b) * J.T + t;
        if (in) *dst = v;
        int x = top_of(v, ec);
        if (b == 7) {
            v *= att;
            if (in) dst[J.T] = v;
            x = max(x, top_of(v, ec8));
        }
        x = __reduce_max_sync(0xffffffffu, x);
        if (lane == 0) atomicMax(s_top + kind, x);
    }
    __syncthreads();
    if ((int)threadIdx.x < KINDS) {
        const int job = r * KINDS + threadIdx.x - J.job0;
        if (job >= 0 && job < nj && s_top[threadIdx.x]) atomicMax(B.ef + job, s_top[threadIdx.x]);
    }
}

// Envelopes as integers: v 2^(ec - Ef + be) with v 2^ec < 2^Ef, modulo the primes: grid (9 T / 256, job).
__global__ void __launch_bounds__(256) k_ntt_env_res(__grid_constant__ const Tables t, Bufs B, int T) {
    const int job = blockIdx.y, i = blockIdx.x * 256 + threadIdx.x;
    if (i >= 9 * T) return;
    const int ef = B.ef[job];
    u64 q = 0;
    const double v = B.env[(size_t)job * 9 * T + i];
    if (ef && ef < kExpNan) {
        int e;
        const u64 m = (u64)mantissa(v, e);
        q = shift_round(m, e + B.ec[i / T] + B.ec[10] - (ef - kExpBias));
    }
    u32 *dst = B.res + (size_t)job * kPrimes * 9 * T + i;
#pragma unroll
    for (int k = 0; k < kPrimes; ++k) dst[(size_t)k * 9 * T] = residue(q, t.P[k]);
}

// One class of one prime of one filter: nine transforms, their products with the carriers, the transform back.
// Bound: integer issue (56 % of slots, 45 instructions a point and transform), shared memory and the waits for
// residues and spectra near it; four CTAs an SM (64 registers, 54 KB).  4.3 us a filter of 32768 points, where the
// FP64 transforms take 25 us with their pipe 85 % busy.  With the factors read from constant memory 4.6 us.
template <int K>
__device__ __forceinline__ void filter_class(const Tables &t, const Bufs &B, int T, int cls, int job) {
    extern __shared__ unsigned char smem[];
    ClassSmem &s = *reinterpret_cast<ClassSmem *>(smem);
    constexpr u32 np = PC<K>::np;
    const int u = threadIdx.x, a = u >> 4, b = u & 15;
    load_class(s, B, t, K, cls);
    const size_t pc = (size_t)K * t.R + cls;
    const u32 *src = B.res + ((size_t)job * kPrimes + K) * 9 * T;
    const Fac *spec = B.spec + pc * 9 * kN + u;
    u32 acc[16];  // nine values below 2p
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] = 0;
    for (int band = 0; band < 9; ++band) {
        u32 x[16];
        __syncthreads();  // the tables are there, and the last transform has read the buffer
        load_folded<K>(x, src + (size_t)band * T, T, s.pre);
        ntt4096<K>(x, s.twA, s.twB, s.buf);
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] += shoup(x[i], __ldg(spec + (size_t)band * kN + i * 256), np);
    }
    // back: over k3, k2, k1
    u32 x[16], *row = s.buf + a * kRow;
#pragma unroll
    for (int i = 0; i < 16; ++i) x[br4(i)] = reduce<K>(acc[i]);
    dft16<K, true>(x);
    const Fac *itwB = B.itwB + K * 256;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 16; ++i) row[b * 17 + br4(i)] = shoup(x[i], __ldg(itwB + b * 16 + br4(i)), np);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = row[i * 17 + b];
    dft16<K, true>(x);
    const Fac *itwA = B.itwA + pc * 4096 + a * 256 + b;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 16; ++i) row[b + 16 * br4(i)] = shoup(x[i], __ldg(itwA + 16 * br4(i)), np);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = s.buf[i * kRow + u];
    dft16<K, true>(x);
    u32 *y = B.y + (((size_t)job * kPrimes + K) * t.R + cls) * kN + u;
    const Fac *post = B.post + pc * 16;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const u32 v = shoup(x[i], __ldg(post + br4(i)), np);
        y[256 * br4(i)] = min(v, v - PC<K>::p);
    }
}

// grid (class, job, prime): blocks of one prime run together, as each prime has its own code.
__global__ void __launch_bounds__(256, 4) k_ntt_class(__grid_constant__ const Tables t, Bufs B, int T) {
#define PACH_CALL(K) filter_class<K>(t, B, T, blockIdx.x, blockIdx.y)
    PACH_BY_PRIME(PACH_CALL)
#undef PACH_CALL
}
#undef PACH_BY_PRIME

// Garner constants: inverses of earlier primes modulo later ones, and the primes' products.
struct Garner {
    Fac inv[kPrimes][kPrimes];  // inv[i][k] = p_i^-1 mod p_k, i < k
    u64 m1;                     // p0 p1
    u64 m2_lo, m2_hi;           // p0 p1 p2
    double m3;                  // p0 p1 p2 p3
};

// R-point transforms over the classes, remaindering, scaling: grid (4096 / 128, job).
template <int R>
__global__ void __launch_bounds__(128) k_ntt_out(__grid_constant__ const Tables t, __grid_constant__ const Garner G, Bufs B,
                                                 const double *scale, int kinds, double *out, int L, int job0) {
    const int tp = blockIdx.x * 128 + threadIdx.x, job = blockIdx.y;
    u32 x[kPrimes][R];
#pragma unroll
    for (int k = 0; k < kPrimes; ++k) {
        const u32 *y = B.y + ((size_t)job * kPrimes + k) * R * kN + tp;
#pragma unroll
        for (int r = 0; r < R; ++r) x[k][r] = y[(size_t)r * kN];
        const Prime &P = t.P[k];
        u32 below = P.p;  // the inputs are below p, the outputs below R p
#pragma unroll
        for (int h = R / 2; h >= 1; h >>= 1, below <<= 1)
#pragma unroll
            for (int g = 0; g < R; g += 2 * h)
#pragma unroll
                for (int j = 0; j < h; ++j) {
                    const u32 a = x[k][g + j], b = x[k][g + j + h], d = a - b + below;
                    x[k][g + j] = a + b;
                    x[k][g + j + h] = j == 0 ? d : shoup(d, P.iR[j * (R / 2 / h)], P.np);
                }
    }
    const int ef = B.ef[job];
    const int sh = ef - kExpBias - B.ec[9] - B.ec[10];
    double *o = out + (size_t)(job0 + job) * L;
    // the envelopes are magnitudes: a receiver's factor below zero turns its filters here
    const bool turn = scale && scale[(job0 + job) / kinds] < 0.0;
#pragma unroll
    for (int q = 0; q < R; ++q) {
        int j = 0;  // q bit-reversed
#pragma unroll
        for (int v = 1, w = R / 2; v < R; v <<= 1, w >>= 1) j |= (q & v) ? w : 0;
        const int n = tp + kN * j;
        if (n >= L) continue;
        // Garner: value = v0 + v1 p0 + v2 p0 p1 + v3 p0 p1 p2 + v4 p0 p1 p2 p3; a value in the upper half of the
        // primes' product (by its last digit: the sum is bounded away from the middle) is negative, and the
        // digits' complements plus one are its magnitude
        u32 v[kPrimes];
#pragma unroll
        for (int k = 0; k < kPrimes; ++k) {
            const u32 p = t.P[k].p;
            u32 c = reduce(x[k][q], t.P[k]);
#pragma unroll
            for (int i = 0; i < k; ++i) c = shoup(c + 2 * p - v[i], G.inv[i][k], t.P[k].np);  // (c - v_i) / p_i; v_i < 2p
            v[k] = min(c, c - p);
        }
        const bool neg = v[4] > t.P[4].p / 2;
        if (neg) {
#pragma unroll
            for (int k = 0; k < kPrimes; ++k) v[k] = t.P[k].p - 1 - v[k];
            ++v[0];
        }
        u64 lo = (u64)v[0] + (u64)v[1] * t.P[0].p, hi = 0;
        {
            const u64 a = (u64)v[2] * (G.m1 & 0xFFFFFFFFull), c = (u64)v[2] * (G.m1 >> 32);
            const u64 pl = a + (c << 32);
            hi += (c >> 32) + (pl < a);
            lo += pl;
            hi += lo < pl;
        }
        {
            const u64 a = (u64)v[3] * (G.m2_lo & 0xFFFFFFFFull), c = (u64)v[3] * (G.m2_lo >> 32);
            const u64 pl = a + (c << 32);
            hi += (c >> 32) + (pl < a) + (u64)v[3] * G.m2_hi;
            lo += pl;
            hi += lo < pl;
        }
        double d = fma((double)v[4], G.m3, (double)hi * 18446744073709551616.0 + (double)lo);
        d = neg != turn ? -d : d;
        o[n] = ef >= kExpNan ? __longlong_as_double(0x7FF8000000000000ll) : (ef == 0 ? 0.0 : scalbn(d, sh));
    }
}

size_t align_up(size_t x) { return (x + 255) & ~size_t(255); }

int transform_len(int T) {
    int W = 16384;
    while (W < T + kCarrierLen - 1) W <<= 1;
    return W;
}

template <class F>
size_t lay(char *base, size_t &off, F *&p, size_t n) {
    p = reinterpret_cast<F *>(base + off);
    off += align_up(n * sizeof(F));
    return off;
}

size_t fixed_layout(char *base, Bufs &B, int T, int W) {
    const size_t R = (size_t)W / kN;
    size_t off = 0;
    lay(base, off, B.twA, (size_t)kPrimes * W);
    lay(base, off, B.itwA, (size_t)kPrimes * W);
    lay(base, off, B.twB, (size_t)kPrimes * 256);
    lay(base, off, B.itwB, (size_t)kPrimes * 256);
    lay(base, off, B.pre, (size_t)kPrimes * R * 16 * R);
    lay(base, off, B.post, (size_t)kPrimes * R * 16);
    lay(base, off, B.spec, (size_t)kPrimes * 9 * W);
    lay(base, off, B.car, (size_t)9 * kCarrierLen);
    lay(base, off, B.part, (size_t)9 * 64 * 2);
    lay(base, off, B.norm, (size_t)9);
    lay(base, off, B.att, (size_t)T);
    lay(base, off, B.ec, (size_t)11);
    lay(base, off, B.cres, (size_t)kPrimes * 9 * kCarrierLen);
    return off;
}

// Filters at a time, however much workspace there is: their buffers stay within L2, and k_ntt_env's grid (eight rows a
// receiver) within 65535.
size_t chunk_max(size_t job) { return std::max<size_t>(1, std::min<size_t>(kChunkBytes / job, 65535 / 8 - 1)); }

size_t job_bytes(int T, int W) {
    return align_up((size_t)9 * T * 8 + (size_t)kPrimes * 9 * T * 4 + (size_t)kPrimes * W * 4 + 4) + 1024;
}

}  // namespace

bool ntt_supported(int T) { return T + kCarrierLen - 1 <= 65536; }

size_t ntt_workspace_bytes(int n_filters, int T) {
    Bufs B{};
    const int W = transform_len(T);
    const size_t pj = job_bytes(T, W);
    return fixed_layout(nullptr, B, T, W) + std::min<size_t>((size_t)n_filters, chunk_max(pj)) * pj;
}

cudaError_t ntt_filters(FilterJob J, int n, int fs, double add, int L, double *out, void *ws, size_t ws_bytes,
                        cudaStream_t st) {
    const int T = J.T, W = transform_len(T), R = W / kN;
    Bufs B{};
    char *base = static_cast<char *>(ws);
    size_t off = fixed_layout(base, B, T, W);
    const size_t pj = job_bytes(T, W);
    const int chunk = (int)std::min<size_t>(std::min<size_t>((size_t)n, (ws_bytes - off) / pj), chunk_max(pj));
    lay(base, off, B.env, (size_t)chunk * 9 * T);
    lay(base, off, B.res, (size_t)chunk * kPrimes * 9 * T);
    lay(base, off, B.y, (size_t)chunk * kPrimes * W);
    lay(base, off, B.ef, (size_t)chunk);

    Tables t{};
    Powers pw;
    Garner G{};
    t.W = W;
    t.R = R;
    for (int k = 0; k < kPrimes; ++k) {
        const u32 p = kP[k];
        Prime &P = t.P[k];
        P.p = p;
        P.np = 0u - p;
        P.inv = ~0ull / p;  // p does not divide 2^64
        P.one = (u32)((1ull << 32) / p);
        P.c32 = fac_h((u32)((1ull << 32) % p), p);
        const u32 w = powmod_h(kG[k], (p - 1) / W, p);
        const u32 wR = powmod_h(w, W / R, p);
        for (int i = 0; i < 8; ++i) {
            P.iR[i] = fac_h(powmod_h(wR, 2 * R - i, p), p);
        }
        const u32 w256 = powmod_h(w, 256, p);
        u32 a = 1, b = 1;
        for (int i = 0; i < 256; ++i) {
            pw.lo[k][i] = a;
            pw.hi[k][i] = b;
            a = mulmod_h(a, w, p);
            b = mulmod_h(b, w256, p);
        }
        for (int i = 0; i < k; ++i) G.inv[i][k] = fac_h(powmod_h(kP[i] % p, p - 2, p), p);
    }
    {
        typedef unsigned __int128 u128;
        const u128 m1 = (u128)kP[0] * kP[1], m2 = m1 * kP[2], m3 = m2 * kP[3];
        G.m1 = (u64)m1;
        G.m2_lo = (u64)m2;
        G.m2_hi = (u64)(m2 >> 64);
        G.m3 = (double)m3;
    }
    const size_t smem = sizeof(ClassSmem);
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(k_ntt_spec, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(k_ntt_class, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess)
        return e;
    k_ntt_carriers<<<dim3(64, 10), 128, 0, st>>>(B, fs, T, add);
    k_ntt_tables<<<dim3(W / 256 + 1, kPrimes), 256, 0, st>>>(pw, t, B);
    k_ntt_scale<<<1, 288, 0, st>>>(B);
    k_ntt_carrier_res<<<dim3(64, 9), 256, 0, st>>>(t, B);
    k_ntt_spec<<<dim3(R, 9, kPrimes), 256, smem, st>>>(t, B);
    for (int j0 = 0; j0 < n; j0 += chunk) {
        const int nj = std::min(chunk, n - j0);
        J.job0 = j0;
        const int r0 = j0 / J.kinds, r1 = (j0 + nj - 1) / J.kinds;
        if ((e = cudaMemsetAsync(B.ef, 0, (size_t)nj * sizeof(int), st)) != cudaSuccess) return e;
        FilterJob Q = J;
        Q.att = B.att;
        const dim3 eg((T + 255) / 256, (r1 - r0 + 1) * 8);
        if (J.kinds == 1) k_ntt_env<1><<<eg, 256, 0, st>>>(Q, B, nj);
        else k_ntt_env<7><<<eg, 256, 0, st>>>(Q, B, nj);
        k_ntt_env_res<<<dim3((9 * T + 255) / 256, nj), 256, 0, st>>>(t, B, T);
        k_ntt_class<<<dim3(R, nj, kPrimes), 256, smem, st>>>(t, B, T);
        const dim3 grid(kN / 128, nj);
        if (R == 4) k_ntt_out<4><<<grid, 128, 0, st>>>(t, G, B, J.scale, J.kinds, out, L, j0);
        else if (R == 8) k_ntt_out<8><<<grid, 128, 0, st>>>(t, G, B, J.scale, J.kinds, out, L, j0);
        else k_ntt_out<16><<<grid, 128, 0, st>>>(t, G, B, J.scale, J.kinds, out, L, j0);
    }
    return cudaGetLastError();
}

}  // namespace pach
