// Floating-point arithmetic on 64-bit integer mantissas.
//
// On this GPU an FP64 instruction holds an SM sub-partition's FP64 unit for
// 64 to 76 clocks (1.68 lane operations per SM and clock), while the integer
// pipes issue a warp instruction every one to two clocks (64 to 122 lane
// operations per SM and clock).  A floating-point multiply-add written in
// about fifteen integer instructions is therefore several times cheaper than
// one DFMA, and runs beside the FP64 unit.  The right-hand side uses it for
// its stencils, where sums of neighbours with small integer weights are exact
// in 64-bit integers.
//
// A number is m * 2^e with a signed 64-bit mantissa, normalised to
// 2^61 <= |m| < 2^62 (the unnormalised rest of a cancellation and zero have a
// smaller |m|).  Multiplication and addition are the schoolbook algorithms on
// mantissas and exponents.  A product of normalised numbers is cut, not
// rounded, at 2.25 * 2^-58 of its value, a sum at 2^-58 of its largest term:
// both are nearer to the exact result than a correctly rounded FP64 operation
// (2^-53) can be relied on to be.  What is left of a cancellation of more than
// 30 bits is moved up by 29, so a product of it is cut at 2^-86 of what the
// product of the terms before the cancellation would have been.
//
// Results below the normal range are subnormal, results above it infinite;
// a NaN or an infinity among the inputs makes the result NaN.
#pragma once
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define OLLIN_HD __host__ __device__ __forceinline__
#else
#define OLLIN_HD inline
#endif

namespace ollin {

// arithmetic shift right by any count (more than 63 leaves the sign)
OLLIN_HD long long sf_shr(long long m, int n) {
#if defined(__CUDA_ARCH__)
    long long r;
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(m), "r"(n));
    return r;
#else
    return m >> ((unsigned)n > 63u ? 63 : n);
#endif
}

OLLIN_HD unsigned long long sf_shr_u(unsigned long long m, unsigned n) {
#if defined(__CUDA_ARCH__)
    unsigned long long r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(m), "r"(n));
    return r;
#else
    return n > 63u ? 0ull : m >> n;
#endif
}

OLLIN_HD unsigned long long sf_shl_u(unsigned long long m, unsigned n) {
#if defined(__CUDA_ARCH__)
    unsigned long long r;
    asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(m), "r"(n));
    return r;
#else
    return n > 63u ? 0ull : m << n;
#endif
}

// the left shift that moves the highest bit of the 32-bit word that differs
// from its sign to bit 31; 2^32-1 where there is none
OLLIN_HD unsigned sf_lead(int hi) {
#if defined(__CUDA_ARCH__)
    unsigned r;
    asm("bfind.shiftamt.s32 %0, %1;" : "=r"(r) : "r"(hi));
    return r;
#else
    const unsigned x = (unsigned)(hi < 0 ? ~hi : hi);
    return x ? (unsigned)__builtin_clz(x) : 0xffffffffu;
#endif
}

OLLIN_HD int sf_clz64(unsigned long long a) {
#if defined(__CUDA_ARCH__)
    return __clzll((long long)a);
#else
    return a ? __builtin_clzll(a) : 64;
#endif
}

OLLIN_HD unsigned long long sf_bits(double x) {
    unsigned long long b;
    memcpy(&b, &x, sizeof(b));
    return b;
}

OLLIN_HD double sf_from_bits(unsigned long long b) {
    double x;
    memcpy(&x, &b, sizeof(x));
    return x;
}

struct sf {
    long long m;
    int e;
};
// a product before normalisation: |m| < 2^60
struct sfp {
    long long m;
    int e;
};

constexpr int kSfNaN = 1 << 20;  // an exponent that to_double turns into NaN

// |m| < 2^62.  A high word of sign bits only (a cancellation of more than 30
// bits) is moved up by 29 bits; the bits that are left stay exact.
OLLIN_HD sf sf_norm(long long m, int e) {
    unsigned s = sf_lead((int)(m >> 32));
    s = (s < 31u ? s : 31u) - 2u;
    return {(long long)((unsigned long long)m << s), e - (int)s};
}

// the same for |m| < 2^63
OLLIN_HD sf sf_norm63(long long m, int e) {
    unsigned s = sf_lead((int)(m >> 32));
    s = s < 31u ? s : 31u;
    return {(long long)((unsigned long long)m << (s - 1u)) >> 1, e + 2 - (int)s};
}

OLLIN_HD sf to_sf(double x) {
    const unsigned long long b = sf_bits(x);
    const int e = (int)(b >> 52) & 0x7ff;
    const unsigned long long a = ((b & 0x000fffffffffffffull) | (e == 0 ? 0 : 0x0010000000000000ull)) << 9;
    const long long s = (long long)b >> 63;
    return {(long long)(a ^ (unsigned long long)s) - s, e == 0x7ff ? kSfNaN : (e == 0 ? 1 : e) - 1084};
}

// The magnitude bits of a result outside the normal range: 1.f with f below
// the highest bit of a, bit 63, and the biased exponent x + 1.  Infinity above
// the range, NaN for kSfNaN, and below it the nearest subnormal number.
OLLIN_HD unsigned long long sf_outside(unsigned long long a, int x) {
    if (x > 0) return x > kSfNaN / 2 ? 0x7ff8000000000000ull : 0x7ff0000000000000ull;
    return (sf_shr_u(a, (unsigned)(10 - x)) + 1) >> 1;
}

// the nearest double of m * 2^e
OLLIN_HD double to_double(long long m, int e) {
    const long long s = m >> 63;
    unsigned long long a = (unsigned long long)((m ^ s) - s);
    const int z = sf_clz64(a);
    a <<= z & 63;
    const int x = e + 1085 - z;               // biased exponent of 1.f, less one: the kept bit 52 adds it
    unsigned long long r = ((unsigned long long)(unsigned)x << 52) + ((a >> 11) + ((a >> 10) & 1));
    if ((unsigned)x >= 0x7feu) r = sf_outside(a, x);
    if (m == 0 && e < kSfNaN / 2) r = 0;
    return sf_from_bits(r | ((unsigned long long)s & 0x8000000000000000ull));
}
OLLIN_HD double to_double(sf a) { return to_double(a.m, a.e); }
OLLIN_HD double to_double(sfp a) { return to_double(a.m, a.e); }

OLLIN_HD sfp operator*(sf a, sf b) {
    const int ah = (int)(a.m >> 32), bh = (int)(b.m >> 32);
    const int al = (int)((unsigned)a.m >> 1), bl = (int)((unsigned)b.m >> 1);
    const long long c = (long long)(ah * 2) * bl + (long long)(bh * 2) * al;
    return {(long long)ah * bh + (c >> 32), a.e + b.e + 64};
}

OLLIN_HD sf sf_norm(sfp p) { return sf_norm(p.m, p.e); }
// a number as a term of a sum of products
OLLIN_HD sfp sf_term(sf a) { return {a.m >> 2, a.e + 2}; }
OLLIN_HD sfp operator-(sfp a) { return {-a.m, a.e}; }
OLLIN_HD sf operator-(sf a) { return {-a.m, a.e}; }

// a positive factor with all 64 bits of its mantissa in use: hi lo * 2^e
struct sfc {
    unsigned hi, lo;
    int e;
};
OLLIN_HD sfc to_sfc(double x) {
    const unsigned long long b = sf_bits(x);
    const unsigned long long a = ((b & 0x000fffffffffffffull) | 0x0010000000000000ull) << 11;
    return {(unsigned)(a >> 32), (unsigned)a, ((int)(b >> 52) & 0x7ff) - 1086};
}
// the nearest double of n * 2^e * c, for any n: the magnitude is normalised to
// 64 bits, so the product is cut at 2^-62 of its value before the rounding
OLLIN_HD double sf_scaled(long long n, int e, sfc c) {
    const long long s = n >> 63;
    unsigned long long a = (unsigned long long)((n ^ s) - s);
    const int z = sf_clz64(a);
    a <<= z & 63;
    const unsigned ah = (unsigned)(a >> 32), al = (unsigned)a;
    const unsigned long long t = (unsigned long long)ah * c.lo, u = (unsigned long long)al * c.hi;
    unsigned long long p = (unsigned long long)ah * c.hi + (t >> 32) + (u >> 32);
    const int k = (p >> 63) ? 0 : 1;
    p <<= k;
    const int x = e + c.e + 1149 - z - k;
    unsigned long long r = ((unsigned long long)(unsigned)x << 52) + ((p >> 11) + ((p >> 10) & 1));
    if ((unsigned)x >= 0x7feu) r = sf_outside(p, x);
    if (a == 0) r = 0;
    return sf_from_bits(r | ((unsigned long long)s & 0x8000000000000000ull));
}

// sums of two to four products
OLLIN_HD sf sf_sum(sfp a, sfp b) {
    const int e = a.e > b.e ? a.e : b.e;
    return sf_norm(sf_shr(a.m, e - a.e) + sf_shr(b.m, e - b.e), e);
}
OLLIN_HD sf sf_sum(sfp a, sfp b, sfp c) {
    int e = a.e > b.e ? a.e : b.e;
    e = e > c.e ? e : c.e;
    return sf_norm(sf_shr(a.m, e - a.e) + sf_shr(b.m, e - b.e) + sf_shr(c.m, e - c.e), e);
}
OLLIN_HD sf sf_sum(sfp a, sfp b, sfp c, sfp d) {
    int e = a.e > b.e ? a.e : b.e;
    const int f = c.e > d.e ? c.e : d.e;
    e = e > f ? e : f;
    return sf_norm(sf_shr(a.m, e - a.e) + sf_shr(b.m, e - b.e) + (sf_shr(c.m, e - c.e) + sf_shr(d.m, e - d.e)), e);
}

// N neighbouring values as integers in one unit, 2^e of e = (largest exponent)
// - 1075 - G: every value whose exponent is within G of the largest is exact,
// the others are cut at that unit.  With G = 4 a sum with integer weights of
// total 64 stays below 2^63, with G = 2 one of total 128 below 2^62.  ``top``:
// the largest exponent, as bits of the high word.  True if every value is exact
// (zeros too); false otherwise, and for values that sf_spread has more to say
// about.
template <int G, int N>
OLLIN_HD bool sf_align_fast(const unsigned long long (&b)[N], long long (&m)[N], int& e, int& top) {
    int t = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const int x = (int)(b[k] >> 32) & 0x7ff00000;
        t = x > t ? x : t;
    }
    // the smallest distance from the largest exponent beyond G; zeros lie 128
    // and more away, values within G wrap around
    unsigned beyond = ~0u;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const unsigned d = (unsigned)(t - ((int)(b[k] >> 32) & 0x7ff00000));
        beyond = d - ((G + 1) << 20) < beyond ? d - ((G + 1) << 20) : beyond;
        unsigned long long a = ((b[k] & 0x000fffffffffffffull) | 0x0010000000000000ull) << G;
        a = sf_shr_u(a, d >> 20);
        const long long s = (long long)b[k] >> 63;
        m[k] = (long long)(a ^ (unsigned long long)s) - s;
    }
    top = t;
    e = (t >> 20) - 1075 - G;
    const bool plain = (unsigned)(t - (128 << 20)) < (unsigned)(0x7ff00000 - (128 << 20));
    return plain && beyond >= (unsigned)((128 - (G + 1)) << 20);
}

// Values that are not all exact: 0 if they are all zero, 1 if sf_rest gives what
// was cut off, 2 if they are too far apart for that (by more than G + kSfRest in
// their exponents), too small (below 2^-895) or not finite.
constexpr int kSfRest = 21;
template <int G, int N>
OLLIN_HD int sf_spread(const unsigned long long (&b)[N], int top) {
    if ((unsigned)(top - (128 << 20)) >= (unsigned)(0x7ff00000 - (128 << 20))) {
        unsigned long long any = 0;
#pragma unroll
        for (int k = 0; k < N; ++k) any |= b[k] << 1;
        return any == 0 ? 0 : 2;
    }
    unsigned far = 0;  // the largest distance of one that is not zero
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const unsigned h = (unsigned)(b[k] >> 32) & 0x7ff00000u, d = h == 0 ? 0u : (unsigned)top - h;
        far = d > far ? d : far;
    }
    return far <= (unsigned)((G + kSfRest) << 20) ? 1 : 2;
}

// Keeps the compiler from running what follows, which is rarely needed, in
// advance of the branch that leads to it.
OLLIN_HD void sf_rare() { asm volatile("" ::: "memory"); }

// N values as by sf_align_fast, for a caller that takes them cut: zero if they
// are all below 2^-958, and such that every weighted sum is NaN if one of them
// is a NaN or an infinity.
template <int G, int N>
OLLIN_HD int sf_align(const unsigned long long (&b)[N], long long (&m)[N]) {
    int e, top;
    sf_align_fast<G>(b, m, e, top);
    if (top == 0x7ff00000 || top < (64 << 20)) {
#pragma unroll
        for (int k = 0; k < N; ++k) m[k] = top == 0x7ff00000 ? 1ll << (4 * k + 8) : 0;
        return top == 0x7ff00000 ? kSfNaN : -1200;
    }
    return e;
}

// What was cut off the aligned values: kSfRest more bits of each, in units of
// 2^(e - kSfRest), with the sign of the value.  Sums with integer weights of
// total 640 fit in 32 bits.
template <int G, int N>
OLLIN_HD void sf_rest(const unsigned long long (&b)[N], int top, int (&r)[N]) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const unsigned n = (unsigned)(top - ((int)(b[k] >> 32) & 0x7ff00000)) >> 20;
        // the bits below bit n of the mantissa with its G zeros, bit n - 1 first
        const unsigned long long a = ((b[k] & 0x000fffffffffffffull) | 0x0010000000000000ull) << G;
        const unsigned q = (unsigned)(sf_shl_u(a, (unsigned)(64 - (int)n)) >> (64 - kSfRest));
        r[k] = (long long)b[k] < 0 ? -(int)q : (int)q;
    }
}
// a weighted sum n of the aligned values and the same sum c of their rests as
// one integer; ``lift``: by how much its unit is smaller
OLLIN_HD long long sf_join(long long n, int c, int& lift) {
    int s = sf_clz64((unsigned long long)(n ^ (n >> 63))) - 2;
    s = s < 0 ? 0 : (s < kSfRest ? s : kSfRest);
    lift = s;
    return (long long)((unsigned long long)n << s) + (c >> (kSfRest - s));
}

}  // namespace ollin
