// The right-hand side's stencils in integer arithmetic (softfp.cuh).
//
// Every centred, one-sided, mixed and lopsided difference of
// src/base/derivatives.f90 and derivadvect.f90, and the dissipation of
// dissipation.f90, is a sum of neighbours with small integer weights times
// one scale.  The neighbours are aligned to one 64-bit integer unit, so that
// sum is exact where FP64 would round each product and addition; only the
// product with the scale is rounded.  Where the neighbours are further apart
// than the unit reaches (a factor of 16, of 4 at the ends of a line: in some 8%
// of the warps' lines next to a puncture, 25% in the tails of a shell), the sum
// of what was cut off is added, and where they are 2^25 (2^23) apart, smaller
// than 2^-895 or not finite (far out in a shell's tails, on coarse grids), the
// sums are formed in FP64.  So a difference is nowhere further from its exact value than
// FP64 has it (the shell exp(-(r-5)^2) for r from 8 to 16 with h = 0.25: first
// difference to 2e-16 of its value, second to 3e-16; in FP64 8e-16 and 5e-15;
// with neighbours cut at the unit 4e-14 and 1e-13).  A field's five derivatives,
// advection and dissipation take some 700 integer instructions instead of 45 FP64
// ones of 64-76 clocks each, and leave the FP64 unit to the pointwise algebra.
// The rests cost 0.6% of a step of six 512^2 levels of a puncture (145.2 / 146.2
// ms) and 3% of a lone shell's (7.63 / 7.83 ms), 18% of 24 shells side by side
// (30.6 / 36.0 ms), whose cells wait for their stencils.
#pragma once
#include <math.h>

#include "softfp.cuh"

namespace ollin {

namespace {

// Integer sums of one line of a field around a point: value = sum * 2^e, each
// below 2^63.
struct LineSums {
    long long d1, d2;  // first and second difference (scales 1/(12h), 1/(12h^2); order two 1/(2h), 1/h^2)
    long long na;      // advection: beta (na) / (24h) - |beta| (nk) / (24h) (order two: 4h), or, if ``lop``,
    long long nk;      // beta (na) / (24h) alone; the dissipation's bracket, zero outside its range
    int e1, e2, ea, ek;
    bool lop;
};

#if defined(__CUDA_ARCH__)
__device__ __forceinline__ unsigned long long ldb(const double* p) { return sf_bits(__ldg(p)); }
#else
OLLIN_HD unsigned long long ldb(const double* p) { return sf_bits(*p); }
#endif

// The sums of N = 5 or 7 aligned values (or their rests) around the middle one.
// Inside, d1 and d2 are centred.  The lopsided advective difference against the
// shift is the average of its mirror images, (21 D1 - 6 D2 + D3) / 24, and, with
// the sign of the shift, the dissipation bracket over 24 (Dk, Sk: difference and
// sum of the points k away), so both upwind directions share their sums with the
// dissipation.
template <int ORD, typename T, int N>
OLLIN_HD void inside_sums(const T (&m)[N], T& d1, T& d2, T& na, T& nk) {
    constexpr int H = N / 2;
    const T c = m[H], D1 = m[H + 1] - m[H - 1], S1 = m[H + 1] + m[H - 1];
    const T D2 = m[H + 2] - m[H - 2], S2 = m[H + 2] + m[H - 2];
    if constexpr (ORD == 2) {
        d1 = D1;
        d2 = S1 - 2 * c;
        na = 4 * D1 - D2;
        nk = 6 * c - 4 * S1 + S2;
    } else {
        const T D3 = m[N - 1] - m[0], S3 = m[N - 1] + m[0];
        d1 = 8 * D1 - D2;
        d2 = 16 * S1 - S2 - 30 * c;
        na = 21 * D1 - 6 * D2 + D3;
        nk = 20 * c - 15 * S1 + 6 * S2 - S3;
    }
}
OLLIN_HD void put_sum(double v, long long& n, int& e) {
    const sf a = to_sf(v);
    n = a.m;
    e = a.e;
}

// ``wide``: whether na and nk are wanted; the outermost points are not read
// otherwise.  ``second``: whether d2 is.  ``neg``: the sign of the shift.
template <int ORD>
OLLIN_HD LineSums line_inside(const double* p, long st, bool wide, bool second, bool neg) {
    constexpr int H = ORD == 2 ? 2 : 3, N = 2 * H + 1, G = 4;
    unsigned long long b[N];
    const long far = wide ? H * st : 0;
    b[0] = ldb(p - far);
    b[N - 1] = ldb(p + far);
#pragma unroll
    for (int k = 1; k < N - 1; ++k) b[k] = ldb(p + (k - H) * st);
    long long m[N];
    LineSums s;
    int top;
    const bool exact = sf_align_fast<G>(b, m, s.e1, top);
    s.e2 = s.ea = s.ek = s.e1;
    s.lop = false;
    inside_sums<ORD>(m, s.d1, s.d2, s.na, s.nk);
    if (exact) return s;
    sf_rare();
    const int kind = sf_spread<G>(b, top);
    if (kind == 0) {
        s.d1 = s.d2 = s.na = s.nk = 0;
        s.e1 = s.e2 = s.ea = s.ek = -1200;
    } else if (kind == 1) {
        int r[N], d1, d2, na, nk, l;
        sf_rest<G>(b, top, r);
        inside_sums<ORD>(r, d1, d2, na, nk);
        s.d1 = sf_join(s.d1, d1, l); s.e1 -= l;
        if (second) { s.d2 = sf_join(s.d2, d2, l); s.e2 -= l; }
        if (wide) {
            s.na = sf_join(s.na, na, l); s.ea -= l;
            s.nk = sf_join(s.nk, nk, l); s.ek -= l;
        }
    } else {
        sf_rare();
        double f[N];
#pragma unroll
        for (int k = 0; k < N; ++k) f[k] = sf_from_bits(b[k]);
        const double c = f[H], D1 = f[H + 1] - f[H - 1], S1 = f[H + 1] + f[H - 1];
        const double D2 = f[H + 2] - f[H - 2], S2 = f[H + 2] + f[H - 2];
        const double u = neg ? f[H + 1] : f[H - 1], v = neg ? f[H - 1] : f[H + 1], w = neg ? f[H - 2] : f[H + 2];
        if constexpr (ORD == 2) {
            put_sum(D1, s.d1, s.e1);
            put_sum(S1 - 2.0 * c, s.d2, s.e2);
            put_sum(2.0 * fma(3.0, c, fma(-4.0, v, w)), s.na, s.ea);
            put_sum(fma(6.0, c, fma(-4.0, S1, S2)), s.nk, s.ek);
        } else {
            const double x = neg ? f[0] : f[N - 1], S3 = f[N - 1] + f[0];
            put_sum(fma(8.0, D1, -D2), s.d1, s.e1);
            put_sum(-fma(30.0, c, fma(-16.0, S1, S2)), s.d2, s.e2);
            put_sum(2.0 * (fma(6.0, w, fma(-18.0, v, fma(10.0, c, 3.0 * u))) - x), s.na, s.ea);
            put_sum(fma(20.0, c, fma(-15.0, S1, fma(6.0, S2, -S3))), s.nk, s.ek);
        }
        if (!neg) s.na = -s.na;
        s.lop = true;
    }
    return s;
}

// The sums of a line's end: within two points (order two: one) of it the
// stencils are one-sided.  d: points from the end, from which the values are
// taken inwards.
template <int ORD>
OLLIN_HD void edge_weights(int k, int d, bool lop, int& w1, int& w2, int& wl) {
    if constexpr (ORD == 2) {
        constexpr int a1[2][4] = {{3, -4, 1, 0}, {1, 0, -1, 0}}, a2[2][4] = {{2, -5, 4, -1}, {1, -2, 1, 0}};
        constexpr int al[4] = {0, 3, -4, 1};
        w1 = d == 0 ? a1[0][k] : a1[1][k];
        w2 = d == 0 ? a2[0][k] : a2[1][k];
        wl = (d == 1 && lop) ? al[k] : w1;
    } else {
        constexpr int a1[3][6] = {{25, -48, 36, -16, 3, 0}, {3, 10, -18, 6, -1, 0}, {-1, 8, 0, -8, 1, 0}};
        constexpr int a2[3][6] = {{45, -154, 214, -156, 61, -10}, {10, -15, -4, 14, -6, 1}, {-1, 16, -30, 16, -1, 0}};
        constexpr int al[6] = {0, 3, 10, -18, 6, -1};
        w1 = d == 0 ? a1[0][k] : (d == 1 ? a1[1][k] : a1[2][k]);
        w2 = d == 0 ? a2[0][k] : (d == 1 ? a2[1][k] : a2[2][k]);
        wl = (d == 2 && lop) ? al[k] : w1;
    }
}

// d points from the line's end, on the upper side or (mirrored) the lower one;
// ``lop``: whether the innermost of these points takes the lopsided advective
// difference or the centred one (derivadvect.f90).
template <int ORD>
OLLIN_HD LineSums line_edge(const double* p, long st, int d, bool lower, bool lop) {
    constexpr int N = ORD == 2 ? 4 : 6, G = 2;
    const long in = lower ? st : -st;
    unsigned long long b[N];
#pragma unroll
    for (int k = 0; k < N; ++k) b[k] = ldb(p + (k - d) * in);
    long long m[N];
    LineSums s;
    int top;
    const bool exact = sf_align_fast<G>(b, m, s.e1, top);
    // the second difference's weights (640 in all) leave 64 bits: it is summed
    // in two halves, and cut at 2^-59 of its value from 2^62
    long long d1 = 0, na = 0, hi = 0, lo = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        int w1, w2, wl;
        edge_weights<ORD>(k, d, lop, w1, w2, wl);
        d1 += m[k] * w1;
        hi += (long long)(int)(m[k] >> 32) * w2;
        lo += (long long)(unsigned)m[k] * w2;
        na += m[k] * wl;
    }
    hi += lo >> 32;
    const int cut = ((hi ^ (hi >> 63)) >> 30) != 0 ? 3 : 0;
    long long d2 = (long long)((unsigned long long)hi << (32 - cut)) + ((unsigned)lo >> cut);
    s.ea = s.e1;
    s.e2 = s.e1 + cut;
    int kind = 0;
    if (!exact) {
        sf_rare();
        kind = sf_spread<G>(b, top);
        if (kind == 0) {
            d1 = d2 = na = 0;
            s.e1 = s.e2 = s.ea = -1200;
        }
    }
    if (kind == 1) {
        sf_rare();
        int r[N], c1 = 0, c2 = 0, ca = 0, l;
        sf_rest<G>(b, top, r);
#pragma unroll
        for (int k = 0; k < N; ++k) {
            int w1, w2, wl;
            edge_weights<ORD>(k, d, lop, w1, w2, wl);
            c1 += r[k] * w1;
            c2 += r[k] * w2;
            ca += r[k] * wl;
        }
        d1 = sf_join(d1, c1, l); s.e1 -= l;
        d2 = sf_join(d2, c2 >> cut, l); s.e2 -= l;
        na = sf_join(na, ca, l); s.ea -= l;
    } else if (kind == 2) {
        sf_rare();
        double f1 = 0.0, f2 = 0.0, fl = 0.0;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            int w1, w2, wl;
            edge_weights<ORD>(k, d, lop, w1, w2, wl);
            const double v = sf_from_bits(b[k]);
            if (w1 != 0) f1 = fma((double)w1, v, f1);
            if (w2 != 0) f2 = fma((double)w2, v, f2);
            if (wl != 0) fl = fma((double)wl, v, fl);
        }
        put_sum(f1, d1, s.e1);
        put_sum(f2, d2, s.e2);
        put_sum(fl, na, s.ea);
    }
    s.d1 = lower ? -d1 : d1;
    s.d2 = d2;
    s.na = lower ? -na : na;
    s.ea += 1;
    s.nk = 0;
    s.ek = -1200;
    s.lop = true;
    return s;
}

// the first difference alone, at position x of 1-g..n; c: its scale
template <int ORD>
OLLIN_HD double first_difference(const double* p, long st, int x, int n, int g, sfc c) {
    constexpr int lo = ORD == 2 ? 3 : 4, hi = ORD == 2 ? 2 : 3;
    if (x >= lo - g && x <= n - hi) {
        const LineSums u = line_inside<ORD>(p, st, false, false, false);
        return sf_scaled(u.d1, u.e1, c);
    }
    const bool lower = x < lo - g;
    const LineSums u = line_edge<ORD>(p, st, lower ? x - (1 - g) : n - x, lower, false);
    return sf_scaled(u.d1, u.e1, c);
}

// DelDef_r/z (auxiliary_geometry.f90:1085-1094) and the divergence terms of the
// scalar field from the differences a, b: (D_r g_A, D_z g_C) for r and
// (D_r g_C, D_z g_B) for z.  With the contraction written out, so that the two
// kernels that form them give the same bits.
OLLIN_HD double deldef_r(double a, double b, double r, double glam) { return fma(-r, glam, fma(-r, b, -a)); }
OLLIN_HD double deldef_z(double a, double b, double r, double gc) { return fma(-2.0, gc, fma(-r, a, -b)); }
OLLIN_HD double grad_r(double a, double b, double r) { return fma(r, b, a); }
OLLIN_HD double grad_z(double a, double b, double r) { return fma(r, a, b); }

// The mixed derivative (derivatives.f90:615-700): order four inside, times
// 1/(48 dr dz); on the two outermost rows and columns (order two: everywhere)
// the product of second-order first differences, centred or on the last row
// and column one-sided, times 1/(4 dr dz).  Returns which.
template <int ORD>
OLLIN_HD bool mixed_sum(const double* p, long ld, int i, int j, int nr, int nz, int g, long long& n, int& e) {
    constexpr int G = 3;
    const bool in = ORD == 4 && i >= 3 - g && i <= nr - 2 && j >= 3 - g && j <= nz - 2;
    if (in) {
        const unsigned long long b[8] = {ldb(p + 1 + ld),     ldb(p - 1 - ld),     ldb(p + 1 - ld),     ldb(p - 1 + ld),
                                         ldb(p + 2 + 2 * ld), ldb(p - 2 - 2 * ld), ldb(p + 2 - 2 * ld), ldb(p - 2 + 2 * ld)};
        long long m[8];
        int top;
        auto sum = [](const auto& q) { return 16 * ((q[0] + q[1]) - (q[2] + q[3])) - ((q[4] + q[5]) - (q[6] + q[7])); };
        const bool exact = sf_align_fast<G>(b, m, e, top);
        n = sum(m);
        if (exact) return in;
        sf_rare();
        const int kind = sf_spread<G>(b, top);
        if (kind == 0) {
            n = 0;
            e = -1200;
        } else if (kind == 1) {
            int r[8], l;
            sf_rest<G>(b, top, r);
            n = sf_join(n, sum(r), l);
            e -= l;
        } else {
            sf_rare();
            double f[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) f[k] = sf_from_bits(b[k]);
            put_sum(fma(16.0, (f[0] + f[1]) - (f[2] + f[3]), -((f[4] + f[5]) - (f[6] + f[7]))), n, e);
        }
    } else {
        // offsets o, o+1, o+2 with weights w0, w1, w2 in each direction
        const bool ur = i == nr, lr = i == 1 - g, uz = j == nz, lz = j == 1 - g;
        const int r0 = ur ? -2 : (lr ? 0 : -1), z0 = uz ? -2 : (lz ? 0 : -1);
        const int wr[3] = {ur ? 1 : (lr ? -3 : -1), ur ? -4 : (lr ? 4 : 0), ur ? 3 : (lr ? -1 : 1)};
        const int wz[3] = {uz ? 1 : (lz ? -3 : -1), uz ? -4 : (lz ? 4 : 0), uz ? 3 : (lz ? -1 : 1)};
        unsigned long long b[9];
        long long m[9];
        int top;
        const double* q = p + r0 + z0 * ld;
        // points of weight zero are not read: they would widen the range
#pragma unroll
        for (int k = 0; k < 9; ++k) b[k] = wr[k % 3] * wz[k / 3] == 0 ? 0 : ldb(q + k % 3 + (k / 3) * ld);
        const bool exact = sf_align_fast<G>(b, m, e, top);
        n = 0;
#pragma unroll
        for (int k = 0; k < 9; ++k) n += m[k] * (wr[k % 3] * wz[k / 3]);
        if (exact) return in;
        sf_rare();
        const int kind = sf_spread<G>(b, top);
        if (kind == 0) {
            n = 0;
            e = -1200;
        } else if (kind == 1) {
            int r[9], c = 0, l;
            sf_rest<G>(b, top, r);
#pragma unroll
            for (int k = 0; k < 9; ++k) c += r[k] * (wr[k % 3] * wz[k / 3]);
            n = sf_join(n, c, l);
            e -= l;
        } else {
            sf_rare();
            double f = 0.0;
#pragma unroll
            for (int k = 0; k < 9; ++k)
                if (wr[k % 3] * wz[k / 3] != 0) f = fma((double)(wr[k % 3] * wz[k / 3]), sf_from_bits(b[k]), f);
            put_sum(f, n, e);
        }
    }
    return in;
}

}  // namespace

}  // namespace ollin
