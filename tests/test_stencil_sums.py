"""The stencils of csrc/rhs_stencil.cuh, compiled for the host and held to exact
rational arithmetic on fields whose differences FP64 forms with a small error:
steep tails, neighbours of very different size, values next to the ends of the
range."""
import ctypes
import math
import os
import random
import subprocess
from fractions import Fraction

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ollinaxis-bib_gb300", "csrc")

DRIVER = r"""
#include "rhs_stencil.cuh"
using namespace ollin;
extern "C" {
// d1, d2 scaled and rounded; na, nk as integers with their exponents
int t_inside(int order, const double* p, int wide, int neg, double c1, double c2, double* d, long long* n, int* e) {
    const LineSums s = order == 2 ? line_inside<2>(p, 1, wide != 0, true, neg != 0) : line_inside<4>(p, 1, wide != 0, true, neg != 0);
    d[0] = sf_scaled(s.d1, s.e1, to_sfc(c1));
    d[1] = sf_scaled(s.d2, s.e2, to_sfc(c2));
    n[0] = s.na; e[0] = s.ea;
    n[1] = s.nk; e[1] = s.ek;
    return s.lop;
}
void t_edge(int order, const double* p, int d0, int lower, int lop, double c1, double c2, double* d, long long* n, int* e) {
    const LineSums s = order == 2 ? line_edge<2>(p, 1, d0, lower != 0, lop != 0) : line_edge<4>(p, 1, d0, lower != 0, lop != 0);
    d[0] = sf_scaled(s.d1, s.e1, to_sfc(c1));
    d[1] = sf_scaled(s.d2, s.e2, to_sfc(c2));
    n[0] = s.na; e[0] = s.ea;
}
double t_mixed(int order, const double* p, long ld, int i, int j, int nr, int nz, double c) {
    long long n;
    int e;
    if (order == 2) mixed_sum<2>(p, ld, i, j, nr, nz, 3, n, e);
    else mixed_sum<4>(p, ld, i, j, nr, nz, 3, n, e);
    return sf_scaled(n, e, to_sfc(c));
}
// (sum of the aligned na, times a) - (sum of nk, times b), as the kernel adds advection and dissipation
double t_advect(const double* p, double a, double b) {
    const LineSums s = line_inside<4>(p, 1, true, true, false);
    return to_double(sf_sum(sf_norm63(s.na, s.ea) * to_sf(a), -(sf_norm63(s.nk, s.ek) * to_sf(b))));
}
double t_product(long long m, int e, double b) { return to_double(sf_norm63(m, e) * to_sf(b)); }
double t_full_product(const double* x) {
    return to_double(sf_sum(to_sf(x[0]) * to_sf(x[1]), to_sf(x[2]) * to_sf(x[3]))
                     * sf_sum(to_sf(x[4]) * to_sf(x[5]), to_sf(x[6]) * to_sf(x[7])));
}
double t_round(double a) { return to_double(to_sf(a)); }
}
"""

W = {  # weights of d1, d2, na, nk around the middle
    4: ([0, 1, -8, 0, 8, -1, 0], [0, -1, 16, -30, 16, -1, 0], [-1, 6, -21, 0, 21, -6, 1], [-1, 6, -15, 20, -15, 6, -1]),
    2: ([0, -1, 0, 1, 0], [0, 1, -2, 1, 0], [1, -4, 0, 4, -1], [1, -4, 6, -4, 1]),
}
EDGE = {  # d1, d2 by the distance from the end, inwards; the lopsided one
    4: ([[25, -48, 36, -16, 3, 0], [3, 10, -18, 6, -1, 0], [-1, 8, 0, -8, 1, 0]],
        [[45, -154, 214, -156, 61, -10], [10, -15, -4, 14, -6, 1], [-1, 16, -30, 16, -1, 0]], [0, 3, 10, -18, 6, -1]),
    2: ([[3, -4, 1, 0], [1, 0, -1, 0]], [[2, -5, 4, -1], [1, -2, 1, 0]], [0, 3, -4, 1]),
}
ROUND = Fraction(1, 2 ** 53)
CUT = Fraction(1, 2 ** 59)          # what a sum or its scale may lose beside the rounding
TINY = Fraction(1, 2 ** 1075)       # half a subnormal unit


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("stencil")
    src, so = str(d / "driver.cpp"), str(d / "driver.so")
    with open(src, "w") as f:
        f.write(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, "-o", so, src], check=True)
    L = ctypes.CDLL(so)
    d_, p_, i_ = ctypes.c_double, ctypes.c_void_p, ctypes.c_int
    L.t_inside.argtypes = [i_, p_, i_, i_, d_, d_, p_, p_, p_]
    L.t_edge.argtypes = [i_, p_, i_, i_, i_, d_, d_, p_, p_, p_]
    for name, args in (("t_mixed", [i_, p_, ctypes.c_long, i_, i_, i_, i_, d_]), ("t_advect", [p_, d_, d_]),
                       ("t_product", [ctypes.c_longlong, i_, d_]), ("t_full_product", [p_]), ("t_round", [d_])):
        f = getattr(L, name)
        f.argtypes, f.restype = args, d_
    return L


def array(x):
    return (ctypes.c_double * len(x))(*x)


def at(a, k):
    return ctypes.cast(ctypes.addressof(a) + 8 * k, ctypes.c_void_p)


# seven values of each kind of field, as they come
def steep(rng):
    x0, h, p = rng.uniform(6.0, 16.0), rng.choice([0.25, 0.32]), rng.choice([0, 1])
    r = [x0 + k * h for k in range(7)]
    return [q ** p * math.exp(-(q - 5.0) ** 2) for q in r]


def steeper(rng):
    x0 = rng.uniform(0.5, 20.0)
    return [(x0 + 0.64 * k) ** 2 * math.exp(-(x0 + 0.64 * k) ** 2) for k in range(7)]


def spread(rng):
    return [rng.choice([-1, 1]) * math.ldexp(1 + rng.random(), rng.randint(-25, 25)) for _ in range(7)]


def crossing(rng):
    a, b = rng.uniform(-3, 3), rng.uniform(1e-3, 1)
    return [b * (k - 3 + a) * (1 + 0.01 * k) for k in range(7)]


def smooth(rng):
    a, b = rng.uniform(0, 6), rng.uniform(0.01, 0.1)
    return [1.0 + 0.1 * math.sin(a + b * k) for k in range(7)]


def tiny(rng):
    return [rng.choice([-1, 1]) * math.ldexp(1 + rng.random(), rng.randint(-1070, -960)) for _ in range(7)]


def subnormal(rng):
    return [rng.choice([0.0, -0.0, 5e-324, rng.uniform(-1, 1) * 1e-310, rng.uniform(-1, 1) * 1e-307]) for _ in range(7)]


FIELDS = [steep, steeper, spread, crossing, smooth, tiny, subnormal]


def far(x, reach):
    """Whether the values are too far apart, or too small, for the integers."""
    e = [math.frexp(float(v))[1] for v in x if v != 0]
    return bool(e) and (max(e) - min(e) > reach or max(e) < -800)


def close(got, want, weights, x, reach, c=Fraction(1), rounded=True):
    """Exact but for the last rounding; where the values are far apart, FP64
    sums of them, each of at most six roundings."""
    bound = (CUT + (ROUND if rounded else 0)) * abs(want * c) + (TINY if rounded else 0)
    if far(x, reach):
        bound += 6 * ROUND * sum(abs(w * Fraction(v)) for w, v in zip(weights, x)) * abs(c)
    return abs(Fraction(got) - want * c) <= bound


@pytest.mark.parametrize("field", FIELDS)
@pytest.mark.parametrize("order", [4, 2])
def test_inside(lib, field, order):
    rng = random.Random(11)
    n = 7 if order == 4 else 5
    d, q, e = (ctypes.c_double * 2)(), (ctypes.c_longlong * 2)(), (ctypes.c_int * 2)()
    for trial in range(3000):
        x = field(rng)[:n]
        a = array(x)
        wide, neg = trial % 3 != 0, trial % 2
        used = x if wide else [x[k] if 0 < k < n - 1 else 0.0 for k in range(n)]
        c1, c2 = rng.uniform(0.5, 50.0), rng.uniform(0.5, 2000.0)
        lop = lib.t_inside(order, at(a, n // 2), wide, neg, c1, c2, d, q, e)
        w = [list(ws) for ws in W[order]]
        if lop:  # the lopsided difference itself
            w[2] = [p + (k if neg else -k) for p, k in zip(w[2], w[3])]
            assert far(used, 25)
        s = [sum(p * Fraction(v) for p, v in zip(ws, x)) for ws in w]
        assert close(d[0], s[0], w[0], used, 25, Fraction(c1)), (x, d[0])
        assert close(d[1], s[1], w[1], used, 25, Fraction(c2)), (x, d[1])
        if wide:
            for k in (0, 1):
                assert abs(q[k]) < 2 ** 63
                assert close(Fraction(q[k]) * Fraction(2) ** e[k], s[2 + k], w[2 + k], x, 25, rounded=False), (k, x)


@pytest.mark.parametrize("field", FIELDS)
@pytest.mark.parametrize("order", [4, 2])
def test_edge(lib, field, order):
    rng = random.Random(12)
    n = 6 if order == 4 else 4
    d, q, e = (ctypes.c_double * 2)(), (ctypes.c_longlong * 2)(), (ctypes.c_int * 2)()
    for trial in range(3000):
        x = field(rng)[:n]
        if trial % 50 == 0:  # the largest second difference there is
            big = math.ldexp(1 + rng.random(), 3)
            x = [math.copysign(big, w) for w in EDGE[order][1][0]]
        lower, lop, dist = trial % 2, rng.randint(0, 1), rng.randint(0, len(EDGE[order][0]) - 1)
        a = array(x if lower else x[::-1])
        c1, c2 = rng.uniform(0.5, 50.0), rng.uniform(0.5, 2000.0)
        lib.t_edge(order, at(a, dist if lower else n - 1 - dist), dist, lower, lop, c1, c2, d, q, e)
        w1, w2 = EDGE[order][0][dist], EDGE[order][1][dist]
        wl = EDGE[order][2] if lop and dist == len(EDGE[order][0]) - 1 else w1
        s1, s2, sl = (sum(w * Fraction(v) for w, v in zip(ws, x)) for ws in (w1, w2, wl))
        sign = -1 if lower else 1
        assert close(d[0], sign * s1, w1, x, 23, Fraction(c1)), (x, dist)
        assert close(d[1], s2, w2, x, 23, Fraction(c2)), (x, dist)
        # the advection takes twice the one-sided difference
        assert close(Fraction(q[0]) * Fraction(2) ** e[0], 2 * sign * sl, [2 * w for w in wl], x, 23, rounded=False), (x, dist, lop)


@pytest.mark.parametrize("field", FIELDS)
@pytest.mark.parametrize("order", [4, 2])
def test_mixed(lib, field, order):
    rng = random.Random(13)
    for trial in range(1500):
        rows = [field(rng) for _ in range(7)]
        a = array([v for row in rows for v in row])
        i, j = rng.choice([-2, 4, 10]), rng.choice([-2, 4, 10])
        c = rng.uniform(0.1, 100.0)
        got = lib.t_mixed(order, at(a, 3 + 7 * 3), 7, i, j, 10, 10, c)
        f = lambda k, m: Fraction(rows[3 + m][3 + k])  # noqa: E731
        if order == 4 and i == 4 and j == 4:
            want = 16 * (f(1, 1) + f(-1, -1) - f(1, -1) - f(-1, 1)) - (f(2, 2) + f(-2, -2) - f(2, -2) - f(-2, 2))
            used = [f(p, q) for p in (-2, -1, 1, 2) for q in (-2, -1, 1, 2) if abs(p) == abs(q)]
            weights = [16 if abs(v) == 1 else 1 for v in (-2, -2, -1, -1, 1, 1, 2, 2)]
        else:
            end = {-2: ([0, 1, 2], [-3, 4, -1]), 4: ([-1, 0, 1], [-1, 0, 1]), 10: ([-2, -1, 0], [1, -4, 3])}
            (ps, wp), (qs, wq) = end[i], end[j]
            want = sum(u * v * f(p, q) for p, u in zip(ps, wp) for q, v in zip(qs, wq))
            used = [f(p, q) if u * v else 0 for p, u in zip(ps, wp) for q, v in zip(qs, wq)]
            weights = [u * v for u in wp for v in wq]
        assert close(got, want, weights, used, 24, Fraction(c)), (i, j)


@pytest.mark.parametrize("field", [crossing, smooth])
def test_advection_and_dissipation(lib, field):
    """The two products of sums and their sum: cut at 2^-55 of the larger
    product, where FP64 rounds at 2^-53 of each term."""
    rng = random.Random(14)
    for _ in range(2000):
        x = field(rng)
        v7 = array(x)
        a, b = rng.uniform(-1, 1), rng.uniform(0, 1)
        got = Fraction(lib.t_advect(at(v7, 3), a, b))
        sums = [Fraction(c) * sum(w * Fraction(v) for w, v in zip(ws, x)) for c, ws in ((a, W[4][2]), (b, W[4][3]))]
        want = sums[0] - sums[1]
        assert abs(got - want) <= ROUND * abs(want) + Fraction(1, 2 ** 55) * max(abs(s) for s in sums)


def test_products_of_sums(lib):
    """Mantissas with all 62 bits in use: 2.25 units of 2^-58 beside the
    rounding; the rest of a cancellation: 2^-26 of it."""
    rng = random.Random(15)
    for _ in range(5000):
        x = [rng.choice([-1, 1]) * (1 + rng.random()) for _ in range(8)]
        x[2] *= 0.1
        x[6] *= 0.1
        u = [Fraction(x[k]) * Fraction(x[k + 1]) + Fraction(x[k + 2]) * Fraction(x[k + 3]) for k in (0, 4)]
        got = Fraction(lib.t_full_product(array(x)))
        assert abs(got - u[0] * u[1]) <= (ROUND + Fraction(9, 2 ** 60) + Fraction(3, 2 ** 56)) * abs(u[0] * u[1])
        n, b = rng.choice([-1, 1]) * rng.getrandbits(12), 1 + rng.random()
        p = Fraction(n) * Fraction(b)
        assert abs(Fraction(lib.t_product(n, 0, b)) - p) <= Fraction(1, 2 ** 26) * abs(p)


def test_ends_of_the_range(lib):
    for x in (5e-324, -3e-310, 2.2250738585072014e-308, 1.7976931348623157e308, -1.7976931348623157e308):
        assert lib.t_round(x) == x
    d, q, e = (ctypes.c_double * 2)(), (ctypes.c_longlong * 2)(), (ctypes.c_int * 2)()
    big = array([0.0, 0.0, -1e308, 0.0, 1e308, 0.0, 0.0])
    lib.t_inside(4, at(big, 3), 1, 0, 10.0, 1.0, d, q, e)
    assert d[0] == math.inf and d[1] == 0.0
    for bad in (math.nan, math.inf, -math.inf):
        for k in (2, 4):  # in both sums
            x = [1.0, 2.0, 3.0, 1.5, 0.5, 1.0, 7.0]
            x[k] = bad
            v7 = array(x)
            lib.t_inside(4, at(v7, 3), 1, 0, 1.0, 1.0, d, q, e)
            assert math.isnan(d[0]) and math.isnan(d[1])
