"""csrc/rhs_algebra_gen.cuh, compiled for the host: the tasks against the
formulas they are generated from, in exact rational arithmetic."""
import ctypes
import os
import random
import re
import subprocess
import sys
from fractions import Fraction

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ollinaxis-bib_gb300", "csrc")
sys.path.insert(0, os.path.join(CSRC, "gen"))
bssn_spec = pytest.importorskip("bssn_spec")


class Exact:
    """The spec's inputs as rationals."""

    def __init__(self, values):
        self.__dict__.update(values)


def formulas(values):
    """Every temporary and output of the spec, by its formula, in exact
    arithmetic."""
    out = {}

    def let(name, expr):
        out[name] = expr
        return expr

    half = bssn_spec.sp.Rational
    try:
        bssn_spec.sp.Rational = Fraction
        out.update(bssn_spec.algebra(Exact(values), let))
    finally:
        bssn_spec.sp.Rational = half
    return out


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("algebra")
    tasks = [(n, o) for g in bssn_spec.GROUPS for n, o in g.items()]
    src = ["#include <math.h>", "#define __device__", "#define __forceinline__ inline", '#include "rhs_algebra_gen.cuh"',
           "using namespace ollin;"]
    for n, o in tasks:
        src.append('extern "C" void t_%s(const double* in, double* out) { alg_%s(*(const AlgIn*)in, %s); }' % (
            n, n, ", ".join("out[%d]" % k for k in range(len(o)))))
    (d / "a.cpp").write_text("\n".join(src) + "\n")
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "a.so"),
                    str(d / "a.cpp")], check=True)
    return ctypes.CDLL(str(d / "a.so")), tasks


def test_every_task_is_its_formula(lib):
    L, tasks = lib
    rng = random.Random(5)
    for _ in range(40):
        v = {n: rng.uniform(-1, 1) for n in bssn_spec.INPUTS}
        v["r"] = rng.uniform(0.5, 2.0)
        v["ir"] = 1.0 / v["r"]
        want = formulas({n: Fraction(x) for n, x in v.items()})
        scale = formulas({n: abs(Fraction(x)) for n, x in v.items()})
        inputs = (ctypes.c_double * len(v))(*[v[n] for n in bssn_spec.INPUTS])
        for name, outputs in tasks:
            out = (ctypes.c_double * len(outputs))()
            getattr(L, "t_" + name)(inputs, out)
            for o, x in zip(outputs, out):
                # some 100 terms of the size that all of them together have
                # without their signs, a few roundings each
                size = max(abs(scale[o]), abs(want[o]), 1)
                assert abs(Fraction(x) - want[o]) <= Fraction(400, 2 ** 53) * 10 * size, (name, o)


def test_temporaries_that_tasks_share_are_written_alike():
    """One warp that runs several tasks and several warps that run one each give
    the same bits only if a shared temporary has one definition."""
    with open(os.path.join(CSRC, "rhs_algebra_gen.cuh")) as f:
        text = f.read()
    bodies = dict(re.findall(r"void alg_(\w+)\(.*?\{\n(.*?)\n\}", text, flags=re.S))
    for group in bssn_spec.GROUPS:
        seen = {}
        for name in group:
            for sym, expr in re.findall(r"const double (\w+) = (.*);", bodies[name]):
                assert seen.setdefault(sym, expr) == expr, (name, sym)
