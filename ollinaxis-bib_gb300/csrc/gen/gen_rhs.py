"""Generates csrc/rhs_algebra_gen.cuh from bssn_spec.py.

FP64 arithmetic, not memory, bounds the right-hand side on GB300, so the
pointwise algebra is emitted in a form with fewer FP64 instructions than the
reference's Maple-generated monomial sums:
  * every temporary of the spec is expanded to a polynomial in its inputs
    (1/r is an independent symbol), collected by powers of r and 1/r, and each
    coefficient is put in multivariate Horner form with the variables ordered
    by how many monomials they occur in (the cheapest of a few orderings under
    an FMA-aware cost model is kept);
  * common subexpressions across all temporaries of a group of tasks are then
    shared;
  * the result is printed as straight-line CUDA, a function per task with what
    its outputs need.  Every rounding is written out (fma, and products and
    sums that the compiler may not contract): a warp that runs several tasks
    forms their common subexpressions once, warps that run one task each form
    them again, and both get the same bits.
Every rewritten temporary is checked to be algebraically identical to the
spec expression before it is emitted.

    python gen_rhs.py            # writes ../rhs_algebra_gen.cuh
"""
import os
import sys

import sympy as sp

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, HERE)
import bssn_spec  # noqa: E402

sys.setrecursionlimit(100000)


def cost(e):
    """FP64 instructions of ``e`` with a*b+c contracted to one FMA."""
    if e.is_Symbol or e.is_Number:
        return 0
    if e.is_Pow:
        b, k = e.args
        k = int(k)
        return cost(b) + {1: 0, 2: 1, 3: 2, 4: 2, 5: 3, 6: 3, 7: 4, 8: 3}.get(k, 4)
    if e.is_Mul:
        nums = [a for a in e.args if a.is_Number]
        others = [a for a in e.args if not a.is_Number]
        c = sum(cost(a) for a in others) + max(len(others) - 1, 0)
        if nums and abs(nums[0]) != 1:
            c += 1
        return c
    if e.is_Add:
        c = sum(cost(a) for a in e.args) + len(e.args) - 1
        # a product takes the addition in; -a is not one
        fus = sum(1 for a in e.args if a.is_Pow or a.is_Mul and not (
            len(a.args) == 2 and a.args[0] == -1 and not a.args[1].is_Pow))
        return c - min(fus, len(e.args) - 1)
    return sum(cost(a) for a in e.args)


METRIC = ("gA", "gB", "gC", "gH", "r", "ir", "glam", "lam", "ipsi4")


def _horner(poly_expr, gens):
    try:
        return sp.polys.polyfuncs.horner(poly_expr, *gens)
    except Exception:
        return poly_expr


def horner_by_frequency(poly_expr, exclude=()):
    """Cheapest multivariate Horner form over a few variable orderings:
    by frequency, data (derivatives, curvature) first, metric first."""
    if not poly_expr.free_symbols:
        return poly_expr
    terms = sp.Add.make_args(poly_expr)
    freq = {}
    for t in terms:
        for s in t.free_symbols:
            freq[s] = freq.get(s, 0) + 1
    gens = sorted((s for s in freq if s not in exclude), key=lambda s: (-freq[s], s.name))
    if not gens:
        return poly_expr
    data = [g for g in gens if g.name not in METRIC]
    metric = [g for g in gens if g.name in METRIC]
    cands = [_horner(poly_expr, gens), _horner(poly_expr, data + metric), _horner(poly_expr, metric + data),
             _horner(poly_expr, list(reversed(gens)))]
    return min(cands, key=cost)


def optimise(expr, r, ir):
    """Pick the cheapest of a few exact rewritings of ``expr``."""
    cands = [expr]
    ex = sp.expand(expr)
    cands.append(ex)
    if len(sp.Add.make_args(ex)) > 2:
        cands.append(horner_by_frequency(ex))
        # collect by powers of r and 1/r, Horner inside each coefficient
        parts = sp.collect(ex, [r, ir], evaluate=False)
        acc = 0
        for k, v in parts.items():
            acc += k * horner_by_frequency(sp.expand(v))
        cands.append(acc)
        # Horner in r on the outside
        try:
            P = sp.Poly(ex, r)
            coeffs = [horner_by_frequency(sp.expand(c)) for c in P.all_coeffs()]
            h = 0
            for c in coeffs:
                h = h * r + c
            cands.append(h)
        except sp.PolynomialError:
            pass
    best = min(cands, key=cost)
    if sp.expand(best - expr) != 0:
        raise AssertionError("rewriting changed the value")
    return best


def number(q):
    return "%d.0" % q.p if q.q == 1 else repr(float(q.p) / float(q.q))


def factors(e):
    """The factors of a product, powers multiplied out, without its sign."""
    out = []
    for f in e.args if e.is_Mul else (e,):
        if f.is_Pow:
            k = int(f.args[1])
            if k == 4:
                out += [sp.Pow(f.args[0], 2, evaluate=False)] * 2
            elif k in (2, 3):
                out += [f.args[0]] * k
            else:
                raise ValueError("power %d" % k)
        elif not (f.is_Number and abs(f) == 1):
            out.append(abs(f) if f.is_Number else f)
    return out


def negative(e):
    return e.is_Number and e < 0 or e.is_Mul and e.args[0].is_Number and e.args[0] < 0


def product(fs):
    return " * ".join(text(f, True) for f in fs)


def text(e, inner=False):
    """``e`` in CUDA with its roundings: sums of products as chains of fma."""
    if e.is_Symbol:
        return e.name
    if e.is_Number:
        t = number(e)
        return "(%s)" % t if inner and e < 0 else t
    if e.is_Mul or e.is_Pow:
        if e.is_Pow and int(e.args[1]) == 2:
            b = text(e.args[0], True)
            t = "%s * %s" % (b, b)
        else:
            t = ("-" if negative(e) else "") + product(factors(e))
        return "(%s)" % t if inner else t
    if e.is_Add:
        single = [t for t in e.args if len(factors(t)) == 1]
        products = [t for t in e.args if len(factors(t)) > 1]
        if single:
            single.sort(key=lambda t: (bool(negative(t)), str(t)))
            acc = ("-" if negative(single[0]) else "") + text(factors(single[0])[0], True)
            for t in single[1:]:
                acc += (" - " if negative(t) else " + ") + text(factors(t)[0], True)
        else:
            t, products = products[0], products[1:]
            acc = ("-" if negative(t) else "") + product(factors(t))
        for t in products:
            fs = factors(t)
            acc = "fma(%s(%s), %s, %s)" % ("-" if negative(t) else "", product(fs[:-1]), text(fs[-1]), acc)
        return "(%s)" % acc if inner and not products else acc
    raise ValueError(str(e))


def group(outputs):
    """The temporaries and outputs of a group of tasks, optimised together:
    definitions, the outputs' expressions, and the instruction counts."""
    syms = {n: sp.Symbol(n) for n in bssn_spec.INPUTS}

    class X:
        pass
    x = X()
    for n, s in syms.items():
        setattr(x, n, s)
    lets = []

    def let(name, expr):
        s = sp.Symbol("t_" + name)
        lets.append((s, expr))
        return s

    outs = bssn_spec.algebra(x, let)
    letmap = dict(lets)
    exprs = [outs[o] if o in outs else letmap[sp.Symbol("t_" + o)] for o in outputs]
    # the temporaries these outputs need; an output that another one uses is
    # one of them
    need, stack = set(), list(exprs)
    while stack:
        for s in stack.pop().free_symbols:
            if s in letmap and s not in need:
                need.add(s)
                stack.append(letmap[s])
    stmts = [(s, e) for s, e in lets if s in need]
    r, ir = syms["r"], syms["ir"]
    before = sum(cost(e) for _, e in stmts) + sum(cost(e) for e in exprs)
    opt = [(s, optimise(e, r, ir)) for s, e in stmts]
    oexp = [sp.Symbol("t_" + o) if sp.Symbol("t_" + o) in need else optimise(e, r, ir) for o, e in zip(outputs, exprs)]
    # common subexpressions across everything
    repl, reduced = sp.cse([e for _, e in opt] + oexp, symbols=sp.numbered_symbols("c"), optimizations="basic")
    after = sum(cost(e) for _, e in repl) + sum(cost(e) for e in reduced)
    defs = dict(list(repl) + [(s, e) for (s, _), e in zip(opt, reduced[:len(opt)])])
    return defs, dict(zip(outputs, reduced[len(opt):])), before, after


def task(defs, exprs, outputs):
    """The lines of one task.  Emission order: depth-first from each output,
    every definition placed just before its first use, so that temporaries
    live briefly (the register pressure of the straight-line code follows the
    text order)."""
    used, emitted, lines, count = set(), set(), [], 0

    def emit(sym):
        nonlocal count
        if sym in emitted or sym not in defs:
            return
        for dep in sorted(defs[sym].free_symbols, key=lambda q: q.name):
            emit(dep)
        lines.append("    const double %s = %s;" % (sym, text(defs[sym])))
        used.update(defs[sym].free_symbols)
        count += cost(defs[sym])
        emitted.add(sym)

    for o in outputs:
        for dep in sorted(exprs[o].free_symbols, key=lambda q: q.name):
            emit(dep)
        lines.append("    o_%s = %s;" % (o, text(exprs[o])))
        used.update(exprs[o].free_symbols)
        count += cost(exprs[o])
    names = set(s.name for s in used)
    return ["    const double %s = in.%s;" % (n, n) for n in bssn_spec.INPUTS if n in names] + lines, count


HEADER = """// Generated by csrc/gen/gen_rhs.py from csrc/gen/bssn_spec.py -- do not edit.
//
// Pointwise BSSN algebra (lapse Laplacian, Ricci tensor, traceless-curvature
// contractions, divergence of KT, geometric sources and constraints) in an
// FP64-instruction-minimised form, cut into tasks that one warp runs after one
// another or the warps of a block side by side, with the same bits.  Estimated
// FP64 instructions per point (FMA-contracted): of a group of tasks as written
// in the spec -> with all its common subexpressions, and of each task alone:
%(costs)s
#pragma once

namespace ollin {

struct AlgIn {
    double %(inputs)s;
};

%(bodies)s
}  // namespace ollin
"""


def main():
    costs, bodies = [], []
    for tasks in bssn_spec.GROUPS:
        defs, exprs, before, after = group(sum(tasks.values(), []))
        costs.append("//   %4d -> %d" % (before, after))
        for name, outputs in tasks.items():
            lines, count = task(defs, exprs, outputs)
            costs.append("//     %-10s %4d" % (name, count))
            bodies.append("__device__ __forceinline__ void alg_%s(const AlgIn& in, %s) {\n%s\n}\n" % (
                name, ", ".join("double& o_" + o for o in outputs), "\n".join(lines)))
    out = HEADER % dict(costs="\n".join(costs), inputs=", ".join(bssn_spec.INPUTS), bodies="\n".join(bodies))
    path = os.path.join(os.path.dirname(HERE), "rhs_algebra_gen.cuh")
    with open(path, "w") as f:
        f.write(out)
    print("\n".join(costs))
    print("wrote", path)


if __name__ == "__main__":
    main()
