"""Generate ``ldk_estimators.cuh``: straight-line two-locus LD estimators for P = 1..4.

The moments statistics of P populations (names and averaging weights as in
``ld_pipeline.py:357-457`` of pg_gpu) are sums of raw estimator calls DD(i,j), Dz(i,j,k),
pi2(i,j,k,l).  Every raw call of the haplotype path is a product of per-population
features (counts, allele counts, D, and a handful of quadratic/cubic count
polynomials) times per-population reciprocal denominators, so a pair's full statistic
vector is computed here as

  1. per population: features + reciprocals 1/n, 1/(n(n-1)), 1/(n(n-1)(n-2)),
     1/(n(n-1)(n-2)(n-3)) (0 where the reference's guard ``den > 0`` fails);
  2. per distinct raw call (calls equal by symmetry evaluated once): a few products;
  3. per statistic: the weighted sum, added into an accumulator.

The feature algebra was derived with sympy from the reference's formulas
(``haplotype_kernels.py:69-304``); ``check()`` re-verifies every identity
symbolically and the unit tests evaluate the same expression strings with NumPy
against the float64 oracle.  The genotype path (``genotype_kernels.py``) keeps the
reference's polynomials in Horner form.

Run ``python -m pg_gpu_b200.csrc.gen_estimators`` to regenerate; ``build()`` does it.
"""
from __future__ import annotations

import functools
import os

HERE = os.path.dirname(os.path.abspath(__file__))

# ---------------------------------------------------------------------------
# statistic specs (moments order and _call_sgc averaging)
# ---------------------------------------------------------------------------


def ld_names(P):
    names = []
    for i in range(P):
        for j in range(i, P):
            names.append(("dd", (i, j)))
    for i in range(P):
        for j in range(P):
            for k in range(j, P):
                names.append(("dz", (i, j, k)))
    for i in range(P):
        for j in range(i, P):
            for k in range(i, P):
                for l in range(k, P):
                    if k == i == l and j != i:
                        continue
                    if i == k and l < j:
                        continue
                    names.append(("pi2", (i, j, k, l)))
    return names


def stat_name(kind, p):
    return {"dd": "DD", "dz": "Dz", "pi2": "pi2"}[kind] + "_" + "_".join(str(x) for x in p)


def stat_specs(P):
    out = []
    for kind, p in ld_names(P):
        if kind == "dd":
            calls = [(1.0, "dd", p)]
        elif kind == "dz":
            i, j, k = p
            calls = [(1.0, "dz", p)] if j == k else [(0.5, "dz", (i, j, k)), (0.5, "dz", (i, k, j))]
        else:
            i, j, k, l = p
            if i == j and k == l:
                qs = [(1.0, p)] if i == k else [(0.5, (i, j, k, l)), (0.5, (k, l, i, j))]
            elif i == j:
                qs = [(0.25, q) for q in ((i, j, k, l), (i, j, l, k), (k, l, i, j), (l, k, i, j))]
            elif k == l:
                qs = [(0.25, q) for q in ((i, j, k, l), (j, i, k, l), (k, l, i, j), (k, l, j, i))]
            else:
                qs = [(0.125, q) for q in ((i, j, k, l), (i, j, l, k), (j, i, k, l), (j, i, l, k),
                                            (k, l, i, j), (l, k, i, j), (k, l, j, i), (l, k, j, i))]
            calls = [(w, "pi2", q) for w, q in qs]
        out.append((stat_name(kind, p), calls))
    return out


def _pi2_case(p):
    i, j, k, l = p
    cnt = {}
    for q in p:
        cnt[q] = cnt.get(q, 0) + 1
    nu, mc = len(cnt), max(cnt.values())
    if nu == 1:
        return "same"
    if mc == 3:
        return "triple"
    if i == j and k == l:
        return "iikk"
    if i == j:
        return "iikl"
    if k == l:
        return "ijkk"
    if (i == k and j == l) or (i == l and j == k):
        return "ijij"
    if nu == 3:
        return "shared"
    return "alldiff"


def _counts_of(p):
    cnt = {}
    for q in p:
        cnt[q] = cnt.get(q, 0) + 1
    return cnt


def canonical(kind, p, geno=False):
    """Canonical (case, args) of a raw call; calls with equal canonical form are equal."""
    if kind == "dd":
        return ("dd1", (p[0],)) if p[0] == p[1] else ("dd2", p)
    if kind == "dz":
        a, b, c = p
        if a == b == c:
            return ("dz_iii", (a,))
        if a == b:
            return ("dz_iij", (a, c))
        if a == c:
            return ("dz_iji", (a, b))
        if b == c:
            return ("dz_ijj", (a, b))
        return ("dz_ijk", p)
    case = _pi2_case(p)
    i, j, k, l = p
    if case == "same":
        return ("pi2_same", (i,))
    if case == "triple":
        cnt = _counts_of(p)
        t = [q for q, c in cnt.items() if c == 3][0]
        s = [q for q, c in cnt.items() if c == 1][0]
        if geno:
            return ("pi2_iiij" if (i == t and j == t) else "pi2_ijii", (t, s))
        return ("pi2_triple", (t, s))
    if case == "iikk":
        return ("pi2_iikk", (i, k))
    if case == "iikl":
        return ("pi2_iikl", (i,) + tuple(sorted((k, l))))
    if case == "ijkk":
        return ("pi2_ijkk", tuple(sorted((i, j))) + (k,))
    if case == "ijij":
        return ("pi2_ijij", (i, j))
    if case == "shared":
        if i == k:
            r = (i, j, l)
        elif i == l:
            r = (i, j, k)
        elif j == k:
            r = (j, i, l)
        else:
            r = (j, i, k)
        return ("pi2_shared", r)
    return ("pi2_alldiff", tuple(sorted((i, j))) + tuple(sorted((k, l))))


# ---------------------------------------------------------------------------
# haplotype path: per-population features and raw-call expressions
# ---------------------------------------------------------------------------

# Per-population feature definitions (C and Python share the syntax).  x.c1..c4 are the
# two-locus counts n11, n10, n01, n00 of ld_statistics.py:281-290; x.ns their sum; x.n the
# sample size used in denominators (n_valid; equal to ns on the haplotype path).
HAP_FEATURES = [
    ("pA", "x.c1 + x.c2"),
    ("qA", "x.c3 + x.c4"),
    ("pB", "x.c1 + x.c3"),
    ("qB", "x.c2 + x.c4"),
    ("E", "x.c1 * x.c4 - x.c2 * x.c3"),          # = -D of ld_pipeline.py:478
    ("a", "x.qA - x.pA"),
    ("b", "x.qB - x.pB"),
    ("s", "(x.c2 + x.c3) - (x.c1 + x.c4)"),
    ("fA", "x.pA * x.qA"),
    ("fB", "x.pB * x.qB"),
    # coefficients of the bilinear pi2(i,j,i,j) correction and of pi2 shared
    ("Q1", "x.c1 * (1 - x.ns + x.c4) - x.c2 * x.c3"),
    ("Q2", "x.c2 * (1 - x.ns + x.c3) - x.c1 * x.c4"),
    ("Q3", "x.c3 * (1 - x.ns + x.c2) - x.c1 * x.c4"),
    ("Q4", "x.c4 * (1 - x.ns + x.c1) - x.c2 * x.c3"),
    ("L1", "x.c4 * (x.ns - x.c1) + x.c2 * x.c3"),
    ("L2", "x.c3 * (x.ns - x.c2) + x.c1 * x.c4"),
    ("L3", "x.c2 * (x.ns - x.c3) + x.c1 * x.c4"),
    ("L4", "x.c1 * (x.ns - x.c4) + x.c2 * x.c3"),
    # pi2 with one population three times: 2*num = pB_s*T1_t + qB_s*T2_t
    ("T1", "x.fA * x.qB - x.c1 * x.c4 - x.c2 * x.c3 - 2 * x.c2 * x.c4"),
    ("T2", "x.fA * x.pB - 2 * x.c1 * x.c3 - x.c1 * x.c4 - x.c2 * x.c3"),
    # single-population numerators
    ("DDs", "x.E * x.E - x.c1 * x.c4 * (x.c1 + x.c4 - 1) - x.c2 * x.c3 * (x.c2 + x.c3 - 1)"),
    ("DZs", "x.E * x.a * x.b + x.E * x.s + 2 * (x.c2 * x.c3 + x.c1 * x.c4)"),
    ("PIs", "x.fA * x.fB - x.c1 * x.c4 * (-1 + x.c1 + 3 * x.c2 + 3 * x.c3 + x.c4)"
            " - x.c2 * x.c3 * (-1 + 3 * x.c1 + x.c2 + x.c3 + 3 * x.c4)"),
]

# which features each case reads (besides counts); drives what is computed per P
HAP_CASE_FEATURES = {
    "dd1": ["DDs", "r4"], "dd2": ["E", "r2"],
    "dz_iii": ["DZs", "r4"], "dz_iij": ["a", "E", "b", "r3", "r1"],
    "dz_iji": ["a", "E", "b", "r3", "r1"], "dz_ijj": ["E", "s", "a", "b", "r2"],
    "dz_ijk": ["E", "a", "b", "r2", "r1"],
    "pi2_same": ["PIs", "r4"], "pi2_iikk": ["fA", "fB", "r2"],
    "pi2_iikl": ["fA", "pB", "qB", "r2", "r1"], "pi2_ijkk": ["fB", "pA", "qA", "r2", "r1"],
    "pi2_alldiff": ["pA", "qA", "pB", "qB", "r1"], "pi2_triple": ["T1", "T2", "pB", "qB", "r3", "r1"],
    "pi2_ijij": ["pA", "qA", "pB", "qB", "Q1", "Q2", "Q3", "Q4", "L1", "L2", "L3", "L4", "r2"],
    "pi2_shared": ["pA", "qA", "pB", "qB", "L1", "L2", "L3", "L4", "r2", "r1"],
}


def hap_call_expr(case, args):
    """Expression (C and Python syntax) of one canonical raw haplotype call."""
    f = lambda p, name: f"f[{p}].{name}"  # noqa: E731
    if case == "dd1":
        (i,) = args
        return f"{f(i,'DDs')} * {f(i,'r4')}"
    if case == "dd2":
        i, j = args
        return f"({f(i,'E')} * {f(j,'E')}) * ({f(i,'r2')} * {f(j,'r2')})"
    if case == "dz_iii":
        (i,) = args
        return f"{f(i,'DZs')} * {f(i,'r4')}"
    if case == "dz_iij":
        i, j = args
        return f"({f(i,'a')} * {f(i,'E')} * {f(j,'b')}) * ({f(i,'r3')} * {f(j,'r1')})"
    if case == "dz_iji":
        i, j = args
        return f"({f(i,'b')} * {f(i,'E')} * {f(j,'a')}) * ({f(i,'r3')} * {f(j,'r1')})"
    if case == "dz_ijj":
        i, j = args
        return (f"({f(i,'E')} * ({f(j,'s')} + {f(j,'b')} * {f(j,'a')}))"
                f" * ({f(i,'r2')} * {f(j,'r2')})")
    if case == "dz_ijk":
        i, j, k = args
        return (f"({f(i,'E')} * {f(j,'a')} * {f(k,'b')})"
                f" * ({f(i,'r2')} * {f(j,'r1')} * {f(k,'r1')})")
    if case == "pi2_same":
        (i,) = args
        return f"{f(i,'PIs')} * {f(i,'r4')}"
    if case == "pi2_iikk":
        i, k = args
        return f"({f(i,'fA')} * {f(k,'fB')}) * ({f(i,'r2')} * {f(k,'r2')})"
    if case == "pi2_iikl":
        i, k, l = args
        return (f"0.5 * ({f(i,'fA')} * ({f(k,'pB')} * {f(l,'qB')} + {f(k,'qB')} * {f(l,'pB')}))"
                f" * ({f(i,'r2')} * {f(k,'r1')} * {f(l,'r1')})")
    if case == "pi2_ijkk":
        i, j, k = args
        return (f"0.5 * ({f(k,'fB')} * ({f(i,'pA')} * {f(j,'qA')} + {f(i,'qA')} * {f(j,'pA')}))"
                f" * ({f(k,'r2')} * {f(i,'r1')} * {f(j,'r1')})")
    if case == "pi2_alldiff":
        i, j, k, l = args
        return (f"0.25 * (({f(i,'pA')} * {f(j,'qA')} + {f(i,'qA')} * {f(j,'pA')})"
                f" * ({f(k,'pB')} * {f(l,'qB')} + {f(k,'qB')} * {f(l,'pB')}))"
                f" * ({f(i,'r1')} * {f(j,'r1')} * {f(k,'r1')} * {f(l,'r1')})")
    if case == "pi2_triple":
        t, s = args
        return (f"0.5 * ({f(s,'pB')} * {f(t,'T1')} + {f(s,'qB')} * {f(t,'T2')})"
                f" * ({f(t,'r3')} * {f(s,'r1')})")
    if case == "pi2_ijij":
        i, j = args
        HA = f"({f(i,'pA')} * {f(j,'qA')} + {f(i,'qA')} * {f(j,'pA')})"
        HB = f"({f(i,'pB')} * {f(j,'qB')} + {f(i,'qB')} * {f(j,'pB')})"
        corr = (f"({f(i,'Q1')} * {f(j,'c4')} + {f(i,'Q2')} * {f(j,'c3')} + {f(i,'Q3')} * {f(j,'c2')}"
                f" + {f(i,'Q4')} * {f(j,'c1')} - ({f(i,'c1')} * {f(j,'L1')} + {f(i,'c2')} * {f(j,'L2')}"
                f" + {f(i,'c3')} * {f(j,'L3')} + {f(i,'c4')} * {f(j,'L4')}))")
        return f"0.25 * ({HA} * {HB} + {corr}) * ({f(i,'r2')} * {f(j,'r2')})"
    if case == "pi2_shared":
        s, a, b = args
        F1 = f"({f(s,'L1')} - {f(s,'c4')})"
        F2 = f"({f(s,'L2')} - {f(s,'c3')})"
        F3 = f"({f(s,'L3')} - {f(s,'c2')})"
        F4 = f"({f(s,'L4')} - {f(s,'c1')})"
        return (f"0.25 * ({f(a,'pA')} * ({f(b,'pB')} * {F1} + {f(b,'qB')} * {F2})"
                f" + {f(a,'qA')} * ({f(b,'pB')} * {F3} + {f(b,'qB')} * {F4}))"
                f" * ({f(s,'r2')} * {f(a,'r1')} * {f(b,'r1')})")
    raise ValueError(case)


# Case ids of ldk_raw_hap (order is part of the C ABI).
RAW_CASES = ["dd1", "dd2", "dz_iii", "dz_iij", "dz_iji", "dz_ijj", "dz_ijk", "pi2_same",
             "pi2_iikk", "pi2_iikl", "pi2_ijkk", "pi2_alldiff", "pi2_triple", "pi2_ijij",
             "pi2_shared"]
RAW_ARITY = {"dd1": 1, "dd2": 2, "dz_iii": 1, "dz_iij": 2, "dz_iji": 2, "dz_ijj": 2, "dz_ijk": 3,
             "pi2_same": 1, "pi2_iikk": 2, "pi2_iikl": 3, "pi2_ijkk": 3, "pi2_alldiff": 4,
             "pi2_triple": 2, "pi2_ijij": 2, "pi2_shared": 3}


def emit_raw_dispatch():
    L = ["template <typename T>",
         "LDK_DEV T hap_raw_by_case(int case_id, const int* g, const HapFeat<T>* f) {",
         "    switch (case_id) {"]
    for cid, case in enumerate(RAW_CASES):
        args = tuple(f"g[{k}]" for k in range(RAW_ARITY[case]))
        expr = hap_call_expr(case, args)
        L.append(f"    case {cid}: return {_cexpr(expr)};  // {case}")
    L.append("    default: return T(0);")
    L.append("    }")
    L.append("}")
    return "\n".join(L)


def plan(P, geno=False):
    """(calls, stats): distinct canonical calls in first-use order and, per statistic,
    the list of (weight, call index)."""
    calls, index, stats = [], {}, []
    for name, cl in stat_specs(P):
        terms = {}
        for w, kind, p in cl:
            key = canonical(kind, p, geno)
            if key not in index:
                index[key] = len(calls)
                calls.append(key)
            terms[index[key]] = terms.get(index[key], 0.0) + w
        stats.append((name, sorted(terms.items())))
    return calls, stats


def hap_features_needed(P):
    calls, _ = plan(P)
    need = set()
    for case, _ in calls:
        need.update(HAP_CASE_FEATURES[case])
    # close over feature dependencies
    order = [n for n, _ in HAP_FEATURES]
    deps = {n: {d.split(".")[1].split()[0].rstrip(")") for d in e.replace("(", " ").split() if d.startswith("x.")}
            for n, e in HAP_FEATURES}
    changed = True
    while changed:
        changed = False
        for n in list(need):
            for d in deps.get(n, ()):
                if d in order and d not in need:
                    need.add(d)
                    changed = True
    return [n for n in order if n in need], sorted(r for r in need if r.startswith("r"))


# ---------------------------------------------------------------------------
# genotype path (moments order g1..g9 = n22, n21, n20, n12, n11, n10, n02, n01, n00)
# ---------------------------------------------------------------------------

# 16x the polynomial part of genotype DD(i,i) (genotype_kernels.py:43-68)
GENO_DD_POLY = (
    "(x.g2 * x.g4 - x.g2 * x.g2 * x.g4 + 4 * x.g3 * x.g4 - 4 * x.g2 * x.g3 * x.g4 - 4 * x.g3 * x.g3 * "
    "x.g4) + (-x.g2 * x.g4 * x.g4 - 4 * x.g3 * x.g4 * x.g4) + (x.g1 * x.g5 - x.g1 * x.g1 * x.g5 + "
    "x.g3 * x.g5 + 2 * x.g1 * x.g3 * x.g5 - x.g3 * x.g3 * x.g5 - 4 * x.g3 * x.g4 * x.g5 - x.g1 * x.g5 "
    "* x.g5 - x.g3 * x.g5 * x.g5) + (4 * x.g1 * x.g6 - 4 * x.g1 * x.g1 * x.g6 + x.g2 * x.g6 - 4 * "
    "x.g1 * x.g2 * x.g6 - x.g2 * x.g2 * x.g6 + 2 * x.g2 * x.g4 * x.g6 - 4 * x.g1 * x.g5 * x.g6 - 4 * "
    "x.g1 * x.g6 * x.g6 - x.g2 * x.g6 * x.g6) + (4 * x.g2 * x.g7 - 4 * x.g2 * x.g2 * x.g7 + 16 * x.g3 "
    "* x.g7 - 16 * x.g2 * x.g3 * x.g7 - 16 * x.g3 * x.g3 * x.g7 - 4 * x.g2 * x.g4 * x.g7 - 16 * x.g3 "
    "* x.g4 * x.g7 + x.g5 * x.g7 + 2 * x.g1 * x.g5 * x.g7 - 4 * x.g2 * x.g5 * x.g7 - 18 * x.g3 * x.g5 "
    "* x.g7 - x.g5 * x.g5 * x.g7 + 4 * x.g6 * x.g7 + 8 * x.g1 * x.g6 * x.g7 - 16 * x.g3 * x.g6 * x.g7 "
    "- 4 * x.g5 * x.g6 * x.g7 - 4 * x.g6 * x.g6 * x.g7 - 4 * x.g2 * x.g7 * x.g7 - 16 * x.g3 * x.g7 * "
    "x.g7 - x.g5 * x.g7 * x.g7 - 4 * x.g6 * x.g7 * x.g7) + (4 * x.g1 * x.g8 - 4 * x.g1 * x.g1 * x.g8 "
    "+ 4 * x.g3 * x.g8 + 8 * x.g1 * x.g3 * x.g8 - 4 * x.g3 * x.g3 * x.g8 + x.g4 * x.g8 - 4 * x.g1 * "
    "x.g4 * x.g8 + 2 * x.g2 * x.g4 * x.g8 - x.g4 * x.g4 * x.g8 - 4 * x.g1 * x.g5 * x.g8 - 4 * x.g3 * "
    "x.g5 * x.g8 + x.g6 * x.g8 + 2 * x.g2 * x.g6 * x.g8 - 4 * x.g3 * x.g6 * x.g8 + 2 * x.g4 * x.g6 * "
    "x.g8 - x.g6 * x.g6 * x.g8 - 16 * x.g3 * x.g7 * x.g8 - 4 * x.g6 * x.g7 * x.g8 - 4 * x.g1 * x.g8 * "
    "x.g8 - 4 * x.g3 * x.g8 * x.g8 - x.g4 * x.g8 * x.g8 - x.g6 * x.g8 * x.g8) + (16 * x.g1 * x.g9 - "
    "16 * x.g1 * x.g1 * x.g9 + 4 * x.g2 * x.g9 - 16 * x.g1 * x.g2 * x.g9 - 4 * x.g2 * x.g2 * x.g9 + 4 "
    "* x.g4 * x.g9 - 16 * x.g1 * x.g4 * x.g9 + 8 * x.g3 * x.g4 * x.g9 - 4 * x.g4 * x.g4 * x.g9 + x.g5 "
    "* x.g9 - 18 * x.g1 * x.g5 * x.g9 - 4 * x.g2 * x.g5 * x.g9 + 2 * x.g3 * x.g5 * x.g9 - 4 * x.g4 * "
    "x.g5 * x.g9 - x.g5 * x.g5 * x.g9 - 16 * x.g1 * x.g6 * x.g9 - 4 * x.g2 * x.g6 * x.g9 + 8 * x.g2 * "
    "x.g7 * x.g9 + 2 * x.g5 * x.g7 * x.g9 - 16 * x.g1 * x.g8 * x.g9 - 4 * x.g4 * x.g8 * x.g9 - 16 * "
    "x.g1 * x.g9 * x.g9 - 4 * x.g2 * x.g9 * x.g9 - 4 * x.g4 * x.g9 * x.g9 - x.g5 * x.g9 * x.g9) "
)

# quartic part of genotype Dz(i,i,i) (genotype_kernels.py:249-269)
GENO_DZ_QUARTIC = (
    "-(x.g2 * x.g4) + 3 * x.g1 * x.g2 * x.g4 + x.g2 * x.g2 * x.g4 + 2 * x.g3 * x.g4 + 4 * x.g1 * x.g3 "
    "* x.g4 - x.g2 * x.g3 * x.g4 - 4 * x.g3 * x.g3 * x.g4 + x.g2 * x.g4 * x.g4 + 2 * x.g3 * x.g4 * "
    "x.g4 + 2 * x.g1 * x.g5 - 3 * x.g1 * x.g1 * x.g5 - x.g1 * x.g2 * x.g5 + 2 * x.g3 * x.g5 + 2 * "
    "x.g1 * x.g3 * x.g5 - x.g2 * x.g3 * x.g5 - 3 * x.g3 * x.g3 * x.g5 - x.g1 * x.g4 * x.g5 + x.g3 * "
    "x.g4 * x.g5 + 2 * x.g1 * x.g6 - 4 * x.g1 * x.g1 * x.g6 - x.g2 * x.g6 - x.g1 * x.g2 * x.g6 + x.g2 "
    "* x.g2 * x.g6 + 4 * x.g1 * x.g3 * x.g6 + 3 * x.g2 * x.g3 * x.g6 - 2 * x.g1 * x.g4 * x.g6 - 2 * "
    "x.g2 * x.g4 * x.g6 - 2 * x.g3 * x.g4 * x.g6 + x.g1 * x.g5 * x.g6 - x.g3 * x.g5 * x.g6 + 2 * x.g1 "
    "* x.g6 * x.g6 + x.g2 * x.g6 * x.g6 + 2 * x.g2 * x.g7 + 4 * x.g1 * x.g2 * x.g7 + 2 * x.g2 * x.g2 "
    "* x.g7 + 8 * x.g3 * x.g7 + 4 * x.g1 * x.g3 * x.g7 - 4 * x.g3 * x.g3 * x.g7 - x.g2 * x.g4 * x.g7 "
    "+ 2 * x.g5 * x.g7 + 2 * x.g1 * x.g5 * x.g7 + x.g2 * x.g5 * x.g7 + 2 * x.g3 * x.g5 * x.g7 - x.g4 "
    "* x.g5 * x.g7 + 2 * x.g6 * x.g7 - x.g2 * x.g6 * x.g7 - 2 * x.g4 * x.g6 * x.g7 + x.g5 * x.g6 * "
    "x.g7 + 2 * x.g6 * x.g6 * x.g7 - 4 * x.g2 * x.g7 * x.g7 - 4 * x.g3 * x.g7 * x.g7 - 3 * x.g5 * "
    "x.g7 * x.g7 - 4 * x.g6 * x.g7 * x.g7 + 2 * x.g1 * x.g8 - 4 * x.g1 * x.g1 * x.g8 - 2 * x.g1 * "
    "x.g2 * x.g8 + 2 * x.g3 * x.g8 - 2 * x.g2 * x.g3 * x.g8 - 4 * x.g3 * x.g3 * x.g8 - x.g4 * x.g8 - "
    "x.g1 * x.g4 * x.g8 - 2 * x.g2 * x.g4 * x.g8 - x.g3 * x.g4 * x.g8 + x.g4 * x.g4 * x.g8 + x.g1 * "
    "x.g5 * x.g8 + x.g3 * x.g5 * x.g8 - x.g6 * x.g8 - x.g1 * x.g6 * x.g8 - 2 * x.g2 * x.g6 * x.g8 - "
    "x.g3 * x.g6 * x.g8 - 2 * x.g4 * x.g6 * x.g8 + x.g6 * x.g6 * x.g8 + 4 * x.g1 * x.g7 * x.g8 - 2 * "
    "x.g2 * x.g7 * x.g8 + 3 * x.g4 * x.g7 * x.g8 - x.g5 * x.g7 * x.g8 - x.g6 * x.g7 * x.g8 + 2 * x.g1 "
    "* x.g8 * x.g8 + 2 * x.g3 * x.g8 * x.g8 + x.g4 * x.g8 * x.g8 + x.g6 * x.g8 * x.g8 + 8 * x.g1 * "
    "x.g9 - 4 * x.g1 * x.g1 * x.g9 + 2 * x.g2 * x.g9 + 2 * x.g2 * x.g2 * x.g9 + 4 * x.g1 * x.g3 * "
    "x.g9 + 4 * x.g2 * x.g3 * x.g9 + 2 * x.g4 * x.g9 - x.g2 * x.g4 * x.g9 + 2 * x.g4 * x.g4 * x.g9 + "
    "2 * x.g5 * x.g9 + 2 * x.g1 * x.g5 * x.g9 + x.g2 * x.g5 * x.g9 + 2 * x.g3 * x.g5 * x.g9 + x.g4 * "
    "x.g5 * x.g9 - x.g2 * x.g6 * x.g9 - 2 * x.g4 * x.g6 * x.g9 - x.g5 * x.g6 * x.g9 + 4 * x.g1 * x.g7 "
    "* x.g9 + 4 * x.g3 * x.g7 * x.g9 + 4 * x.g4 * x.g7 * x.g9 + 2 * x.g5 * x.g7 * x.g9 + 4 * x.g6 * "
    "x.g7 * x.g9 - 2 * x.g2 * x.g8 * x.g9 + 4 * x.g3 * x.g8 * x.g9 - x.g4 * x.g8 * x.g9 - x.g5 * x.g8 "
    "* x.g9 + 3 * x.g6 * x.g8 * x.g9 - 4 * x.g1 * x.g9 * x.g9 - 4 * x.g2 * x.g9 * x.g9 - 4 * x.g4 * "
    "x.g9 * x.g9 - 3 * x.g5 * x.g9 * x.g9 "
)

# 16x the correction part of genotype pi2(i,i,i,i) (genotype_kernels.py:377-403)
GENO_PI2_CORR = (
    "(13 * x.g2 * x.g4 - 16 * x.g1 * x.g2 * x.g4 - 11 * x.g2 * x.g2 * x.g4 + 16 * x.g3 * x.g4 - 28 * "
    "x.g1 * x.g3 * x.g4 - 24 * x.g2 * x.g3 * x.g4) + (-8 * x.g3 * x.g3 * x.g4 - 11 * x.g2 * x.g4 * "
    "x.g4 - 20 * x.g3 * x.g4 * x.g4 - 6 * x.g5 + 12 * x.g1 * x.g5 - 4 * x.g1 * x.g1 * x.g5 + 17 * "
    "x.g2 * x.g5) + (-20 * x.g1 * x.g2 * x.g5 - 11 * x.g2 * x.g2 * x.g5 + 12 * x.g3 * x.g5 - 28 * "
    "x.g1 * x.g3 * x.g5 - 20 * x.g2 * x.g3 * x.g5 - 4 * x.g3 * x.g3 * x.g5) + (17 * x.g4 * x.g5 - 20 "
    "* x.g1 * x.g4 * x.g5 - 32 * x.g2 * x.g4 * x.g5 - 40 * x.g3 * x.g4 * x.g5 - 11 * x.g4 * x.g4 * "
    "x.g5 + 11 * x.g5 * x.g5) + (-16 * x.g1 * x.g5 * x.g5 - 17 * x.g2 * x.g5 * x.g5 - 16 * x.g3 * "
    "x.g5 * x.g5 - 17 * x.g4 * x.g5 * x.g5 - 6 * x.g5 * x.g5 * x.g5 + 16 * x.g1 * x.g6 - 8 * x.g1 * "
    "x.g1 * x.g6) + (13 * x.g2 * x.g6 - 24 * x.g1 * x.g2 * x.g6 - 11 * x.g2 * x.g2 * x.g6 - 28 * x.g1 "
    "* x.g3 * x.g6 - 16 * x.g2 * x.g3 * x.g6 + 24 * x.g4 * x.g6) + (-36 * x.g1 * x.g4 * x.g6 - 38 * "
    "x.g2 * x.g4 * x.g6 - 36 * x.g3 * x.g4 * x.g6 - 20 * x.g4 * x.g4 * x.g6 + 17 * x.g5 * x.g6 - 40 * "
    "x.g1 * x.g5 * x.g6) + (-32 * x.g2 * x.g5 * x.g6 - 20 * x.g3 * x.g5 * x.g6 - 42 * x.g4 * x.g5 * "
    "x.g6 - 17 * x.g5 * x.g5 * x.g6 - 20 * x.g1 * x.g6 * x.g6 - 11 * x.g2 * x.g6 * x.g6) + (-20 * "
    "x.g4 * x.g6 * x.g6 - 11 * x.g5 * x.g6 * x.g6 + 16 * x.g2 * x.g7 - 28 * x.g1 * x.g2 * x.g7 - 20 * "
    "x.g2 * x.g2 * x.g7 + 16 * x.g3 * x.g7) + (-48 * x.g1 * x.g3 * x.g7 - 44 * x.g2 * x.g3 * x.g7 - "
    "16 * x.g3 * x.g3 * x.g7 - 24 * x.g2 * x.g4 * x.g7 - 44 * x.g3 * x.g4 * x.g7) + (12 * x.g5 * x.g7 "
    "- 28 * x.g1 * x.g5 * x.g7 - 40 * x.g2 * x.g5 * x.g7 - 48 * x.g3 * x.g5 * x.g7 - 20 * x.g4 * x.g5 "
    "* x.g7 - 16 * x.g5 * x.g5 * x.g7) + (16 * x.g6 * x.g7 - 48 * x.g1 * x.g6 * x.g7 - 48 * x.g2 * "
    "x.g6 * x.g7 - 44 * x.g3 * x.g6 * x.g7 - 36 * x.g4 * x.g6 * x.g7 - 40 * x.g5 * x.g6 * x.g7) + "
    "(-20 * x.g6 * x.g6 * x.g7 - 8 * x.g2 * x.g7 * x.g7 - 16 * x.g3 * x.g7 * x.g7 - 4 * x.g5 * x.g7 * "
    "x.g7 - 8 * x.g6 * x.g7 * x.g7 + 16 * x.g1 * x.g8 - 8 * x.g1 * x.g1 * x.g8) + (24 * x.g2 * x.g8 - "
    "36 * x.g1 * x.g2 * x.g8 - 20 * x.g2 * x.g2 * x.g8 + 16 * x.g3 * x.g8 - 48 * x.g1 * x.g3 * x.g8 - "
    "36 * x.g2 * x.g3 * x.g8 - 8 * x.g3 * x.g3 * x.g8) + (13 * x.g4 * x.g8 - 24 * x.g1 * x.g4 * x.g8 "
    "- 38 * x.g2 * x.g4 * x.g8 - 48 * x.g3 * x.g4 * x.g8 - 11 * x.g4 * x.g4 * x.g8 + 17 * x.g5 * x.g8 "
    "- 40 * x.g1 * x.g5 * x.g8) + (-42 * x.g2 * x.g5 * x.g8 - 40 * x.g3 * x.g5 * x.g8 - 32 * x.g4 * "
    "x.g5 * x.g8 - 17 * x.g5 * x.g5 * x.g8 + 13 * x.g6 * x.g8 - 48 * x.g1 * x.g6 * x.g8) + (-38 * "
    "x.g2 * x.g6 * x.g8 - 24 * x.g3 * x.g6 * x.g8 - 38 * x.g4 * x.g6 * x.g8 - 32 * x.g5 * x.g6 * x.g8 "
    "- 11 * x.g6 * x.g6 * x.g8 - 28 * x.g1 * x.g7 * x.g8) + (-36 * x.g2 * x.g7 * x.g8 - 44 * x.g3 * "
    "x.g7 * x.g8 - 16 * x.g4 * x.g7 * x.g8 - 20 * x.g5 * x.g7 * x.g8 - 24 * x.g6 * x.g7 * x.g8 - 20 * "
    "x.g1 * x.g8 * x.g8) + (-20 * x.g2 * x.g8 * x.g8 - 20 * x.g3 * x.g8 * x.g8 - 11 * x.g4 * x.g8 * "
    "x.g8 - 11 * x.g5 * x.g8 * x.g8 - 11 * x.g6 * x.g8 * x.g8 + 16 * x.g1 * x.g9 - 16 * x.g1 * x.g1 * "
    "x.g9) + (16 * x.g2 * x.g9 - 44 * x.g1 * x.g2 * x.g9 - 20 * x.g2 * x.g2 * x.g9 - 48 * x.g1 * x.g3 "
    "* x.g9 - 28 * x.g2 * x.g3 * x.g9 + 16 * x.g4 * x.g9) + (-44 * x.g1 * x.g4 * x.g9 - 48 * x.g2 * "
    "x.g4 * x.g9 - 48 * x.g3 * x.g4 * x.g9 - 20 * x.g4 * x.g4 * x.g9 + 12 * x.g5 * x.g9 - 48 * x.g1 * "
    "x.g5 * x.g9) + (-40 * x.g2 * x.g5 * x.g9 - 28 * x.g3 * x.g5 * x.g9 - 40 * x.g4 * x.g5 * x.g9 - "
    "16 * x.g5 * x.g5 * x.g9 - 44 * x.g1 * x.g6 * x.g9 - 24 * x.g2 * x.g6 * x.g9) + (-36 * x.g4 * "
    "x.g6 * x.g9 - 20 * x.g5 * x.g6 * x.g9 - 48 * x.g1 * x.g7 * x.g9 - 48 * x.g2 * x.g7 * x.g9 - 48 * "
    "x.g3 * x.g7 * x.g9 - 28 * x.g4 * x.g7 * x.g9) + (-28 * x.g5 * x.g7 * x.g9 - 28 * x.g6 * x.g7 * "
    "x.g9 - 44 * x.g1 * x.g8 * x.g9 - 36 * x.g2 * x.g8 * x.g9 - 28 * x.g3 * x.g8 * x.g9 - 24 * x.g4 * "
    "x.g8 * x.g9) + (-20 * x.g5 * x.g8 * x.g9 - 16 * x.g6 * x.g8 * x.g9 - 16 * x.g1 * x.g9 * x.g9 - 8 "
    "* x.g2 * x.g9 * x.g9 - 8 * x.g4 * x.g9 * x.g9 - 4 * x.g5 * x.g9 * x.g9) "
)

# Per-population genotype features (pg_gpu genotype_kernels.py:412-492 and :176-197).
# x.ns = sum of the nine counts, x.n = n_valid (equal on the genotype path).
GENO_FEATURES = [
    ("xAB", "x.g1 + 0.5 * x.g2 + 0.5 * x.g4 + 0.25 * x.g5"),
    ("xAb", "0.5 * x.g2 + x.g3 + 0.25 * x.g5 + 0.5 * x.g6"),
    ("xaB", "0.5 * x.g4 + 0.25 * x.g5 + x.g7 + 0.5 * x.g8"),
    ("xab", "0.25 * x.g5 + 0.5 * x.g6 + 0.5 * x.g8 + x.g9"),
    ("D", "x.xAB * x.xab - x.xAb * x.xaB"),
    ("pA", "x.g1 + x.g2 + x.g3 + 0.5 * (x.g4 + x.g5 + x.g6)"),
    ("qA", "0.5 * (x.g4 + x.g5 + x.g6) + x.g7 + x.g8 + x.g9"),
    ("pB", "x.g1 + 0.5 * x.g2 + x.g4 + 0.5 * x.g5 + x.g7 + 0.5 * x.g8"),
    ("qB", "0.5 * x.g2 + x.g3 + 0.5 * x.g5 + x.g6 + 0.5 * x.g8 + x.g9"),
    ("BL", "(4 * x.pA * x.qA - (x.g4 + x.g5 + x.g6)) * x.inn1"),
    ("BR", "(4 * x.pB * x.qB - (x.g2 + x.g5 + x.g8)) * x.inn1"),
    ("C00", "(x.pA * x.pB - x.xAB) * x.inn1"),
    ("C01", "(x.pA * x.qB - x.xAb) * x.inn1"),
    ("C10", "(x.qA * x.pB - x.xaB) * x.inn1"),
    ("C11", "(x.qA * x.qB - x.xab) * x.inn1"),
    ("Bsgn", "x.xAB - x.xAb - x.xaB + x.xab"),
    ("p", "x.pA * x.invn"),
    ("r", "x.qA * x.invn"),
    ("q", "x.pB * x.invn"),
    ("s", "x.qB * x.invn"),
    ("L0", "x.g5 + 2 * x.g6 + 2 * x.g8 + 4 * x.g9"),
    ("AQ3", "-(x.qB * (3 * x.g4 + 3 * x.g5 + 3 * x.g6 + 4 * x.g7 + 4 * x.g8 + 4 * x.g9)) / 8"
            " + x.pA * x.qB * x.qA / 2 + (x.qA * x.L0) / 8 + (x.g5 + 2 * x.g6) / 8 - (x.pA * x.L0) / 8"),
    ("AS3", "-(x.pB * (5 * x.g4 + 5 * x.g5 + 5 * x.g6 + 8 * x.g7 + 8 * x.g8 + 8 * x.g9)) / 8"
            " + x.pA * x.pB * x.qA / 2"
            " + (x.qA * (-2 * x.g2 - 4 * x.g3 + 4 * x.g4 + x.g5 - 2 * x.g6 + 8 * x.g7 + 4 * x.g8 + 4)) / 8"
            " + (-x.g5 - 2 * x.g6 - 4 * x.g7 - 4 * x.g8 - 4 * x.g9) / 8 + (x.pA * x.L0) / 8"),
    ("BP3", "-(x.qA * (3 * x.g2 + 4 * x.g3 + 3 * x.g5 + 4 * x.g6 + 3 * x.g8 + 4 * x.g9)) / 8"
            " + x.pB * x.qB * x.qA / 2 + (x.qB * x.L0) / 8 + (x.g5 + 2 * x.g8) / 8 - (x.pB * x.L0) / 8"),
    ("BR3", "-(x.pA * (5 * x.g2 + 8 * x.g3 + 5 * x.g5 + 8 * x.g6 + 5 * x.g8 + 8 * x.g9)) / 8"
            " + x.pA * x.pB * x.qB / 2"
            " + (x.qB * (4 * x.g2 + 8 * x.g3 - 2 * x.g4 + x.g5 + 4 * x.g6 - 4 * x.g7 - 2 * x.g8 + 4)) / 8"
            " + (-4 * x.g3 - x.g5 - 4 * x.g6 - 2 * x.g8 - 4 * x.g9) / 8 + (x.pB * x.L0) / 8"),
    ("A", "-x.g1 + x.g3 - x.g4 + x.g6 - x.g7 + x.g9"),
    ("Bv", "-x.g1 - x.g2 - x.g3 + x.g7 + x.g8 + x.g9"),
    ("Wjj", "(-x.g1 + x.g3 + x.g7 - x.g9) + x.A * x.Bv"),
    ("U", "x.D * (1 + x.Bv) + 0.25 * (2 * x.g2 * x.g7 + 4 * x.g3 * x.g7 + 2 * x.g5 * x.g7"
          " + 4 * x.g6 * x.g7 - 2 * x.g1 * x.g8 + 2 * x.g3 * x.g8 - 2 * x.g4 * x.g8 + 2 * x.g6 * x.g8"
          " - 4 * x.g1 * x.g9 - 2 * x.g2 * x.g9 - 4 * x.g4 * x.g9 - 2 * x.g5 * x.g9)"),
    ("V", "x.D * (1 + x.A) + 0.25 * (2 * x.g3 * x.g4 + 2 * x.g3 * x.g5 - 2 * x.g1 * x.g6"
          " - 2 * x.g2 * x.g6 + 4 * x.g3 * x.g7 + 2 * x.g6 * x.g7 + 4 * x.g3 * x.g8 + 2 * x.g6 * x.g8"
          " - 4 * x.g1 * x.g9 - 4 * x.g2 * x.g9 - 2 * x.g4 * x.g9 - 2 * x.g5 * x.g9)"),
    # single-population statistics, numerators over ns(ns-1)(ns-2)(ns-3) (zero if ns < 4)
    ("DD1", "4 * ((" + GENO_DD_POLY + ") * 0.0625 + x.D * x.D) * x.w4"),
    ("DZ1", "2 * (0.25 * (" + GENO_DZ_QUARTIC + ") + x.A * x.Bv * x.D) * x.w4"),
    ("PI1", "(x.pA * x.pB * x.qB * x.qA + (" + GENO_PI2_CORR + ") * 0.0625) * x.w4"),
]


# The three single-population polynomials, as pg_gpu writes them, are sums of up to 155
# integer-coefficient monomials of degree <= 3 in the nine cell counts (~950 FP64 instructions
# per population and pair with a*b + c fused).  The generated code evaluates them in
# multivariate Horner form over g1, ..., g9 instead (~400): with integer counts every
# intermediate of either form is an integer, so FP64 gives the same value exactly while the
# intermediates stay below 2^53 (more than 10^4 individuals per population before that can
# fail; the expanded form has the same limit).  check() proves each Horner form equal to its
# polynomial.
_HORNER_POLYS = {"GENO_DD_POLY": GENO_DD_POLY, "GENO_DZ_QUARTIC": GENO_DZ_QUARTIC, "GENO_PI2_CORR": GENO_PI2_CORR}


def _horner_sympy(poly):
    import sympy as sp
    from sympy.polys.polyfuncs import horner
    g = sp.symbols("g1:10")
    loc = {f"g{i + 1}": g[i] for i in range(9)}
    e = sp.expand(sp.sympify(poly.replace("x.g", "g"), locals=loc))
    return e, horner(e, *g), g


@functools.lru_cache(maxsize=None)
def horner_form(poly):
    """``poly`` (a polynomial string in x.g1 .. x.g9) in multivariate Horner form, as an
    expression string in the same variables (C and Python syntax)."""
    import re
    _, h, _ = _horner_sympy(poly)
    out = re.sub(r"\bg(\d)\b", r"x.g\1", str(h))
    if "**" in out:
        raise ValueError("power left in a Horner form")
    return out


@functools.lru_cache(maxsize=None)
def geno_features():
    """GENO_FEATURES with the three single-population polynomials in Horner form (the form
    the generated code and the NumPy evaluation use)."""
    out = []
    for n, e in GENO_FEATURES:
        for poly in _HORNER_POLYS.values():
            e = e.replace("(" + poly + ")", "(" + horner_form(poly) + ")")
        out.append((n, e))
    for n in ("DD1", "DZ1", "PI1"):
        e = dict(out)[n]
        if any(poly in e for poly in _HORNER_POLYS.values()):
            raise ValueError(f"{n}: polynomial not replaced")
    return out


def geno_call_expr(case, args):
    """Expression of one canonical raw genotype call (genotype_kernels.py:27-405)."""
    f = lambda p, name: f"f[{p}].{name}"  # noqa: E731
    if case == "dd1":
        return f(args[0], "DD1")
    if case == "dd2":
        i, j = args
        return f"4 * ({f(i,'D')} * {f(j,'D')}) * ({f(i,'r2')} * {f(j,'r2')})"
    if case == "dz_iii":
        return f(args[0], "DZ1")
    if case == "dz_iij":
        i, j = args
        return f"(2 * {f(i,'U')} * {f(j,'A')}) * ({f(i,'u3')} * {f(j,'u1')})"
    if case == "dz_iji":
        i, j = args
        return f"(2 * {f(i,'V')} * {f(j,'Bv')}) * ({f(i,'u3')} * {f(j,'u1')})"
    if case == "dz_ijj":
        i, j = args
        return f"(2 * {f(i,'D')} * {f(j,'Wjj')}) * ({f(j,'u2')} * {f(i,'u2')})"
    if case == "dz_ijk":
        i, j, k = args
        return f"(2 * {f(i,'D')} * {f(j,'Bv')} * {f(k,'A')}) * ({f(i,'u2')} * {f(j,'u1')} * {f(k,'u1')})"
    if case == "pi2_same":
        return f(args[0], "PI1")
    if case == "pi2_alldiff":
        i, j, k, l = args
        return (f"0.25 * ({f(i,'p')} * {f(j,'r')} + {f(i,'r')} * {f(j,'p')})"
                f" * ({f(k,'q')} * {f(l,'s')} + {f(k,'s')} * {f(l,'q')})")
    if case == "pi2_iikk":
        i, k = args
        return f"{f(i,'BL')} * {f(k,'BR')}"
    if case == "pi2_iikl":
        i, k, l = args
        return f"{f(i,'BL')} * 0.5 * ({f(k,'q')} * {f(l,'s')} + {f(k,'s')} * {f(l,'q')})"
    if case == "pi2_ijkk":
        i, j, k = args
        return f"0.5 * ({f(i,'p')} * {f(j,'r')} + {f(i,'r')} * {f(j,'p')}) * {f(k,'BR')}"
    if case == "pi2_shared":
        s, a, b = args
        return (f"{f(a,'r')} * ({f(s,'C00')} * {f(b,'s')} + {f(s,'C01')} * {f(b,'q')})"
                f" + {f(a,'p')} * ({f(s,'C10')} * {f(b,'s')} + {f(s,'C11')} * {f(b,'q')})")
    if case == "pi2_iiij":
        t, s = args
        return (f"({f(t,'AQ3')} * {f(s,'pB')} + {f(t,'AS3')} * {f(s,'qB')})"
                f" * ({f(t,'r3')} * {f(s,'r1')})")
    if case == "pi2_ijii":
        t, s = args
        return (f"({f(t,'BP3')} * {f(s,'pA')} + {f(t,'BR3')} * {f(s,'qA')})"
                f" * ({f(t,'r3')} * {f(s,'r1')})")
    if case == "pi2_ijij":
        i, j = args
        P_i, Q_i, R_i, S_i = f(i, "pA"), f(i, "pB"), f(i, "qA"), f(i, "qB")
        P_j, Q_j, R_j, S_j = f(j, "pA"), f(j, "pB"), f(j, "qA"), f(j, "qB")
        X01i, X10i, X11i, Bi = f(i, "xAb"), f(i, "xaB"), f(i, "xab"), f(i, "Bsgn")
        X11j, X01j, Bj = f(j, "xab"), f(j, "xAb"), f(j, "Bsgn")
        num = (f"-0.25 * ({R_i} * {S_i}) * {Q_j} - 0.25 * {X11i} * ({P_j} * {Q_j})"
               f" + 0.25 * ({R_i} * {S_i}) * ({P_j} * {Q_j}) - 0.25 * {R_i} * ({P_j} * {S_j})"
               f" - 0.25 * ({P_i} * {Q_i}) * {X11j} - 0.25 * ({R_i} * {S_i}) * {X11j}"
               f" + 0.25 * ({P_i} * {S_i}) * {X11j} + 0.25 * ({Q_i} * {R_i}) * {X11j}"
               f" - 0.25 * ({P_i} * {R_i}) * {S_j} + 0.25 * ({R_i} * (1 + {X01i} - {X10i})) * {S_j}"
               f" + 0.25 * {X11i} * ({P_j} * {S_j}) + 0.25 * ({Q_i} * {R_i}) * ({P_j} * {S_j})"
               f" + 0.25 * ({S_i} * (1 + {R_i})) * {R_j} - 0.25 * {X01i} * ({Q_j} * {R_j})"
               f" + 0.25 * ({P_i} * {S_i}) * ({Q_j} * {R_j})"
               f" - 0.25 * ({P_i} * {S_i}) * {R_j} - 0.25 * {P_i} * ({R_j} * {S_j})"
               f" + 0.25 * {X01i} * ({R_j} * {S_j}) + 0.25 * ({P_i} * {Q_i}) * ({R_j} * {S_j})"
               f" + 0.25 * {X11i} * {Bj} + 0.25 * {Bi} * {X11j} - {X11i} * {X11j}")
        _ = X01j
        return f"({num}) * ({f(i,'r2')} * {f(j,'r2')})"
    raise ValueError(case)


def geno_features_needed(P):
    calls, _ = plan(P, geno=True)
    need = {"DD1", "DZ1", "PI1"}
    per_case = {
        "dd2": ["D"], "dz_iij": ["U", "A"], "dz_iji": ["V", "Bv"], "dz_ijj": ["D", "Wjj"],
        "dz_ijk": ["D", "Bv", "A"], "pi2_alldiff": ["p", "r", "q", "s"], "pi2_iikk": ["BL", "BR"],
        "pi2_iikl": ["BL", "q", "s"], "pi2_ijkk": ["p", "r", "BR"],
        "pi2_shared": ["r", "p", "s", "q", "C00", "C01", "C10", "C11"],
        "pi2_iiij": ["AQ3", "AS3", "pB", "qB"], "pi2_ijii": ["BP3", "BR3", "pA", "qA"],
        "pi2_ijij": ["pA", "pB", "qA", "qB", "xAb", "xaB", "xab", "Bsgn"],
    }
    for case, _ in calls:
        need.update(per_case.get(case, []))
    order = [n for n, _ in GENO_FEATURES]
    changed = True
    while changed:
        changed = False
        for n, e in GENO_FEATURES:
            if n in need:
                for d in order:
                    if f"x.{d}" in e.replace("x.g", "x.#") and d not in need:
                        need.add(d)
                        changed = True
    return [n for n in order if n in need]


def emit_geno(P):
    feats = geno_features_needed(P)
    calls, stats = plan(P, geno=True)
    L = [f"// genotype path, P = {P}: {len(stats)} statistics from {len(calls)} distinct raw calls",
         "template <typename T, bool PREP = true>", f"LDK_DEV void geno_features_P{P}(GenoFeat<T>& x) {{",
         "    if constexpr (PREP) geno_prepare(x);"]
    for n, e in geno_features():
        if n in feats:
            L.append(f"    x.{n} = {_cexpr(e)};")
    L.append("}")
    L.append("template <typename T, int S = 1>")
    L.append(f"LDK_DEV void geno_stats_P{P}(const GenoFeat<T>* f, T* acc) {{")
    for ci, (case, args) in enumerate(calls):
        L.append(f"    const T v{ci} = {_cexpr(geno_call_expr(case, args))};  // {case}{args}")
    for si, (name, terms) in enumerate(stats):
        groups = {}
        for idx, w in terms:
            groups.setdefault(w, []).append(f"v{idx}")
        parts = []
        for w, vs in sorted(groups.items(), reverse=True):
            sw = _fmt_weight(w)
            body = " + ".join(vs)
            parts.append(body if sw is None else f"T({sw}) * ({body})")
        L.append(f"    acc[{si} * S] += {' + '.join(parts)};  // {name}")
    L.append("}")
    return "\n".join(L)


def numpy_geno_stats(counts9_list, n_list=None):
    """Evaluate the generated genotype expressions with NumPy float64 (test helper)."""
    import numpy as np
    P = len(counts9_list)
    fs = []
    for p, c in enumerate(counts9_list):
        c = np.asarray(c, dtype=np.float64)
        x = _NS()
        for m in range(9):
            setattr(x, f"g{m + 1}", c[:, 8 - m])
        x.ns = c.sum(axis=1)
        x.n = x.ns if (n_list is None or n_list[p] is None) else np.asarray(n_list[p], np.float64)
        with np.errstate(divide="ignore", invalid="ignore"):
            n, ns = x.n, x.ns
            x.inn1 = 1.0 / np.maximum(4 * n * (n - 1), 1)
            x.invn = 1.0 / n
            d1, d2 = n, n * (n - 1)
            d3 = d2 * (n - 2)
            x.r1 = np.where(d1 > 0, 1 / np.where(d1 > 0, d1, 1), 0.0)
            x.r2 = np.where(d2 > 0, 1 / np.where(d2 > 0, d2, 1), 0.0)
            x.r3 = np.where(d3 > 0, 1 / np.where(d3 > 0, d3, 1), 0.0)
            x.u1 = 1.0 / ns
            x.u2 = 1.0 / (ns * (ns - 1))
            x.u3 = 1.0 / (ns * (ns - 1) * (ns - 2))
            w4 = ns * (ns - 1) * (ns - 2) * (ns - 3)
            x.w4 = np.where(ns >= 4, 1 / np.where(ns >= 4, w4, 1), 0.0)
            for name, e in geno_features():
                setattr(x, name, eval(e, {}, {"x": x}))
        fs.append(x)
    calls, stats = plan(P, geno=True)
    with np.errstate(divide="ignore", invalid="ignore"):
        vals = [eval(geno_call_expr(case, args), {}, {"f": fs}) for case, args in calls]
    out = np.zeros((len(fs[0].g1), len(stats)))
    for si, (_, terms) in enumerate(stats):
        for idx, w in terms:
            out[:, si] += w * vals[idx]
    return out

# ---------------------------------------------------------------------------
# code emission
# ---------------------------------------------------------------------------


def _fmt_weight(w):
    return {1.0: None, 0.5: "0.5", 0.25: "0.25", 0.125: "0.125", 0.75: "0.75"}.get(w, repr(w))


def emit_hap(P):
    feats, recips = hap_features_needed(P)
    calls, stats = plan(P)
    L = []
    L.append(f"// P = {P}: {len(stats)} statistics from {len(calls)} distinct raw calls")
    L.append("template <typename T>")
    L.append(f"LDK_DEV void hap_features_P{P}(HapFeat<T>& x) {{")
    for n, e in HAP_FEATURES:
        if n in feats:
            L.append(f"    x.{n} = {_cexpr(e)};")
    L.append("}")
    # every statistic, and (four populations) the halves that two warps share as in spin_order
    order, K = spin_order(P, False)
    halves = [("template <typename T, int S = 1>", f"hap_stats_P{P}", range(len(stats)), " * S")]
    if K:
        halves += [("template <typename T>", f"hap_half_P{P}_{h}", mine, "") for h, mine in ((1, order[:K]), (2, order[K:]))]
    for head, fn, mine, stride in halves:
        mine = list(mine)
        used = {idx for si in mine if si < len(stats) for idx, _ in stats[si][1]}
        L.append(head)
        L.append(f"LDK_DEV void {fn}(const HapFeat<T>* f, T* acc) {{")
        for ci, (case, args) in enumerate(calls):
            if ci in used:
                L.append(f"    const T v{ci} = {_cexpr(hap_call_expr(case, args))};  // {case}{args}")
        for at, si in enumerate(mine):
            if si == len(stats):
                continue  # r^2: the caller's
            name, terms = stats[si]
            groups = {}
            for idx, w in terms:
                groups.setdefault(w, []).append(f"v{idx}")
            parts = []
            for w, vs in sorted(groups.items(), reverse=True):
                sw = _fmt_weight(w)
                body = " + ".join(vs)
                parts.append(body if sw is None else f"T({sw}) * ({body})")
            L.append(f"    acc[{at}{stride}] += {' + '.join(parts)};  // {name}")
        L.append("}")
    return "\n".join(L)


# ---------------------------------------------------------------------------
# fused-path forms (tensor-core parse)
# ---------------------------------------------------------------------------
#
# Spin moments.  Let sigma = 1 - 2a, a being the individual's frequency of allele 1 at the
# left SNP (haplotypes: 0 or 1; genotypes: half the dosage, so sigma = 1 - g), tau the same
# at the right SNP, both 0 where the call is missing.  The tensor-core kernel counts the
# sums over a population's jointly called individuals
#   n,  S = sum sigma,  T = sum tau,  R = sum sigma tau,
#   (genotypes) SS = sum sigma^2, TT, SST = sum sigma^2 tau, STT, SSTT,
# and every statistic is an unbiased mean over distinct individuals of products of sigma and
# tau (a U-statistic), i.e. a polynomial of these integers over n(n-1)..., for both paths:
#   E  = n R - S T            = sum over k != l of sigma_k (tau_k - tau_l)   (4 x / -D)
#   W  = S T - R              = sum over k != l of sigma_k tau_l
#   u  = S^2 - SS, v = T^2 - TT;   hA = n(n-1) - u, hB = n(n-1) - v   (heterozygosities)
#   Q2 = R^2 - SSTT           = sum over k != m of sigma_k tau_k sigma_m tau_m
#   Q3 = R W - S STT - T SST + 2 SSTT   = sum over distinct k, m, o of sigma_k tau_k sigma_m tau_o
#   Q4 = u v - 4 Q3 - 2 Q2    = sum over distinct k, m, l, o of sigma_k sigma_m tau_l tau_o
# (the pairs {k, m} and {l, o} of u v overlap in one index in four ways, in both in two).
# A haplotype has sigma^2 = 1, so SS = TT = SSTT = n, SST = T, STT = S and Q3 = R W - u - v.
# All numerators are integers and no intermediate of theirs exceeds 8 N^4 in populations of at
# most N, so up to N = SPIN_MAX_N = 5,792 (8 N^4 <= 2^53) FP64 holds them exactly and a statistic
# that is exactly zero stays zero; each is scaled by the tabulated reciprocals and added with one
# FMA.  The constant factors (powers of two) are applied once per staged sum (SPIN weights), not
# per pair.  ``check()`` proves the forms equal to the raw calls.
#
# Above SPIN_MAX_N the n^4 terms would cancel to rounding remainders where the alleles are rare
# (DD of singletons 1e-7 off at n = 100,000, sigma_D^2 = 1 where both numerators are 0), so the
# kernels recover the two-locus counts from the moments (HAP_CELLS, GENO_CELLS: exact) and
# evaluate the raw calls on them, whose terms are as small as the rare counts.
#
# Expressions are C and Python syntax over the names below, suffixed with the population.

SPIN_MAX_N = 5792
SPIN_INPUTS = ["n", "S", "T", "R", "r1", "r2", "r3", "r4"]
SPIN_INPUTS_GENO = SPIN_INPUTS + ["SS", "TT", "SST", "STT", "SSTT"]
# counts n11, n10, n01, n00 and n00, n01, ..., n22 (genotypes; column g_i * 3 + g_j) of the moments:
# [x = 1] = (1 - sigma) / 2; [g = 0] = (sigma^2 + sigma) / 2, [g = 1] = 1 - sigma^2, [g = 2] = (sigma^2 - sigma) / 2
HAP_CELLS = ["0.25 * ((n - S) - (T - R))", "0.25 * ((n - S) + (T - R))", "0.25 * ((n + S) - (T + R))",
             "0.25 * ((n + S) + (T + R))"]
GENO_CELLS = ["0.25 * ((SSTT + R) + (SST + STT))", "0.5 * ((SS + S) - (SSTT + STT))", "0.25 * ((SSTT - R) - (SST - STT))",
              "0.5 * ((TT + T) - (SSTT + SST))", "(n - SS) - (TT - SSTT)", "0.5 * ((TT - T) - (SSTT - SST))",
              "0.25 * ((SSTT - R) + (SST - STT))", "0.5 * ((SS - S) - (SSTT - STT))", "0.25 * ((SSTT + R) - (SST + STT))"]


def _spin_pop(p, geno):
    """Definitions (name, expression) of population p's features."""
    d = [
        ("m", "n# - 1.0"), ("nu", "n# * m#"), ("nux", "nu# + nu#"), ("ST", "S# * T#"), ("E", "fma(n#, R#, -ST#)"),
        ("W", "ST# - R#"), ("u", "fma(S#, S#, -SS#)" if geno else "fma(S#, S#, -n#)"),
        ("v", "fma(T#, T#, -TT#)" if geno else "fma(T#, T#, -n#)"), ("hA", "nu# - u#"), ("hB", "nu# - v#"),
        ("uv", "u# + v#"), ("n2", "n# - 2.0"), ("n3", "n# - 3.0"),
        ("Q2", "fma(R#, R#, -SSTT#)" if geno else "fma(R#, R#, -n#)"),
        ("Q3", "fma(-T#, SST#, fma(-S#, STT#, fma(R#, W#, SSTT# + SSTT#)))" if geno else "fma(R#, W#, -uv#)"),
        ("Qx", "Q3# + Q3#"), ("Q4", "fma(-2.0, Qx# + Q2#, u# * v#)"),
        ("DD", "fma(n3#, fma(n2#, Q2#, -Qx#), Q4#)"), ("DZ", "fma(n3#, Q3#, -Q4#)"),
        ("PI", "fma(n2# * n3#, nu# - uv#, Q4#)"),
        ("De", "E# * r2#"), ("Er", "E# * r3#"),
        ("U", "fma(n#, fma(R#, S#, -SST#), -(u# * T#)) * r3#" if geno else "S# * Er#"),
        ("V", "fma(n#, fma(R#, T#, -STT#), -(v# * S#)) * r3#" if geno else "T# * Er#"),
        ("al", "S# * r1#"), ("be", "T# * r1#"), ("w", "W# * r2#"), ("hAr", "hA# * r2#"), ("hBr", "hB# * r2#"),
        ("Sm", "m# * S#"), ("Tm", "m# * T#"),
        # pi2 with one population three times: (X n_s - Y T_s [- Yb S_s]) r3 r1_s
        ("P", "fma(R#, S#, -SST#)" if geno else "fma(R#, S#, -T#)"), ("Y", "fma(fma(-2.0, m#, hA#), T#, P# + P#)"),
        ("X", "n2# * (hA# + hB#)" if geno else "n2# * hA#"),
        ("Pb", "fma(R#, T#, -STT#)" if geno else "fma(R#, T#, -S#)"), ("Yb", "fma(fma(-2.0, m#, hB#), S#, Pb# + Pb#)"),
        # variances behind r^2 (of population 0)
        ("vx", "fma(n#, SS#, -(S# * S#))" if geno else "hA#"), ("vy", "fma(n#, TT#, -(T# * T#))" if geno else "hB#"),
    ]
    return [(n + str(p), e.replace("#", str(p))) for n, e in d]


def _spin_pair(i, j):
    """Definitions of the pair (i < j): symmetric products, suffix ij."""
    d = [("rr", "r2I * r2J"), ("rho", "r1I * r1J"), ("nn", "nI * nJ"), ("HA", "fma(-SI, SJ, nn@)"),
         ("HB", "fma(-TI, TJ, nn@)"), ("K", "fma(SI, TJ, SJ * TI)"), ("Kr", "K@ * rho@"),
         ("La", "fma(SI, nJ, SJ * nI)"), ("Lb", "fma(TI, nJ, TJ * nI)")]
    k = f"{i}{j}"
    return [(n + k, e.replace("r1I", f"r1{i}").replace("r1J", f"r1{j}").replace("r2I", f"r2{i}")
             .replace("r2J", f"r2{j}").replace("SI", f"S{i}").replace("SJ", f"S{j}").replace("TI", f"T{i}")
             .replace("TJ", f"T{j}").replace("nI", f"n{i}").replace("nJ", f"n{j}").replace("@", k)) for n, e in d]


def spin_defs(P, geno):
    d = {}
    for p in range(P):
        d.update(_spin_pop(p, geno))
    for i in range(P):
        for j in range(i + 1, P):
            d.update(_spin_pair(i, j))
    return d


def spin_stats(P, geno):
    """[(name, weight, [(A, B), ...], rank)]: the statistic is weight * sum of A * B; rank
    orders the emission (single populations, pairs, triples, quadruples)."""
    c = 2.0 if geno else 1.0  # the genotype D is the composite one, twice as large
    pr = lambda a, b: f"{min(a, b)}{max(a, b)}"  # noqa: E731
    out = []
    for kind, q in ld_names(P):
        pops = sorted(set(q))
        rank = (len(pops), pops)
        if kind == "dd":
            i, j = q
            t = (c * c / 16, [(f"DD{i}", f"r4{i}")] if i == j else [(f"De{i}", f"De{j}")])
        elif kind == "dz":
            i, j, k = q
            if i == j == k:
                t = (c / 4, [(f"DZ{i}", f"r4{i}")])
            elif j == k:
                t = (c / 4, [(f"De{i}", f"w{j}")])
            elif i in (j, k):
                o = k if i == j else j
                t = (c / 8, [(f"U{i}", f"be{o}"), (f"V{i}", f"al{o}")])
            else:
                t = (c / 8, [(f"De{i}", f"Kr{pr(j, k)}")])
        else:
            i, j, k, l = q
            case = _pi2_case(q)
            if case == "same":
                t = (1 / 16, [(f"PI{i}", f"r4{i}")])
            elif case == "iikk":
                t = (1 / 32, [(f"hAr{i}", f"hBr{k}"), (f"hBr{i}", f"hAr{k}")])
            elif case == "triple":
                cnt = _counts_of(q)
                a = [x for x, m in cnt.items() if m == 3][0]
                s = [x for x, m in cnt.items() if m == 1][0]
                num = f"fma(-Y{a}, T{s}, X{a} * n{s})"
                if geno:
                    num = f"fma(-Yb{a}, S{s}, {num})"
                t = (1 / 32 if geno else 1 / 16, [(num, f"(r3{a} * r1{s})")])
            elif case in ("iikl", "ijkk"):
                a, x, y = (i, k, l) if i == j else (k, i, j)
                t = (1 / 32, [(f"fma(hAr{a}, HB{pr(x, y)}, hBr{a} * HA{pr(x, y)})", f"rho{pr(x, y)}")])
            elif case == "ijij":
                t = (1 / 16, [(f"fma(-Sm{i}, Sm{j}, fma(-Tm{i}, Tm{j}, fma(W{i}, W{j}, nu{i} * nu{j})))", f"rr{pr(i, j)}")])
                # Sm = (n - 1) S on both sides would carry (n_i - 1)(n_j - 1): exactly the form's factor
            elif case == "shared":
                s = [x for x in (i, j) if x in (k, l)][0]
                x, y = (j if i == s else i), (l if k == s else k)
                g = pr(x, y)
                t = (1 / 32, [(f"fma(W{s}, K{g}, fma(-Tm{s}, Lb{g}, fma(-Sm{s}, La{g}, nux{s} * nn{g})))",
                               f"(r2{s} * rho{g})")])
            else:
                a, b = pr(i, j), pr(k, l)
                t = (1 / 32, [(f"fma(HA{a}, HB{b}, HA{b} * HB{a})", f"(rho{a} * rho{b})")])
        out.append((stat_name(kind, q), t[0], t[1], rank))
    return out


def spin_order(P, geno):
    """(order, K): the statistics in the order they are staged (r^2 is index NS) and, for four
    haplotype populations, where two epilogue warps that share a pair split them: [0, K)
    holds DD, Dz, the one-population pi2 (all from Q2, Q3, Q4) and r^2, the rest the other
    pi2, so that the halves need nearly disjoint features.  K = 0: one warp takes all."""
    names = ld_names(P)
    if geno or P < 4:
        return list(range(len(names) + 1)), 0
    first = [k for k, (kind, q) in enumerate(names) if kind != "pi2" or len(set(q)) == 1] + [len(names)]
    return first + [k for k in range(len(names)) if k not in first], len(first)


def _names_in(e):
    import re
    return re.findall(r"[A-Za-z]\w*", e)


def emit_spin(P, geno):
    """spin_{hap,geno}_P{P}_{part}: part 0 = all statistics and r^2; with a split, part 1 =
    staged sums [0, K) and part 2 = [K, NS]."""
    path = "geno" if geno else "hap"
    defs, stats, (order, K) = spin_defs(P, geno), spin_stats(P, geno), spin_order(P, geno)
    inputs = SPIN_INPUTS_GENO if geno else SPIN_INPUTS
    NS = len(stats)
    L = [f"// {path}, P = {P}: {NS} statistics" + (f", split at {K}" if K else "")]
    for part, mine in ({1: order[:K], 2: order[K:]} if K else {0: order}).items():
        lines, done = [], set()

        def use(expr):
            for nm in _names_in(expr):
                if nm in done or nm == "fma":
                    continue
                done.add(nm)
                if nm in defs:
                    use(defs[nm])
                    lines.append(f"    const double {nm} = {defs[nm]};")
                else:
                    base = nm.rstrip("0123456789") if not nm.startswith("r") else nm[:2]
                    assert base in inputs, nm
                    lines.append(f"    const double {nm} = f[{nm[-1]}].{base};")

        for si in sorted((k for k in mine if k < NS), key=lambda k: stats[k][3]):
            name, _, terms, _ = stats[si]
            at = mine.index(si)
            for A, B in terms:
                use(A)
                use(B)
                lines.append(f"    acc[{at}] = fma({A}, {B}, acc[{at}]);  // {name}")
        if NS in mine:
            at = mine.index(NS)
            use("E0 vx0 vy0")
            lines += ["    const double den = vx0 * vy0;", "    const bool has = ok && den > 0.0;",
                      f"    acc[{at}] = fma(E0 * E0, has ? recip_cubic(den) : 0.0, acc[{at}]);", "    nr2 += has;"]
        L.append(f"LDK_DEV void spin_{path}_P{P}_{part}(const SpinPop* f, bool ok, double* acc, unsigned& nr2) {{")
        L += lines
        L.append("}")
    w = [x[1] for x in stats] + [1.0]
    L.append(f"static __constant__ double spin_weight_{path}_P{P}[{NS + 1}] = {{{', '.join(repr(w[k]) for k in order)}}};")
    if K:
        L.append(f"static __constant__ int spin_stat_{path}_P{P}[{NS + 1}] = {{{', '.join(map(str, order))}}};")
    return "\n".join(L)


def emit_spin_numerators(geno):
    """The DD and pi2 numerators of one population (16 times each, over n(n-1)(n-2)(n-3))."""
    defs, lines, done = spin_defs(1, geno), [], set()

    def use(expr):
        for nm in _names_in(expr):
            if nm in done or nm == "fma":
                continue
            done.add(nm)
            if nm in defs:
                use(defs[nm])
                lines.append(f"    const double {nm} = {defs[nm]};")

    use("DD0 PI0")
    if geno:
        head = ["LDK_DEV void spin_geno_numerators(const uint32_t (&G)[3][4], double& dd, double& pi2) {"]
        cells = {"R": (0, 0), "STT": (0, 1), "S": (0, 2), "SST": (1, 0), "SSTT": (1, 1), "SS": (1, 2), "T": (2, 0),
                 "TT": (2, 1), "n": (2, 2)}
        head += [f"    const double {k}0 = i2d_exact((int)G[{x}][{y}]);" for k, (x, y) in cells.items() if f"{k}0" in done]
    else:
        head = ["LDK_DEV void spin_hap_numerators(double n0, double S0, double T0, double R0, double& dd, double& pi2) {"]
    return "\n".join(head + lines + ["    dd = DD0;", "    pi2 = PI0;", "}"])


def emit_cells():
    """The two-locus counts of a population's moments."""
    import re
    members = lambda e: re.sub(r"[A-Z]+\b|\bn\b", lambda m: "m." + m.group(0), e)  # noqa: E731
    L = [f"constexpr int kSpinMaxN = {SPIN_MAX_N};  // largest population of the spin forms",
         "LDK_DEV void spin_hap_cells(const SpinPop& m, double (&c)[4]) {"]
    L += [f"    c[{k}] = {members(e)};" for k, e in enumerate(HAP_CELLS)]
    L += ["}", "LDK_DEV void spin_geno_cells(const SpinPop& m, double (&c)[9]) {"]
    L += [f"    c[{k}] = {members(e)};" for k, e in enumerate(GENO_CELLS)]
    return "\n".join(L + ["}"])


def _cexpr(e):
    """Numeric literals as T(...) so float and double instantiations stay exact."""
    import re
    return re.sub(r"(?<![\w.\[])(\d+\.\d+|\d+)(?![\w.\]])", lambda m: f"T({m.group(1)})", e)


HEADER = """// GENERATED by gen_estimators.py -- do not edit by hand.
//
// Straight-line two-locus LD estimators for P = 1..4 populations (haplotype path).
// Statistic order and averaging weights follow moments.LD (pg_gpu ld_pipeline.py:357-457);
// raw-call algebra restates pg_gpu haplotype_kernels.py:69-304 in factored form.
// hap_stats_P* / geno_stats_P* evaluate every distinct raw call (plain kernel, raw-call entry
// points, tensor-core parse of populations above kSpinMaxN); spin_hap_P* / spin_geno_P* are the
// statistic-level forms of the tensor-core parse.
#pragma once
"""


def generate(path=None):
    path = path or os.path.join(HERE, "ldk_estimators.cuh")
    parts = [HEADER, '#include "ldk_hap_feat.cuh"', ""]
    for P in (1, 2, 3, 4):
        parts.append(emit_hap(P))
        parts.append("")
    parts.append('#include "ldk_geno_feat.cuh"\n#include "ldk_spin.cuh"')
    for P in (1, 2, 3, 4):
        parts.append(emit_geno(P))
        parts.append("")
    for geno in (False, True):
        for P in (1, 2, 3, 4):
            parts.append(emit_spin(P, geno))
            parts.append("")
    for geno in (False, True):
        parts.append(emit_spin_numerators(geno))
        parts.append("")
    parts.append(emit_cells())
    parts.append("")
    parts.append(emit_raw_dispatch())
    parts.append("")
    parts.append("template <int P> struct HapNStats;")
    for P in (1, 2, 3, 4):
        parts.append(f"template <> struct HapNStats<{P}> {{ static constexpr int value = {len(stat_specs(P))}; }};")
    parts.append("// staged sums of the first of two warps that share a pair (haplotypes), 0: no split")
    parts.append("template <int P> struct SpinSplit;")
    for P in (1, 2, 3, 4):
        parts.append(f"template <> struct SpinSplit<{P}> {{ static constexpr int value = {spin_order(P, False)[1]}; }};")
    parts.append("""
template <typename T, int P>
LDK_DEV void hap_features(HapFeat<T>& x) {
    if constexpr (P == 1) hap_features_P1<T>(x);
    else if constexpr (P == 2) hap_features_P2<T>(x);
    else if constexpr (P == 3) hap_features_P3<T>(x);
    else hap_features_P4<T>(x);
}
template <typename T, int P, int S = 1>
LDK_DEV void hap_stats(const HapFeat<T>* f, T* acc) {
    if constexpr (P == 1) hap_stats_P1<T, S>(f, acc);
    else if constexpr (P == 2) hap_stats_P2<T, S>(f, acc);
    else if constexpr (P == 3) hap_stats_P3<T, S>(f, acc);
    else hap_stats_P4<T, S>(f, acc);
}
template <typename T, int P, bool PREP = true>
LDK_DEV void geno_features(GenoFeat<T>& x) {
    if constexpr (P == 1) geno_features_P1<T, PREP>(x);
    else if constexpr (P == 2) geno_features_P2<T, PREP>(x);
    else if constexpr (P == 3) geno_features_P3<T, PREP>(x);
    else geno_features_P4<T, PREP>(x);
}
template <typename T, int P, int S = 1>
LDK_DEV void geno_stats(const GenoFeat<T>* f, T* acc) {
    if constexpr (P == 1) geno_stats_P1<T, S>(f, acc);
    else if constexpr (P == 2) geno_stats_P2<T, S>(f, acc);
    else if constexpr (P == 3) geno_stats_P3<T, S>(f, acc);
    else geno_stats_P4<T, S>(f, acc);
}
// Spin-form statistics of part PART (0: all and r^2; four haplotype populations:
// 1 and 2, the two halves) added into acc[0 ..) of that part, before their weights.  A pair that
// does not count (!ok) has its reciprocals set to 0 by the caller; r^2 looks at ok itself.
template <int P, bool GENO, int PART>
LDK_DEV void spin_stats(const SpinPop* f, bool ok, double* acc, unsigned& nr2) {
    if constexpr (GENO) {
        if constexpr (P == 1) spin_geno_P1_0(f, ok, acc, nr2);
        else if constexpr (P == 2) spin_geno_P2_0(f, ok, acc, nr2);
        else if constexpr (P == 3) spin_geno_P3_0(f, ok, acc, nr2);
        else spin_geno_P4_0(f, ok, acc, nr2);
    } else {
        if constexpr (P == 1) spin_hap_P1_0(f, ok, acc, nr2);
        else if constexpr (P == 2) spin_hap_P2_0(f, ok, acc, nr2);
        else if constexpr (P == 3) spin_hap_P3_0(f, ok, acc, nr2);
        else if constexpr (PART == 1) spin_hap_P4_1(f, ok, acc, nr2);
        else spin_hap_P4_2(f, ok, acc, nr2);
    }
}
// The same statistics, weights applied, from the counts behind the moments: populations of more
// than kSpinMaxN.  The caller sets the pair's n and reciprocals.
template <int P, bool GENO, int PART>
LDK_DEV void count_stats(const SpinPop* m, double* acc, unsigned& nr2) {
    constexpr int NS = HapNStats<P>::value;
    if constexpr (GENO) {
        GenoFeat<double> f[P];
#pragma unroll
        for (int p = 0; p < P; ++p) {
            double c[9];
            spin_geno_cells(m[p], c);
            geno_set_counts(f[p], c);
            f[p].n = m[p].n;
            if constexpr (P < 4) {
                geno_prepare_from(f[p], m[p].r1, m[p].r2, m[p].r3, m[p].r4);
                geno_features<double, P, false>(f[p]);
            } else {  // four populations divide: the table's registers double their spill
                geno_features<double, P>(f[p]);
            }
        }
        geno_stats<double, P>(f, acc);
        const double E = fma(m[0].n, m[0].R, -(m[0].S * m[0].T));
        const double den = fma(m[0].n, m[0].SS, -(m[0].S * m[0].S)) * fma(m[0].n, m[0].TT, -(m[0].T * m[0].T));
        if (den > 0.0) {
            acc[NS] = fma(E * E, recip_cubic(den), acc[NS]);
            ++nr2;
        }
    } else {
        HapFeat<double> f[P];
#pragma unroll
        for (int p = 0; p < P; ++p) {
            double c[4];
            spin_hap_cells(m[p], c);
            hap_set_counts(f[p], c[0], c[1], c[2], c[3]);
            f[p].r1 = m[p].r1;
            f[p].r2 = m[p].r2;
            f[p].r3 = m[p].r3;
            f[p].r4 = m[p].r4;
            hap_features<double, P>(f[p]);
        }
        constexpr int R2 = PART == 1 ? SpinSplit<P>::value - 1 : NS;  // where r^2 is staged
        if constexpr (PART == 0) hap_stats<double, P>(f, acc);
        else if constexpr (PART == 1) hap_half_P4_1<double>(f, acc);
        else hap_half_P4_2<double>(f, acc);
        double r2;
        if (PART != 2 && hap_r2(f[0], r2)) {
            acc[R2] += r2;
            ++nr2;
        }
    }
}
// Weight and statistic (number of statistics: r^2, weight 1) of staged sum s.
template <int P, bool GENO>
LDK_DEV double spin_weight(int s) {
    if constexpr (GENO)
        return P == 1 ? spin_weight_geno_P1[s] : P == 2 ? spin_weight_geno_P2[s] : P == 3 ? spin_weight_geno_P3[s] : spin_weight_geno_P4[s];
    else
        return P == 1 ? spin_weight_hap_P1[s] : P == 2 ? spin_weight_hap_P2[s] : P == 3 ? spin_weight_hap_P3[s] : spin_weight_hap_P4[s];
}
template <int P, bool GENO>
LDK_DEV int spin_stat(int s) {
    if constexpr (GENO || P < 4) return s;
    else return spin_stat_hap_P4[s];
}
""")
    text = "\n".join(parts)
    with open(path, "w") as fh:
        fh.write(text)
    return path


# ---------------------------------------------------------------------------
# NumPy evaluation of the same expressions (used by the unit tests)
# ---------------------------------------------------------------------------


class _NS:
    pass


def _numpy_hap_feats(counts_list, n_list=None, all_features=False):
    import numpy as np
    P = len(counts_list)
    feats = [n for n, _ in HAP_FEATURES] if all_features else hap_features_needed(P)[0]
    fs = []
    for p, c in enumerate(counts_list):
        c = np.asarray(c, dtype=np.float64)
        x = _NS()
        x.c1, x.c2, x.c3, x.c4 = c[:, 0], c[:, 1], c[:, 2], c[:, 3]
        x.ns = x.c1 + x.c2 + x.c3 + x.c4
        x.n = x.ns if (n_list is None or n_list[p] is None) else np.asarray(n_list[p], np.float64)
        for name, e in HAP_FEATURES:
            if name in feats:
                setattr(x, name, eval(e, {}, {"x": x}))
        n = x.n
        with np.errstate(divide="ignore", invalid="ignore"):
            d1, d2 = n, n * (n - 1)
            d3, d4 = d2 * (n - 2), d2 * (n - 2) * (n - 3)
            x.r1 = np.where(d1 > 0, 1 / np.where(d1 > 0, d1, 1), 0.0)
            x.r2 = np.where(d2 > 0, 1 / np.where(d2 > 0, d2, 1), 0.0)
            x.r3 = np.where(d3 > 0, 1 / np.where(d3 > 0, d3, 1), 0.0)
            x.r4 = np.where(d4 > 0, 1 / np.where(d4 > 0, d4, 1), 0.0)
        fs.append(x)
    return fs


def numpy_hap_stats(counts_list, n_list=None):
    """Evaluate the generated expressions with NumPy float64 (test helper)."""
    import numpy as np
    fs = _numpy_hap_feats(counts_list, n_list)
    calls, stats = plan(len(counts_list))
    vals = [eval(hap_call_expr(case, args), {}, {"f": fs}) for case, args in calls]
    out = np.zeros((len(fs[0].c1), len(stats)))
    for si, (_, terms) in enumerate(stats):
        for idx, w in terms:
            out[:, si] += w * vals[idx]
    return out


def check_spin(seed=0, trials=12, small_haplotypes=False):
    """Exact check (rational arithmetic, random integer counts: a polynomial identity test) of
    every spin form against the weighted raw calls it stands for, both paths, P = 1..4.
    ``small_haplotypes``: haplotype samples of 0 to 5 instead (reciprocals of zero products
    are 0); the genotype path divides by n(n-1)(n-2) and has no value there."""
    import random
    import re
    from fractions import Fraction as Fr
    rng = random.Random(seed)
    lit = lambda e: re.sub(r"(?<![\w.])(\d+\.\d+|\d+)(?![\w.\]])", r"Fr('\1')", e)  # noqa: E731
    inv = lambda d: Fr(1) / d if d > 0 else Fr(0)  # noqa: E731
    code = lambda e: compile(lit(e), "<form>", "eval")  # noqa: E731
    feats = {False: [(n, code(e)) for n, e in HAP_FEATURES], True: [(n, code(e)) for n, e in GENO_FEATURES]}
    for geno in ((False,) if small_haplotypes else (False, True)):
        for P in (1, 2, 3, 4):
            calls, raw = plan(P, geno)
            expr = [code((geno_call_expr if geno else hap_call_expr)(c, a)) for c, a in calls]
            defs = {k: code(e) for k, e in spin_defs(P, geno).items()}
            stats = [(w, [(code(A), code(B)) for A, B in t]) for _, w, t, _ in spin_stats(P, geno)]
            for _ in range(trials):
                f, env = [], {"Fr": Fr, "fma": lambda a, b, c: a * b + c}
                for p in range(P):
                    x = _NS()
                    if small_haplotypes:
                        c = [0, 0, 0, 0]
                        for _ in range(rng.randint(0, 5)):
                            c[rng.randrange(4)] += 1
                    else:
                        c = [rng.randint(0, 9) for _ in range(9 if geno else 4)]
                        c[-1] += 4  # at least four individuals: every denominator positive
                    n = Fr(sum(c))
                    x.n = x.ns = n
                    d = [n, n * (n - 1), n * (n - 1) * (n - 2), n * (n - 1) * (n - 2) * (n - 3)]
                    x.r1, x.r2, x.r3, x.r4 = x.u1, x.u2, x.u3, x.w4 = [inv(q) for q in d]
                    x.invn, x.inn1 = x.r1, inv(4 * n * (n - 1))
                    # (sigma, tau) of every cell: genotype cells g1..g9 = n22 .. n00
                    st = [(1 - a, 1 - b) for a in (2, 1, 0) for b in (2, 1, 0)] if geno else [(-1, -1), (-1, 1), (1, -1), (1, 1)]
                    for m, k in enumerate(c):
                        setattr(x, f"g{m + 1}" if geno else f"c{m + 1}", Fr(k))
                    for name, e in feats[geno]:
                        setattr(x, name, eval(e, {"x": x, "Fr": Fr}))
                    f.append(x)
                    for name, (a, b) in {"S": (1, 0), "T": (0, 1), "R": (1, 1), "SS": (2, 0), "TT": (0, 2), "SST": (2, 1),
                                         "STT": (1, 2), "SSTT": (2, 2)}.items():
                        env[f"{name}{p}"] = Fr(sum(k * s ** a * t ** b for k, (s, t) in zip(c, st)))
                    env[f"n{p}"] = n
                    loc = {"n": n, **{k[:-len(str(p))]: v for k, v in env.items() if k.endswith(str(p)) and k[0] in "STR"}}
                    cells = [eval(code(e), {"Fr": Fr}, loc) for e in (GENO_CELLS if geno else HAP_CELLS)]
                    assert cells == (c[::-1] if geno else c), (geno, cells, c)
                    for k in range(4):
                        env[f"r{k + 1}{p}"] = inv(d[k])
                for k, e in defs.items():
                    env[k] = eval(e, env)
                vals = [eval(e, {"f": f, "Fr": Fr}) for e in expr]
                for (w, terms), (name, rt) in zip(stats, raw):
                    want = sum(Fr(q) * vals[idx] for idx, q in rt)
                    got = Fr(w) * sum(eval(A, env) * eval(B, env) for A, B in terms)
                    assert got == want, (geno, P, name)
    return True


def check():
    """Symbolic check of the factored forms against the reference formulas (sympy)."""
    check_spin()
    import sympy as sp
    for poly in _HORNER_POLYS.values():
        e, _, g = _horner_sympy(poly)
        loc = {f"g{i + 1}": g[i] for i in range(9)}
        h = sp.sympify(horner_form(poly).replace("x.g", "g"), locals=loc)
        assert sp.expand(h - e) == 0
    a = sp.symbols("a1:5")
    b = sp.symbols("b1:5")

    def feats(c):
        x = _NS()
        x.c1, x.c2, x.c3, x.c4 = c
        x.ns = sum(c)
        x.n = x.ns
        for name, e in HAP_FEATURES:
            setattr(x, name, eval(e, {}, {"x": x}))
        return x

    X, Y = feats(a), feats(b)
    a1, a2, a3, a4 = a
    b1, b2, b3, b4 = b
    # pi2(i,j,i,j) numerator, haplotype_kernels.py:250-263
    qBa, qAa, pAb, pBb = a2 + a4, a3 + a4, b1 + b2, b1 + b3
    pBa, qAb, qBb, pAa = a1 + a3, b3 + b4, b2 + b4, a1 + a2
    ref_ijij = ((qBa * qAa * pAb * pBb + pBa * qAa * pAb * qBb + pAa * qBa * pBb * qAb + pAa * pBa * qBb * qAb
                 + (-(a2 * a3 * b1) + a4 * b1 - a2 * a4 * b1 - a3 * a4 * b1 - a4 * a4 * b1 - a4 * b1 * b1
                    + a3 * b2 - a1 * a3 * b2 - a3 * a3 * b2 - a1 * a4 * b2 - a3 * a4 * b2 - a3 * b1 * b2
                    - a4 * b1 * b2 - a3 * b2 * b2 + a2 * b3 - a1 * a2 * b3 - a2 * a2 * b3 - a1 * a4 * b3
                    - a2 * a4 * b3 - a2 * b1 * b3 - a4 * b1 * b3 - a1 * b2 * b3 - a4 * b2 * b3 - a2 * b3 * b3
                    + a1 * b4 - a1 * a1 * b4 - a1 * a2 * b4 - a1 * a3 * b4 - a2 * a3 * b4 - a2 * b1 * b4
                    - a3 * b1 * b4 - a1 * b2 * b4 - a3 * b2 * b4 - a1 * b3 * b4 - a2 * b3 * b4
                    - a1 * b4 * b4)) / 4)
    HA = X.pA * Y.qA + X.qA * Y.pA
    HB = X.pB * Y.qB + X.qB * Y.pB
    corr = (X.Q1 * b4 + X.Q2 * b3 + X.Q3 * b2 + X.Q4 * b1
            - (a1 * Y.L1 + a2 * Y.L2 + a3 * Y.L3 + a4 * Y.L4))
    assert sp.expand(ref_ijij - (HA * HB + corr) / 4) == 0
    # single-population numerators, haplotype_kernels.py:76, 102-104, 298-301
    c1, c2, c3, c4 = a
    assert sp.expand(X.DDs - (c1 * (c1 - 1) * c4 * (c4 - 1) + c2 * (c2 - 1) * c3 * (c3 - 1)
                              - 2 * c1 * c2 * c3 * c4)) == 0
    diff = c1 * c4 - c2 * c3
    assert sp.expand(X.DZs - (diff * (c3 + c4 - c1 - c2) * (c2 + c4 - c1 - c3) + diff * (c2 + c3 - c1 - c4)
                              + 2 * (c2 * c3 + c1 * c4))) == 0
    assert sp.expand(X.PIs - ((c1 + c2) * (c1 + c3) * (c2 + c4) * (c3 + c4)
                              - c1 * c4 * (-1 + c1 + 3 * c2 + 3 * c3 + c4)
                              - c2 * c3 * (-1 + 3 * c1 + c2 + c3 + 3 * c4))) == 0
    # triple, haplotype_kernels.py:276-286 (t = a, single = b)
    tpA, tqA = a1 + a2, a3 + a4
    spB, sqB = b1 + b3, b2 + b4
    ref_tr = (-(tpA * a4 * spB) - (a2 * tqA * spB) + (tpA * (a2 + a4) * tqA * spB)
              + (tpA * tqA * (-2 * b2 - 2 * b4)) + (tpA * a4 * sqB) + (a2 * tqA * sqB)
              + (tpA * (a1 + a3) * tqA * sqB)) / 2
    assert sp.expand(ref_tr - (spB * X.T1 + sqB * X.T2) / 2) == 0
    # shared, haplotype_kernels.py:225-238 (s = a, a-pop = b, b-pop = c)
    c = sp.symbols("e1:5")
    Z = feats(c)
    s1, s2, s3, s4 = a
    ca1, ca2 = b1, b2
    cb1, cb2, cb3, cb4 = c
    inner = (-1 + s3) * cb1 + s3 * cb2 - cb3 + s3 * cb3 + s3 * cb4 + s1 * Z.qB
    ref_sh = (s4 * s4 * Y.pA * Z.pB + s2 * s2 * Y.qA * Z.pB
              + (-1 + s1 + s3) * (s3 * Y.pA + s1 * Y.qA) * Z.qB
              + s4 * (s1 * Y.qA * Z.pB + ca1 * inner + ca2 * inner)
              + s2 * (s4 * (Y.pA + Y.qA) * Z.pB + s3 * (ca1 * Z.pB + ca2 * Z.pB + Y.qA * Z.qB)
                      + Y.qA * ((-1 + s1) * cb1 - cb3 + s1 * (cb2 + cb3 + cb4)))) / 4
    mine = (Y.pA * (Z.pB * (X.L1 - s4) + Z.qB * (X.L2 - s3))
            + Y.qA * (Z.pB * (X.L3 - s2) + Z.qB * (X.L4 - s1))) / 4
    assert sp.expand(ref_sh - mine) == 0
    return True


if __name__ == "__main__":
    check()
    print(generate())
