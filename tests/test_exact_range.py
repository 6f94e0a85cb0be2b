"""Where the tensor-core parse's spin forms are exact, and what it evaluates beyond: up to
SPIN_MAX_N individuals no integer intermediate of any form leaves FP64's 2^53 (interval
arithmetic over the generated expressions); above, the counts recovered from the moments and the
raw calls on them, whose numerators stay exact integers where the alleles are rare.  FP64 is
evaluated operation by operation, an fma with one rounding, against integers: no tolerance where
the value itself is below 2^53."""
import random
import re
from fractions import Fraction

import pytest

from pg_gpu_b200.csrc import gen_estimators as G


class Interval:
    """Closed interval of integers; remembers the largest magnitude any operation reached."""
    top = 0

    def __init__(self, lo, hi):
        self.lo, self.hi = lo, hi

    @staticmethod
    def of(x):
        return x if isinstance(x, Interval) else Interval(x, x)

    def seen(self):
        Interval.top = max(Interval.top, abs(self.lo), abs(self.hi))
        return self

    def __neg__(self):
        return Interval(-self.hi, -self.lo)

    def __add__(self, o):
        o = Interval.of(o)
        return Interval(self.lo + o.lo, self.hi + o.hi).seen()

    __radd__ = __add__

    def __sub__(self, o):
        return self + -Interval.of(o)

    def __rsub__(self, o):
        return Interval.of(o) - self

    def product(self, o):
        o = Interval.of(o)
        p = [x * y for x in (self.lo, self.hi) for y in (o.lo, o.hi)]
        return Interval(min(p), max(p))

    def __mul__(self, o):
        return self.product(o).seen()

    __rmul__ = __mul__


def _largest(N, P, geno):
    """Largest magnitude of the forms' integer parts (what holds no reciprocal) at populations <= N."""
    env = {"fma": lambda a, b, c: Interval.of(a).product(b) + c}
    for p in range(P):
        env.update({f"{k}{p}": Interval(-N, N) for k in ("S", "T", "R", "SST", "STT")})
        env.update({f"{k}{p}": Interval(0, N) for k in ("n", "SS", "TT", "SSTT")})
    defs = G.spin_defs(P, geno)

    def value(e):
        for nm in re.findall(r"[A-Za-z]\w*", e):
            if nm not in env:
                if nm not in defs or value(defs[nm]) is None:
                    return None  # a reciprocal
                env[nm] = value(defs[nm])
        return eval(e, env)

    Interval.top = 0
    for _, _, terms, _ in G.spin_stats(P, geno):
        for A, B in terms:
            value(A), value(B)
    for nm in ("E0", "vx0", "vy0"):
        value(nm)
    return Interval.top


@pytest.mark.parametrize("geno", [False, True])
@pytest.mark.parametrize("P", [1, 2, 3, 4])
def test_no_intermediate_leaves_the_exact_range(P, geno):
    assert _largest(G.SPIN_MAX_N, P, geno) <= 2 ** 53


def test_the_limit_is_the_last_such_size():
    assert max(_largest(G.SPIN_MAX_N + 1, 4, g) for g in (False, True)) > 2 ** 53


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def _moments(cells, geno):
    st = [(1 - a, 1 - b) for a in (0, 1, 2) for b in (0, 1, 2)] if geno else [(-1, -1), (-1, 1), (1, -1), (1, 1)]
    m = {"n": float(sum(cells))}
    for name, (a, b) in {"S": (1, 0), "T": (0, 1), "R": (1, 1), "SS": (2, 0), "TT": (0, 2), "SST": (2, 1), "STT": (1, 2),
                         "SSTT": (2, 2)}.items():
        m[name] = float(sum(k * s ** a * t ** b for k, (s, t) in zip(cells, st)))
    return m


def _cells(rng, n, geno, rare):
    """n00 last (haplotypes) or first (genotypes): the common class of a pair of rare alleles."""
    k = 8 if geno else 3
    if rare:
        c = [rng.randint(0, 2) for _ in range(k)]
    else:
        cut = sorted(rng.randint(0, n) for _ in range(k))
        c = [b - a for a, b in zip([0] + cut[:-1], cut)]
    rest = n - sum(c)
    return [rest] + c if geno else c + [rest]


def _exact_numerators(cells, geno):
    """16 times the DD and pi2 numerators as integers, from the U-statistics' own definition."""
    m = {k: int(v) for k, v in _moments(cells, geno).items()}
    n, S, T, R, SS, TT, SST, STT, SSTT = (m[k] for k in ("n", "S", "T", "R", "SS", "TT", "SST", "STT", "SSTT"))
    q2 = R * R - SSTT
    q3 = R * (S * T - R) - S * STT - T * SST + 2 * SSTT
    q4 = (S * S - SS) * (T * T - TT) - 4 * q3 - 2 * q2
    dd = (n - 2) * (n - 3) * q2 - 2 * (n - 3) * q3 + q4
    pi2 = (n - 2) * (n - 3) * (n * (n - 1) - (S * S - SS) - (T * T - TT)) + q4
    return dd, pi2


@pytest.mark.parametrize("geno", [False, True])
@pytest.mark.parametrize("rare", [False, True])
def test_spin_numerators_at_the_limit(geno, rare):
    rng = random.Random(3)
    defs = G.spin_defs(1, geno)
    for _ in range(60):
        cells = _cells(rng, G.SPIN_MAX_N, geno, rare)
        env = {"fma": _fma, **{k + "0": v for k, v in _moments(cells, geno).items()}}

        def value(nm):
            for x in re.findall(r"[A-Za-z]\w*", defs[nm]):
                if x not in env:
                    env[x] = value(x)
            return eval(defs[nm], env)

        assert (value("DD0"), value("PI0")) == _exact_numerators(cells, geno), cells


@pytest.mark.parametrize("n", [5793, 9741, 9742, 13823, 20000, 100003, 500009])
def test_count_numerators_of_rare_alleles(n):
    """DDs, DZs and PIs of the haplotype path on the recovered counts: exact, so pairs whose
    numerators are 0 (two singletons on one haplotype; a site constant among the called) stay 0."""
    rng = random.Random(n)
    x = G._NS()
    fixed = [[1, 0, 0, n - 1], [0, 0, 7, n - 7], [0, 1, 1, n - 2], [2, 0, 0, n - 2]]
    for cells in fixed + [_cells(rng, n, False, True) for _ in range(60)]:
        m = _moments(cells, False)
        got = [eval(e, {}, m) for e in G.HAP_CELLS]
        assert got == cells
        dd, pi2 = _exact_numerators(cells, False)
        for num in (float, Fraction):
            x.c1, x.c2, x.c3, x.c4 = [num(c) for c in got]
            x.ns = x.n = num(n)
            for name, e in G.HAP_FEATURES:
                setattr(x, name, eval(e, {}, {"x": x}))
            if num is float:
                rounded = [x.DDs, x.DZs, x.PIs]
        assert (rounded[0], rounded[2]) == (x.DDs, x.PIs)
        # Dz's own value passes 2^53 with three factors of n: its largest term then has a few roundings
        assert rounded[1] == x.DZs or (abs(x.DZs) > 2 ** 53 and abs(Fraction(rounded[1]) - x.DZs) <= abs(x.DZs) / 2 ** 50)
        assert (16 * x.DDs, 16 * x.PIs) == (dd, pi2)


@pytest.mark.parametrize("n", [5793, 20000, 100003, 500009])
def test_genotype_cells_of_the_moments(n):
    rng = random.Random(n)
    for k in range(60):
        cells = _cells(rng, n, True, k % 2 == 0)
        assert [eval(e, {}, _moments(cells, True)) for e in G.GENO_CELLS] == cells
