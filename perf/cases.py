"""Performance cases of the two-locus LD framework: what a user has it do, over the real range.

A case is a dict of plain values.  ``prepare`` makes what the user's program holds before the
call (seeded inputs on the GPU and the parser or matrix object), ``run`` is one pass through
the public entry points, ``work`` the bytes and operations that pass cannot do without and
``exact`` the same outputs from plain torch in 64 bits.

Inputs are founder mosaics: twenty founders with a 1/k derived-allele spectrum, per-population
drift, haplotypes that switch founders along the chromosome, and missing calls at random.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pg_gpu_b200 import ld_matrix, ld_pipeline, ld_statistics, parse
from pg_gpu_b200.haplotype_matrix import HaplotypeMatrix

FOUNDERS = 20
N_STATS = {1: 3, 2: 15, 3: 45, 4: 105}
BLOCK_BP = 50_000  # bootstrap blocks


def listed():
    return [
        # one short window of a genome scan: the smallest call, latency and launches
        dict(name="window_1pop", kind="parse", pops="60", snps=400, span=40_000, cutoff=40_000, bins=6, log_bins=True,
             missing=0.02),
        # one population over a megabase, complete data, four decade bins
        dict(name="region_1pop", kind="parse", pops="100", snps=5_000, span=1_000_000, cutoff=1_000_000, bins=5,
             log_bins=True, missing=0.0),
        # the two-population parse behind a demographic fit
        dict(name="region_2pop", kind="parse", pops="100,140", snps=50_000, span=5_000_000, cutoff=1_000_000, bins=16,
             log_bins=True, missing=0.05),
        # four populations: the 105-statistic vector
        dict(name="region_4pop", kind="parse", pops="100,120,140,160", snps=8_000, span=800_000, cutoff=800_000,
             bins=16, log_bins=True, missing=0.02),
        # unphased genotypes, one population, linear bins
        dict(name="genotypes_1pop", kind="parse", pops="500", snps=100_000, span=10_000_000, cutoff=200_000, bins=20,
             log_bins=False, missing=0.02, genotypes=True),
        # unphased genotypes, two populations
        dict(name="genotypes_2pop", kind="parse", pops="120,180", snps=20_001, span=2_000_000, cutoff=200_000, bins=20,
             log_bins=False, missing=0.02, genotypes=True),
        # a batch of uneven windows with bootstrap replicates and per-window totals, replayed
        # as one CUDA graph (the headline workload)
        dict(name="windows_3pop_bootstrap", kind="parse", pops="50,120,300", windows=200, median_snps=2_000,
             density=0.01, cutoff=1_000_000, bins=16, log_bins=True, missing=0.03, replicates=100, graph=True),
        # a chromosome of a large sample
        dict(name="chromosome_1pop", kind="parse", pops="2000", snps=1_000_000, span=50_000_000, cutoff=100_000,
             bins=32, log_bins=True, missing=0.01),
        # the full r^2 matrix of a region
        dict(name="matrix_r2", kind="matrix", rows=200, snps=12_000, missing=0.02),
        # Kelly's ZnS with the default (unbiased sigma_D^2) estimator: no matrix is kept
        dict(name="zns_sigma_d2", kind="zns", rows=500, snps=16_000, missing=0.02),
        # dosage r^2 matrix of unphased genotypes
        dict(name="matrix_dosage_r2", kind="dosage", rows=300, snps=6_001, missing=0.02),
        # the pair-list calls of a program that walks the pairs itself: counts of each
        # population, then the two-population statistics
        dict(name="pair_list_2pop", kind="pairs", pops="100,140", snps=50_000, pairs=1_000_000, missing=0.05),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hap"] * 6 + ["geno"] * 3 + ["windows", "matrix", "zns", "dosage", "pairs"])
    missing = rng.choice([0.0, 0.01, 0.03, 0.05])
    if kind == "windows":
        P = rng.choice([1, 2, 3])
        return dict(kind="parse", pops=",".join(str(_log_int(rng, 20, 300)) for _ in range(P)),
                    windows=rng.randint(2, 200), median_snps=_log_int(rng, 300, 2_000), density=0.01,
                    cutoff=_log_int(rng, 50_000, 1_000_000), bins=rng.randint(4, 16), log_bins=True, missing=missing,
                    replicates=rng.choice([20, 100]), graph=rng.choice([True, False]))
    if kind in ("hap", "geno"):
        geno = kind == "geno"
        P = rng.choice([1, 1, 2, 3, 4]) if not geno else rng.choice([1, 1, 2, 3])
        most = {1: 4e8, 2: 2e8, 3: 1e8, 4: 3e7}[P] * (0.4 if geno else 1.0)  # pairs
        snps = _log_int(rng, 300, 200_000 if P == 1 else 60_000)
        density = rng.choice([0.005, 0.01, 0.02])
        span = int(snps / density)
        cutoff = min(_log_int(rng, 5_000, 1_000_000), span, max(1_000, int(most / snps / density)))
        n_top = 2_000 if P == 1 and not geno and snps * cutoff * density < 1e8 else 500 if P == 1 else 300
        return dict(kind="parse", pops=",".join(str(_log_int(rng, 12, n_top)) for _ in range(P)), snps=snps, span=span,
                    cutoff=cutoff, bins=rng.randint(1, 32 if P == 1 else 20), log_bins=rng.random() < 0.7,
                    missing=missing, genotypes=geno, packed=rng.random() < 0.25, map=rng.random() < 0.25)
    if kind in ("matrix", "zns", "dosage"):
        return dict(kind=kind, rows=_log_int(rng, 20, 600), snps=_log_int(rng, 500, 12_000), missing=missing)
    return dict(kind="pairs", pops="%d,%d" % (_log_int(rng, 20, 200), _log_int(rng, 20, 200)),
                snps=_log_int(rng, 2_000, 50_000), pairs=_log_int(rng, 20_000, 1_000_000), missing=missing)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _sizes(case):
    return [int(x) for x in case["pops"].split(",")] if "pops" in case else [int(case["rows"])]


def _window_sizes(case):
    """SNPs per window: the quantiles of a lognormal around the median, clipped to 200 .. 20,000."""
    k = (torch.arange(case["windows"], dtype=torch.float64) + 0.5) / case["windows"]
    z = math.sqrt(2.0) * torch.erfinv(2.0 * k - 1.0)
    return torch.exp(math.log(case["median_snps"]) + z * math.log(10) / 3).clamp(200, 20_000).long().numpy()


def _positions(rng, m, span):
    pos = np.unique(rng.integers(0, span, size=int(m * 1.3) + 16))
    while len(pos) < m:
        pos = np.unique(np.concatenate([pos, rng.integers(0, span, size=m)]))
    return np.sort(rng.permutation(pos)[:m]).astype(np.float64)


def _founders(rng, gen, m):
    k = np.arange(1, FOUNDERS)
    count = torch.as_tensor(rng.choice(k, size=m, p=(1.0 / k) / np.sum(1.0 / k)), device="cuda")
    rank = torch.rand((FOUNDERS, m), generator=gen, device="cuda").argsort(0).argsort(0)
    return rank < count[None, :]


def _mosaic(rng, gen, sizes, gap, missing):
    """(sum(sizes), len(gap)) int8 haplotypes; a founder switch at rate 1e-5 per bp of ``gap``."""
    m = len(gap)
    base = _founders(rng, gen, m)
    p_switch = torch.as_tensor(-np.expm1(-1e-5 * gap), dtype=torch.float32, device="cuda")
    col = torch.arange(m, device="cuda")
    out = torch.empty((sum(sizes), m), dtype=torch.int8, device="cuda")
    at = 0
    for n in sizes:
        f = base
        if len(sizes) > 1:  # drift of every founder allele, F = 0.05
            p = base.double().mean(0).cpu().numpy()
            q = rng.beta(np.maximum(19.0 * p, 1e-6), np.maximum(19.0 * (1 - p), 1e-6))
            f = torch.rand((FOUNDERS, m), generator=gen, device="cuda") < torch.as_tensor(q, device="cuda")
        f = f.to(torch.int8).reshape(-1)
        step = max(1, (1 << 25) // m)
        for r in range(0, n, step):
            k = min(step, n - r)
            last = torch.where(torch.rand((k, m), generator=gen, device="cuda") < p_switch, col, 0).cummax(1).values
            who = torch.randint(FOUNDERS, (k, m), generator=gen, device="cuda").gather(1, last)
            h = f[who * m + col]
            if missing:
                h[torch.rand((k, m), generator=gen, device="cuda") < missing] = -1
            out[at + r:at + r + k] = h
        at += n
    return out


def _diploid(hap, gen, missing):
    g = hap[0::2] + hap[1::2]
    if missing:
        g[torch.rand(g.shape, generator=gen, device="cuda") < missing] = -1
    return g


def _polymorphic(x, top):
    seen = torch.zeros((2, x.shape[1]), dtype=torch.bool, device="cuda")
    for r in range(0, x.shape[0], 64):
        s = x[r:r + 64]
        seen[0] |= ((s >= 0) & (s < top)).any(0)
        seen[1] |= (s > 0).any(0)
    return seen.all(0)


def _data(case, seed):
    """(codes, positions, window offsets or None, rng, order of the windows) of the polymorphic sites."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    geno = bool(case.get("genotypes")) or case["kind"] == "dosage"
    sizes = _sizes(case)
    offs = order = None
    if "windows" in case:
        order = rng.permutation(case["windows"])
        counts = _window_sizes(case)[order]
        parts = [_positions(rng, int(m), int(m / case["density"])) for m in counts]
        pos, offs = np.concatenate(parts), np.concatenate([[0], np.cumsum(counts)])
        gap = np.diff(pos, prepend=-1e9)
        gap[offs[:-1]] = 1e9
    else:
        pos = _positions(rng, case["snps"], case.get("span", case["snps"] * 100))
        gap = np.diff(pos, prepend=-1e9)
    if geno:
        x = _diploid(_mosaic(rng, gen, [2 * n for n in sizes], gap, 0.0), gen, case["missing"])
    else:
        x = _mosaic(rng, gen, sizes, gap, case["missing"])
    keep = _polymorphic(x, 2 if geno else 1)
    x = x[:, keep].contiguous()
    keep = keep.cpu().numpy()
    if offs is not None:
        offs = np.concatenate([[0], np.cumsum(keep)])[offs]
    return x, pos[keep], offs, rng, order


def _edges(case):
    c = float(case["cutoff"])
    return np.logspace(1, math.log10(c), case["bins"] + 1) if case["log_bins"] else np.linspace(0, c, case["bins"] + 1)


def _rows(sizes):
    offs = np.concatenate([[0], np.cumsum(sizes)])
    return [np.arange(a, b) for a, b in zip(offs[:-1], offs[1:])]


def _parse_inputs(case, seed):
    x, pos, offs, rng, order = _data(case, seed)
    d = dict(x=x, pos=pos, rows=_rows(_sizes(case)), edges=_edges(case), offs=offs, coords=None, max_dist=float(case["cutoff"]),
             block=None, n_blocks=1, weights=None)
    if case.get("map"):  # binned by a genetic map with a varying rate, physical cutoff
        d["coords"] = np.cumsum(np.diff(pos, prepend=pos[0]) * np.exp(rng.normal(0, 0.3, len(pos)))) + 0.25
    if offs is not None:
        per = np.ceil(_window_sizes(case)[order] / case["density"] / BLOCK_BP).astype(np.int64)
        local = (pos // BLOCK_BP).astype(np.int64)
        d["block"] = (local + np.repeat(np.cumsum(per) - per, np.diff(offs))).astype(np.int32)
        d["n_blocks"] = int(per.sum())
        w = np.stack([np.bincount(rng.integers(0, d["n_blocks"], d["n_blocks"]), minlength=d["n_blocks"])
                      for _ in range(case["replicates"])])
        one = np.zeros((len(per), d["n_blocks"]), np.int64)
        one[np.repeat(np.arange(len(per)), per), np.arange(d["n_blocks"])] = 1
        d["weights"], d["totals"] = w.astype(np.int32), one.astype(np.int32)
    return d


def _pair_indices(case, m):
    """The first ``pairs`` pairs in anchor order with a cutoff of 2,000 SNPs' width."""
    reach = 2_000
    per = np.minimum(reach, m - 1 - np.arange(m))
    n = min(int(case["pairs"]), int(per.sum()))
    i = torch.repeat_interleave(torch.arange(m), torch.as_tensor(per))[:n]
    start = np.cumsum(per) - per
    j = i + 1 + torch.arange(n) - torch.as_tensor(start)[i]
    return i.to(torch.int32).cuda(), j.to(torch.int32).cuda()


def prepare(case, seed):
    if case["kind"] == "parse":
        d = _parse_inputs(case, seed)
        data = d["x"]
        if case.get("packed"):
            data = torch.as_tensor(parse.pack_codes(data.cpu().numpy()), device="cuda")
        p = parse.Parser(data, torch.as_tensor(d["pos"], device="cuda"), d["rows"], d["edges"],
                         genotypes=bool(case.get("genotypes")), max_dist=d["max_dist"], coords=d["coords"],
                         window_offsets=d["offs"], snp_block=d["block"], n_blocks=d["n_blocks"],
                         packed=bool(case.get("packed")))
        s = dict(kind="parse", parser=p)
        if d["weights"] is not None:
            s["weights"] = torch.as_tensor(d["weights"], device="cuda")
            s["totals"] = torch.as_tensor(d["totals"], device="cuda")
            if case.get("graph"):
                s["graph"], s["extra"] = p.graph(after=lambda out: _combine(s, out))
        return s
    x, pos, *_ = _data(case, seed)
    if case["kind"] == "pairs":
        i, j = _pair_indices(case, x.shape[1])
        return dict(kind="pairs", x=x, i=i, j=j, rows=_rows(_sizes(case)))
    if case["kind"] == "dosage":
        return dict(kind="dosage", x=x)
    return dict(kind=case["kind"], hm=HaplotypeMatrix(x, torch.as_tensor(pos, device="cuda")))


def _combine(s, out):
    return parse.block_combine(out.sums, s["weights"]), parse.block_combine(out.sums, s["totals"])


def run(s):
    if s["kind"] == "parse":
        if "graph" in s:
            s["graph"].replay()
            out, extra = s["parser"].out, s["extra"]
        else:
            out = s["parser"].run()
            extra = _combine(s, out) if "weights" in s else ()
        res = dict(sums=out.sums, r2_sums=out.r2_sums, pairs=out.pairs, r2_counts=out.r2_counts)
        if extra:
            res["replicates"], res["windows"] = extra
        return res
    if s["kind"] == "matrix":
        return s["hm"].pairwise_r2()
    if s["kind"] == "zns":
        return ld_statistics.zns(s["hm"])
    if s["kind"] == "dosage":
        return ld_matrix.diploid_r2_matrix(s["x"])
    c = [ld_pipeline.compute_counts_for_pairs(s["x"], s["i"], s["j"], r) for r in s["rows"]]
    stats = ld_pipeline.compute_two_pop_statistics_batch(c[0][0], c[1][0], c[0][1], c[1][1])
    return dict(counts=[k[0] for k in c], n_valid=[k[1] for k in c if k[1] is not None], stats=stats)


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------


def _pairs_of(m, span, cutoff):
    f = min(1.0, cutoff / span)
    return m * m * (f - 0.5 * f * f)


def work(case):
    n = sum(_sizes(case))
    geno = bool(case.get("genotypes"))
    if case["kind"] == "parse":
        P = len(_sizes(case))
        if "windows" in case:
            sizes = _window_sizes(case)
            m = int(sizes.sum())
            pairs = sum(_pairs_of(k, k / case["density"], case["cutoff"]) for k in sizes.tolist())
            blocks = sum(math.ceil(k / case["density"] / BLOCK_BP) for k in sizes.tolist())
            reps = case["replicates"] + case["windows"]
        else:
            m, pairs, blocks, reps = case["snps"], _pairs_of(case["snps"], case["span"], case["cutoff"]), 1, 0
        x = n * m / (4 if case.get("packed") else 1)
        out = 8 * case["bins"] * (blocks * (N_STATS[P] + 3) + reps * N_STATS[P])
        extra = 4 * m + 4 * reps * blocks if "windows" in case else 8 * m if case.get("map") else 0
        # Gram products of the indicators (4 per haplotype, 9 per genotype; a multiply-add is
        # two) and one multiply-add into every sum
        return {"bytes": x + 8 * m + extra + out, "flops": pairs * (2 * (9 if geno else 4) * n + 2 * (N_STATS[P] + 1))}
    m = case["snps"]
    if case["kind"] == "pairs":
        k = case["pairs"]
        return {"bytes": n * m + 8 * k + k * (2 * 5 * 4 + 15 * 8), "flops": k * (2 * 4 * n + 2 * 15)}
    per = 2 * (9 if case["kind"] == "dosage" else 4) * n
    out = 8 if case["kind"] == "zns" else 8 * m * m
    return {"bytes": n * m + out, "flops": 0.5 * m * m * (per + 10)}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits, plain torch
# ---------------------------------------------------------------------------
#
# With sigma = 1 - 2a (a an individual's allele frequency at the left locus: 0 or 1 for a
# haplotype, 0, 1/2, 1 for a genotype), tau the same at the right locus, every statistic is a
# mean over distinct individuals of a product of these, written with the sums over a
# population's jointly called individuals: S = sum sigma, T = sum tau, R = sum sigma tau,
# SS = sum sigma^2, ... (integers, so the numerators are exact in 64 bits).


def _planes(x, geno):
    x = x.float()
    v = (x >= 0).float()
    s = torch.where(x >= 0, (1.0 - x) if geno else (1.0 - 2.0 * x), torch.zeros_like(x))
    return [v, s, s * s] if geno else [v, s]


def _moments(a, b, geno):
    """(n, S, T, R, SS, TT, SST, STT, SSTT) of all row x column pairs, float64."""
    g = [[(p.t() @ q).double() for q in b] for p in a]
    n, S, T, R = g[0][0], g[1][0], g[0][1], g[1][1]
    if geno:
        return n, S, T, R, g[2][0], g[0][2], g[2][1], g[1][2], g[2][2]
    return n, S, T, R, n, n, T, S, n


def _inverse(d):
    return torch.where(d > 0, 1.0 / torch.where(d > 0, d, torch.ones_like(d)), torch.zeros_like(d))


class _Pop:
    def __init__(self, mom):
        n, S, T, R, SS, TT, SST, STT, SSTT = mom
        self.n, self.S, self.T = n, S, T
        n2, n3 = n * (n - 1), n * (n - 1) * (n - 2)
        self.nu, self.m = n2, n - 1
        self.r1, self.r2, self.r3 = _inverse(n), _inverse(n2), _inverse(n3)
        r4 = _inverse(torch.where(n >= 4, n3 * (n - 3), torch.zeros_like(n)))
        self.E, self.W = n * R - S * T, S * T - R
        u, v = S * S - SS, T * T - TT
        self.hA, self.hB = n2 - u, n2 - v
        RS, RT = R * S - SST, R * T - STT
        self.U, self.V = n * RS - u * T, n * RT - v * S
        k = (n - 1) * (n - 2)
        self.XA, self.YA = (n - 2) * self.hA, (k - u) * T + 2 * RS
        self.XB, self.YB = (n - 2) * self.hB, (k - v) * S + 2 * RT
        Q2 = R * R - SSTT
        Q3 = R * S * T - R * R - S * STT - T * SST + 2 * SSTT
        Q4 = u * v - 4 * Q3 - 2 * Q2
        k23 = (n - 2) * (n - 3)
        self.dd = (k23 * Q2 - 2 * (n - 3) * Q3 + Q4) * r4
        self.dz = ((n - 3) * Q3 - Q4) * r4
        self.pi = (n2 * k23 - k23 * (u + v) + Q4) * r4
        self.vx, self.vy = n * SS - S * S, n * TT - T * T


def _statistics(f, geno):
    """The moments-ordered statistic vector of one set of pairs, a list of float64 tensors."""
    P, c = len(f), (2.0 if geno else 1.0)  # the genotype D is the composite one, twice as large
    out = []
    for i in range(P):
        for j in range(i, P):
            out.append(c * c / 16 * (f[i].dd if i == j else f[i].E * f[j].E * f[i].r2 * f[j].r2))
    for i in range(P):
        for j in range(P):
            for k in range(j, P):
                a, b, d = f[i], f[j], f[k]
                if i == j == k:
                    v = a.dz / 4
                elif j == k:
                    v = a.E * b.W * a.r2 * b.r2 / 4
                elif i in (j, k):
                    o = d if i == j else b
                    v = (a.U * o.T + a.V * o.S) * a.r3 * o.r1 / 8
                else:
                    v = a.E * (b.S * d.T + d.S * b.T) * a.r2 * b.r1 * d.r1 / 8
                out.append(c * v)

    def het(q, w, side):
        return q.n * w.n - getattr(q, side) * getattr(w, side)

    for i in range(P):
        for j in range(i, P):
            for k in range(i, P):
                for l in range(k, P):
                    if (k == i == l and j != i) or (i == k and l < j):
                        continue
                    if i == j == k == l:
                        v = f[i].pi / 16
                    elif i == j and k == l:
                        a, b = f[i], f[k]
                        v = (a.hA * b.hB + b.hA * a.hB) * a.r2 * b.r2 / 32
                    elif i == j or k == l:
                        t, p, q = (i, k, l) if i == j else (k, i, j)
                        if t in (p, q):  # one population three times
                            t, s = f[t], f[q if p == t else p]
                            va = (t.XA * s.n - t.YA * s.T) * t.r3 * s.r1 / 16
                            v = va if not geno else 0.5 * (va + (t.XB * s.n - t.YB * s.S) * t.r3 * s.r1 / 16)
                        else:
                            t, p, q = f[t], f[p], f[q]
                            v = (t.hA * het(p, q, "T") + t.hB * het(p, q, "S")) * t.r2 * p.r1 * q.r1 / 32
                    elif (i, j) == (k, l):
                        a, b = f[i], f[j]
                        v = (a.nu * b.nu - a.m * b.m * (a.S * b.S + a.T * b.T) + a.W * b.W) * a.r2 * b.r2 / 16
                    elif len({i, j, k, l}) == 3:
                        s = ({i, j} & {k, l}).pop()
                        p, q = f[j if i == s else i], f[l if k == s else k]
                        s = f[s]
                        num = (2 * s.nu * p.n * q.n - s.m * (s.S * (p.S * q.n + q.S * p.n) + s.T * (p.T * q.n + q.T * p.n))
                               + s.W * (p.S * q.T + q.S * p.T))
                        v = num * s.r2 * p.r1 * q.r1 / 32
                    else:
                        a, b, d, e = f[i], f[j], f[k], f[l]
                        v = (het(a, b, "S") * het(d, e, "T") + het(d, e, "S") * het(a, b, "T")) * (
                            a.r1 * b.r1 * d.r1 * e.r1) / 32
                    out.append(v)
    return out


def _exact_parse(case, seed):
    d = _parse_inputs(case, seed)
    x, geno, sizes = d["x"], bool(case.get("genotypes")), _sizes(case)
    P, nb = len(sizes), len(d["edges"]) - 1
    pos = torch.as_tensor(d["pos"], device="cuda")
    coord = pos if d["coords"] is None else torch.as_tensor(d["coords"], device="cuda")
    edges = torch.as_tensor(d["edges"], device="cuda")
    sums = torch.zeros((d["n_blocks"], nb, N_STATS[P]), dtype=torch.float64, device="cuda")
    r2s = torch.zeros((d["n_blocks"], nb), dtype=torch.float64, device="cuda")
    offs = [0, x.shape[1]] if d["offs"] is None else d["offs"].tolist()
    for a, e in zip(offs[:-1], offs[1:]):
        if e - a < 2:
            continue
        end = a + torch.searchsorted(pos[a:e], pos[a:e] + d["max_dist"], right=True).cpu().numpy()
        blk = np.zeros(e - a, np.int64) if d["block"] is None else d["block"][a:e]
        r = a
        while r < e:
            top = a + int(np.searchsorted(blk, blk[r - a], side="right"))
            width = max(1, int(end[min(r + 512, e - 1) - a]) - r)
            q = min(top, r + max(16, min(2048, 3_000_000 // width)))
            j1 = int(end[q - 1 - a])
            if j1 > r + 1:
                i, j = torch.arange(r, q, device="cuda"), torch.arange(r + 1, j1, device="cuda")
                dist = (coord[j][None, :] - coord[i][:, None]).abs()
                b = torch.bucketize(dist, edges, right=True) - 1
                ok = (j[None, :] > i[:, None]) & (j[None, :] < torch.as_tensor(end[r - a:q - a], device="cuda")[:, None])
                ok &= (b >= 0) & (b < nb)
                b = b[ok]
                hot = (b[:, None] == torch.arange(nb, device="cuda")).double()
                f = []
                for rows in d["rows"]:
                    mom = _moments(_planes(x[rows[0]:rows[-1] + 1, r:q], geno),
                                   _planes(x[rows[0]:rows[-1] + 1, r + 1:j1], geno), geno)
                    f.append(_Pop([t[ok] for t in mom]))
                k = int(blk[r - a])
                sums[k] += hot.t() @ torch.stack(_statistics(f, geno), 1)
                den = f[0].vx * f[0].vy
                r2s[k] += hot.t() @ (f[0].E * f[0].E * _inverse(den))
            r = q
    res = dict(sums=sums, r2_sums=r2s, pairs=None, r2_counts=None)
    if d["weights"] is not None:
        for name, w in (("replicates", d["weights"]), ("windows", d["totals"])):
            res[name] = (torch.as_tensor(w, device="cuda").double() @ sums.reshape(d["n_blocks"], -1)).reshape(-1, nb, N_STATS[P])
    return res


def exact(case, seed):
    if case["kind"] == "parse":
        return _exact_parse(case, seed)
    x, pos, *_ = _data(case, seed)
    if case["kind"] == "pairs":
        i, j = (t.long() for t in _pair_indices(case, x.shape[1]))
        parts = []
        for k in range(0, len(i), 100_000):
            f = []
            for rows in _rows(_sizes(case)):
                a = _planes(x[rows[0]:rows[-1] + 1][:, i[k:k + 100_000]], False)
                b = _planes(x[rows[0]:rows[-1] + 1][:, j[k:k + 100_000]], False)
                n, S, T, R = ((p * q).sum(0).double() for p, q in ((a[0], b[0]), (a[1], b[0]), (a[0], b[1]), (a[1], b[1])))
                f.append(_Pop((n, S, T, R, n, n, T, S, n)))
            parts.append(torch.stack(_statistics(f, False), 1))
        return dict(counts=[None, None], n_valid=[None, None], stats=torch.cat(parts))
    v = (x >= 0).double()
    val = x.clamp(min=0).double()
    if case["kind"] == "matrix":
        p = val.sum(0) / v.sum(0).clamp(min=1)
        D = (val.t() @ val) / (v.t() @ v) - p[:, None] * p[None, :]
        w = p * (1 - p)
        return (D * D * _inverse(w[:, None] * w[None, :])).fill_diagonal_(0.0)
    if case["kind"] == "dosage":
        c = torch.where(x >= 0, val - val.sum(0) / v.sum(0).clamp(min=1), torch.zeros_like(val))
        w = (c * c).sum(0)
        cov = c.t() @ c
        return (cov * cov * _inverse(w[:, None] * w[None, :])).fill_diagonal_(0.0)
    hap = _planes(x, False)
    total = count = 0.0
    m = x.shape[1]
    for r in range(0, m - 1, 512):
        q = min(m, r + 512)
        up = torch.arange(r + 1, m, device="cuda")[None, :] > torch.arange(r, q, device="cuda")[:, None]
        mom = _moments([t[:, r:q] for t in hap], [t[:, r + 1:] for t in hap], False)
        f = _Pop([t[up] for t in mom])
        ok = (f.n >= 4) & (f.pi != 0)
        total += float((f.dd[ok] / f.pi[ok]).sum())
        count += int((f.n >= 4).sum())
    return total / count
