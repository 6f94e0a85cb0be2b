"""The parse of populations on both sides of the spin forms' exact range (5,792 individuals) and
far beyond, where all alleles are rare: every statistic is then a small integer numerator times
the reciprocals, so the bin sums agree with the oracle's, which counts, to rounding -- 1e-11 of
the sum of absolute values (some hundred roundings a pair, a few hundred pairs a bin; a form that
cancels n^4 terms misses that by orders of magnitude)."""
import numpy as np
import pytest

from oracle import ld_oracle as O
from pg_gpu_b200 import parse

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


def rare(rng, sizes, m, genotypes):
    """Sites of one to three carriers out of a few per population (so that carriers are shared),
    a twin of the site before now and then, missing calls."""
    off = np.concatenate([[0], np.cumsum(sizes)])
    x = np.zeros((off[-1], m), np.int8)
    x[rng.random(x.shape) < 2e-4] = -1
    for v in range(m):
        for a, b in zip(off[:-1], off[1:]):
            few = np.arange(a, min(b, a + 5))
            x[rng.choice(few, size=min(len(few), rng.integers(1, 4)), replace=False), v] = \
                rng.integers(1, 3) if genotypes else 1
    x[:, 1::5] = x[:, 0:-1:5]
    return x, [np.arange(a, b) for a, b in zip(off[:-1], off[1:])]


@pytest.mark.parametrize("genotypes", [False, True])
@pytest.mark.parametrize("sizes", [(5792,), (5793,), (14000,), (100003,), (9743, 9800), (300, 14000), (6000, 40, 6100),
                                   (40, 30, 6000, 50)])
@pytest.mark.parametrize("bins", [3, 60])
def test_rare_alleles(sizes, genotypes, bins):
    if bins == 60 and (len(sizes) > 2 or sizes[0] > 20000):
        bins = 30
    rng = np.random.default_rng(sum(sizes) + genotypes)
    m = 70 if sizes[0] < 20000 else 26
    x, rows = rare(rng, sizes, m, genotypes)
    pos = np.cumsum(rng.integers(1, 40, size=m)).astype(np.float64)
    edges = np.linspace(0.0, 900.0, bins + 1)
    kw = dict(genotypes=genotypes, max_dist=900.0)
    got = parse.ld_parse(x, pos, rows, edges, method="tc", **kw).numpy()
    want = O.bin_sums(x, pos, rows, edges, **kw)
    stats = O.geno_stats if genotypes else O.hap_stats
    size = O.bin_sums(x, pos, rows, edges, stat_fn=lambda c, n: np.abs(stats(c, n)), **kw)["sums"]
    np.testing.assert_array_equal(got["pairs"], want["pairs"])
    np.testing.assert_array_equal(got["r2_counts"], want["r2_count"])
    assert np.max(np.abs(got["sums"] - want["sums"]) / np.maximum(size, 1e-300)) < 1e-11
    assert np.max(np.abs(got["r2_sums"] - want["r2_sum"]) / np.maximum(want["r2_sum"], 1e-300)) < 1e-11
