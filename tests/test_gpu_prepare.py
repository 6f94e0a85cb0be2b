"""The preparation of a parse: the plane kernel's block order and its sixteen-row gather (more
SNP tiles than one group of blocks holds, populations over several K tiles, remainders in
both), codes that are not in the alphabet wherever they stand, and the launches around it
(one-window parses have no plan, small ones take the narrower tile and one-tile items, many
bootstrap blocks are cleared by memsets).  Pair tallies exact; sums within 1e-6 of the oracle,
the tensor-core path's bound everywhere."""
import numpy as np
import pytest

from oracle import ld_oracle as O
from pg_gpu_b200 import parse, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _check(got, want):
    np.testing.assert_array_equal(got["pairs"], want["pairs"])
    np.testing.assert_array_equal(got["r2_counts"], want["r2_count"])
    for k, w in (("sums", want["sums"]), ("r2_sums", want["r2_sum"])):
        assert np.max(np.abs(got[k] - w) / np.maximum(np.abs(w), 1e-300)) < 1e-6


def _hap(rng, sizes, m):
    hap, _ = synth.haplotype_region(rng, list(sizes), m, m * 30, 0.03)
    offs = np.concatenate([[0], np.cumsum(sizes)])
    return hap, [np.arange(a, b) for a, b in zip(offs[:-1], offs[1:])]


# 1,027 SNPs are nine SNP tiles (a whole group of eight and one of the next); 130 and 260
# haplotypes fill two and three K tiles, 128 exactly one
@pytest.mark.parametrize("sizes,m", [((130,), 1027), ((128, 260), 1025), ((16, 15, 17), 131), ((144,), 1)])
@pytest.mark.parametrize("genotypes", [False, True])
def test_planes(sizes, m, genotypes):
    rng = np.random.default_rng(len(sizes) * 1000 + m)
    if genotypes and len(sizes) > 2:
        sizes = sizes[:2]
    data, rows = _hap(rng, sizes, m)
    if genotypes:
        data = np.where(data < 0, -1, data + (rng.random(data.shape) < 0.3)).astype(np.int8)
    pos = np.cumsum(rng.integers(1, 40, size=m)).astype(np.float64)
    edges = np.linspace(0.0, 700.0, 8)
    kw = dict(genotypes=genotypes, max_dist=700.0)
    _check(parse.ld_parse(data, pos, rows, edges, method="tc", **kw).numpy(), O.bin_sums(data, pos, rows, edges, **kw))


# the first and last haplotype of a warp's sixteen rows, of a K tile and of the population; SNPs at
# a quad's four places and the matrix's end; the codes around the alphabet and the byte's limits
@pytest.mark.parametrize("genotypes,codes", [(False, (2, 3, -2, 127, -128, 5)), (True, (3, 4, -2, 127, -128, 6))])
def test_codes_outside_the_alphabet_raise(genotypes, codes):
    rng = np.random.default_rng(11)
    m = 134
    data, rows = _hap(rng, (150,), m)
    pos = np.arange(1, m + 1, dtype=np.float64)
    edges = np.array([0.0, 5.0, 20.0])
    for k, (row, snp) in enumerate([(0, 0), (15, 1), (16, 2), (127, 3), (128, 127), (149, 133)]):
        bad = data.copy()
        bad[row, snp] = codes[k]
        with pytest.raises(Exception):
            parse.ld_parse(bad, pos, rows, edges, method="tc", genotypes=genotypes).numpy()
    parse.ld_parse(data, pos, rows, edges, method="tc", genotypes=genotypes).numpy()  # the device is still usable


# one window: a parse of no pairs, of one tile, of the most tiles that are spread one by one
# (24 row blocks x 6 tiles of 256) and of a few more; anchors cut off in a row block; two windows
@pytest.mark.parametrize("m", [2, 65, 400, 1500, 1600])
@pytest.mark.parametrize("cut", [None, 0.6, "windows"])
def test_small_parses(m, cut):
    rng = np.random.default_rng(m)
    data, rows = _hap(rng, (37,), m)
    pos = np.cumsum(rng.integers(1, 20, size=m)).astype(np.float64)
    edges = np.linspace(0.0, float(pos[-1]), 12)
    kw = dict(max_dist=float(pos[-1]))
    if cut == "windows":
        kw["window_offsets"] = np.array([0, m // 2, m])
    elif cut is not None:
        kw["anchor_end"] = [int(m * cut)]
    _check(parse.ld_parse(data, pos, rows, edges, method="tc", **kw).numpy(), O.bin_sums(data, pos, rows, edges, **kw))


# 2,000 bootstrap blocks of 64 bins for 100 SNPs: more accumulator words than the preparation's
# one SNP tile clears itself (64 a thread); 20 blocks: fewer (a row block of 64 SNPs may hold two
# consecutive bootstrap blocks)
@pytest.mark.parametrize("n_blocks", [20, 2000])
def test_clearing_of_many_blocks(n_blocks):
    rng = np.random.default_rng(n_blocks)
    m = 100
    data, rows = _hap(rng, (40,), m)
    pos = np.cumsum(rng.integers(1, 20, size=m)).astype(np.float64)
    edges = np.linspace(0.0, float(pos[-1]), 65)
    kw = dict(max_dist=float(pos[-1]), n_blocks=n_blocks,
              snp_block=np.repeat([n_blocks - 2, n_blocks - 1], [30, 70]).astype(np.int32))
    p = parse.Parser(data, pos, rows, edges, method="tc", **kw)
    want = O.bin_sums(data, pos, rows, edges, **kw)
    for _ in range(2):  # the second run clears what the first one left
        _check(p.run().numpy(), want)


# untuned genotypes of one population: 12 partners a tile up to 256 individuals or with no more
# tiles than SMs (1,100 SNPs are nine row blocks x 23 tiles of 48 by the rule's bound, 300 three x
# seven), else 24 where that leaves every warp its staging copy (32 bins do not)
@pytest.mark.parametrize("n,m,bins,width", [(256, 1100, 9, 12), (257, 1100, 9, 24), (257, 300, 9, 12),
                                            (400, 1100, 20, 24), (400, 1100, 32, 12)])
def test_genotype_tile_rule(n, m, bins, width):
    rng = np.random.default_rng(n + m)
    data, rows = _hap(rng, (n,), m)
    data = np.where(data < 0, -1, data + (rng.random(data.shape) < 0.3)).astype(np.int8)
    pos = np.cumsum(rng.integers(1, 40, size=m)).astype(np.float64)
    edges = np.linspace(0.0, 2000.0, bins + 1)
    kw = dict(genotypes=True, max_dist=2000.0)
    p = parse.Parser(data, pos, rows, edges, method="tc", **kw)
    assert p.tile_width() == width
    _check(p.run().numpy(), O.bin_sums(data, pos, rows, edges, **kw))
    assert p.reproducible()
