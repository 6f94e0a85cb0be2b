"""The bin flush that adds lane by lane: bins of about one partner, of a few and of many, in one
parse (items of both kinds side by side, at the window's end too), with eight, four, two, one and no
scratch rows per warp (three and two populations by bins and table, bootstrap blocks), and with
the wide genotype tile.  Pair tallies exact; per-bin sums within the tensor-core path's 1e-6 of the
oracle, as everywhere."""
import numpy as np
import pytest

from oracle import ld_oracle as O
from pg_gpu_b200 import parse, synth

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


@pytest.mark.parametrize("genotypes,sizes,bins,blocks,m", [
    (False, (40, 30, 20), 16, True, 700), (False, (40, 30, 20), 18, True, 700), (False, (40, 30, 20), 20, True, 700),
    (False, (40, 30, 20), 21, True, 700), (False, (60, 20, 11), 40, True, 400), (False, (300, 20, 11), 20, True, 400),
    (False, (40, 30, 20), 16, False, 700), (False, (40, 30), 62, True, 700), (False, (40, 30), 64, True, 700),
    (False, (60,), 64, False, 700), (True, (290,), 20, False, 1300), (True, (290,), 24, True, 1300),
    (True, (60,), 40, True, 500)])
@pytest.mark.parametrize("width", [1, 4, 30])
def test_bins_of_few_partners(genotypes, sizes, bins, blocks, m, width):
    rng = np.random.default_rng(bins * 100 + width)
    data, _ = synth.haplotype_region(rng, list(sizes), m, m * 30, 0.03)
    if genotypes:
        data = np.where(data < 0, -1, data + (rng.random(data.shape) < 0.3)).astype(np.int8)
    gap = rng.integers(5, 15, size=m).astype(np.float64)
    gap[m // 3:m // 2] *= 20.0  # a sparse stretch: fewer partners per bin than elsewhere
    pos = np.cumsum(gap)
    offs = np.concatenate([[0], np.cumsum(sizes)])
    rows = [np.arange(a, b) for a, b in zip(offs[:-1], offs[1:])]
    edges = np.linspace(0.0, 10.0 * width * bins, bins + 1)
    kw = dict(genotypes=genotypes, max_dist=float(edges[-1]))
    if blocks:
        kw.update(snp_block=(np.arange(m) // 150).astype(np.int32), n_blocks=m // 150 + 1)
    got = parse.ld_parse(data, pos, rows, edges, method="tc", **kw).numpy()
    want = O.bin_sums(data, pos, rows, edges, **kw)
    np.testing.assert_array_equal(got["pairs"], want["pairs"])
    np.testing.assert_array_equal(got["r2_counts"], want["r2_count"])
    for k, w in (("sums", want["sums"]), ("r2_sums", want["r2_sum"])):
        assert np.max(np.abs(got[k] - w) / np.maximum(np.abs(w), 1e-300)) < 1e-6
