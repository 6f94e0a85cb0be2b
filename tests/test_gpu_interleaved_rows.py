"""Two and three haplotype populations on both sides of the K extent from which the row block's rows
are interleaved (3,072 and 1,920 bytes): ragged populations, bootstrap blocks inside row blocks,
shared staging (64 bins), split anchors.  Pair tallies exact; per-bin sums within
the tensor-core path's 1e-6 of the oracle, as everywhere."""
import numpy as np
import pytest

from oracle import ld_oracle as O
from pg_gpu_b200 import parse, synth

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


@pytest.mark.parametrize("sizes", [(1400, 1500), (1500, 1500), (3001, 33), (33, 3001), (600, 600, 570), (600, 600, 600),
                                   (1900, 7, 5), (6000, 50), (50, 20, 5900)])
@pytest.mark.parametrize("bins,blocks,cut", [(16, False, None), (9, True, 100), (64, False, None)])
def test_sums(sizes, bins, blocks, cut):
    rng = np.random.default_rng(sum(sizes) + bins)
    m = 150
    hap, _ = synth.haplotype_region(rng, list(sizes), m, m * 30, 0.03)
    pos = np.cumsum(rng.integers(1, 40, size=m)).astype(np.float64)
    offs = np.concatenate([[0], np.cumsum(sizes)])
    rows = [rng.permutation(np.arange(a, b)) for a, b in zip(offs[:-1], offs[1:])]
    edges = np.linspace(0.0, 1500.0, bins + 1)
    kw = dict(max_dist=1500.0)
    if blocks:
        kw.update(snp_block=(np.arange(m) // 50).astype(np.int32), n_blocks=3)
    if cut is not None:
        kw["anchor_end"] = [cut]
    got = parse.ld_parse(hap, pos, rows, edges, method="tc", **kw).numpy()
    want = O.bin_sums(hap, pos, rows, edges, **kw)
    np.testing.assert_array_equal(got["pairs"], want["pairs"])
    np.testing.assert_array_equal(got["r2_counts"], want["r2_count"])
    for k, w in (("sums", want["sums"]), ("r2_sums", want["r2_sum"])):
        assert np.max(np.abs(got[k] - w) / np.maximum(np.abs(w), 1e-300)) < 1e-6
