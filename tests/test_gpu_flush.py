"""The bin flush of the tensor-core parse at the edges of its shared-memory room: three
populations and twenty bins leave eight, one or no scratch rows per epilogue warp,
depending on the largest population (its reciprocal table), and many bins share one staging
copy (atomics).  Bootstrap blocks change inside row blocks, so lanes of one warp flush
different (block, bin) sums in the same step.  Pair tallies exact; per-bin sums within the
tensor-core path's 1e-6 of the oracle, as everywhere."""
import numpy as np
import pytest

from oracle import ld_oracle as O
from pg_gpu_b200 import parse, synth

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


@pytest.mark.parametrize("sizes,bins", [((60, 20, 11), 20), ((200, 20, 11), 20), ((300, 20, 11), 20), ((350, 20, 11), 20),
                                        ((60, 20, 11), 40), ((70, 33), 64), ((90,), 64), ((30, 20, 25, 12), 16)])
def test_flush_rows(sizes, bins):
    rng = np.random.default_rng(7 * len(sizes) + bins)
    m = 330
    hap, _ = synth.haplotype_region(rng, list(sizes), m, m * 30, 0.03)
    pos = np.cumsum(rng.integers(1, 40, size=m)).astype(np.float64)
    offs = np.concatenate([[0], np.cumsum(sizes)])
    rows = [np.arange(a, b) for a, b in zip(offs[:-1], offs[1:])]
    blocks = (pos // 2500).astype(np.int32)
    edges = np.linspace(0.0, 4000.0, bins + 1)
    kw = dict(max_dist=4000.0, snp_block=blocks, n_blocks=int(blocks.max()) + 1)
    got = parse.ld_parse(hap, pos, rows, edges, method="tc", **kw).numpy()
    want = O.bin_sums(hap, pos, rows, edges, **kw)
    np.testing.assert_array_equal(got["pairs"], want["pairs"])
    np.testing.assert_array_equal(got["r2_counts"], want["r2_count"])
    for k, w in (("sums", want["sums"]), ("r2_sums", want["r2_sum"])):
        assert np.max(np.abs(got[k] - w) / np.maximum(np.abs(w), 1e-300)) < 1e-6
