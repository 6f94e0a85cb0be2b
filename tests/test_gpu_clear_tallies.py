"""Pair tallies of many bootstrap blocks are cleared by memsets, those of few by the preparation:
just below, at and above 64 words a thread of the one SNP tile (8,192 words), a second run clears
what the first one left."""
import numpy as np
import pytest

from oracle import ld_oracle as O
from pg_gpu_b200 import parse

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


@pytest.mark.parametrize("n_blocks", [4095, 4096, 4097, 50000])
def test_runs_after_one_another(n_blocks):
    rng = np.random.default_rng(n_blocks)
    m = 90
    hap = (rng.random((30, m)) < 0.4).astype(np.int8)
    pos = np.arange(1, m + 1, dtype=np.float64)
    edges = np.array([0.0, 20.0, 60.0])
    blocks = np.repeat([0, n_blocks - 1], [64, m - 64]).astype(np.int32)
    kw = dict(max_dist=60.0, snp_block=blocks, n_blocks=n_blocks)
    p = parse.Parser(hap, pos, [np.arange(30)], edges, method="tc", **kw)
    want = O.bin_sums(hap, pos, [np.arange(30)], edges, **kw)
    for _ in range(2):
        p.out.pairs.fill_(7)
        p.out.r2_counts.fill_(9)
        got = p.run().numpy()
        np.testing.assert_array_equal(got["pairs"], want["pairs"])
        np.testing.assert_array_equal(got["r2_counts"], want["r2_count"])
        assert np.max(np.abs(got["sums"] - want["sums"]) / np.maximum(np.abs(want["sums"]), 1e-300)) < 1e-6
