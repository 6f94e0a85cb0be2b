"""Work items around one piece per SM: 73 and 74 row blocks (the least that are kept whole where their
pieces would need a second round), 86, and 148 of two or three tiles, one window and several.
Pair tallies exact; per-bin sums within the tensor-core path's 1e-6 of the oracle, as everywhere."""
import numpy as np
import pytest

from oracle import ld_oracle as O
from pg_gpu_b200 import parse, synth

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


@pytest.mark.parametrize("m", [4672, 4673, 5500, 9472])
@pytest.mark.parametrize("sizes", [(21,), (12, 9)])
@pytest.mark.parametrize("windows", [1, 3])
def test_row_blocks(m, sizes, windows):
    rng = np.random.default_rng(m + len(sizes))
    hap, _ = synth.haplotype_region(rng, list(sizes), m, m * 30, 0.02)
    pos = np.cumsum(rng.integers(1, 20, size=m)).astype(np.float64)
    offs = np.concatenate([[0], np.cumsum(sizes)])
    rows = [np.arange(a, b) for a, b in zip(offs[:-1], offs[1:])]
    edges = np.linspace(0.0, 500.0, 9)
    kw = dict(max_dist=500.0)
    if windows > 1:
        kw["window_offsets"] = np.linspace(0, m, windows + 1).astype(np.int64)
    got = parse.ld_parse(hap, pos, rows, edges, method="tc", **kw).numpy()
    want = O.bin_sums(hap, pos, rows, edges, **kw)
    np.testing.assert_array_equal(got["pairs"], want["pairs"])
    np.testing.assert_array_equal(got["r2_counts"], want["r2_count"])
    for k, w in (("sums", want["sums"]), ("r2_sums", want["r2_sum"])):
        assert np.max(np.abs(got[k] - w) / np.maximum(np.abs(w), 1e-300)) < 1e-6
