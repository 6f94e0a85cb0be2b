"""Shapes whose staging and reciprocal table end within the last bytes of a CTA's shared memory,
where the kernel's own __shared__ variables (640 to 736 bytes) decide whether they fit: they run,
with whatever staging is left.  Bootstrap blocks, so that every slot is staged.  Pair tallies
exact; per-bin sums within the tensor-core path's 1e-6 of the oracle, as everywhere."""
import numpy as np
import pytest

from oracle import ld_oracle as O
from pg_gpu_b200 import parse, synth

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


@pytest.mark.parametrize("genotypes,sizes,bins", [
    (True, (90,), 33), (True, (90,), 34), (True, (90,), 35), (False, (4451, 40), 1), (False, (4452, 40), 1),
    (False, (4480, 40), 1), (False, (190, 33), 64), (False, (200, 20, 11), 21), (False, (375, 20, 11), 20),
    (False, (376, 20, 11), 20), (False, (398, 20, 11), 20), (False, (399, 20, 11), 20), (False, (1128, 20, 11), 16),
    (False, (1150, 20, 11), 16), (False, (712, 20, 11, 15), 64), (False, (3708, 20, 11, 15), 1)])
def test_last_bytes(genotypes, sizes, bins):
    rng = np.random.default_rng(sizes[0] + bins)
    m = 200
    data, _ = synth.haplotype_region(rng, list(sizes), m, m * 30, 0.03)
    if genotypes:
        data = np.where(data < 0, -1, data + (rng.random(data.shape) < 0.3)).astype(np.int8)
    pos = np.cumsum(rng.integers(1, 40, size=m)).astype(np.float64)
    offs = np.concatenate([[0], np.cumsum(sizes)])
    rows = [np.arange(a, b) for a, b in zip(offs[:-1], offs[1:])]
    blocks = (pos // 2500).astype(np.int32)
    edges = np.linspace(0.0, 2000.0, bins + 1)
    kw = dict(genotypes=genotypes, max_dist=2000.0, snp_block=blocks, n_blocks=int(blocks.max()) + 1)
    got = parse.ld_parse(data, pos, rows, edges, method="tc", **kw).numpy()
    want = O.bin_sums(data, pos, rows, edges, **kw)
    np.testing.assert_array_equal(got["pairs"], want["pairs"])
    np.testing.assert_array_equal(got["r2_counts"], want["r2_count"])
    for k, w in (("sums", want["sums"]), ("r2_sums", want["r2_sum"])):
        assert np.max(np.abs(got[k] - w) / np.maximum(np.abs(w), 1e-300)) < 1e-6
