"""Block sums under bootstrap weights at the edges of the sixteen blocks that are loaded
together.  The blocks are added in order with one rounding each, so whole-number sums are exact;
a block of weight 0 is left out even where its sum is not finite."""
import numpy as np
import pytest

from pg_gpu_b200 import parse

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n_blocks", [1, 15, 16, 17, 33])
def test_block_combine_edges(n_blocks):
    rng = np.random.default_rng(n_blocks)
    bs = rng.integers(-1000, 1000, size=(n_blocks, 5, 3)).astype(np.float64)
    w = rng.integers(0, 4, size=(6, n_blocks)).astype(np.int32)
    dead = n_blocks - 1
    w[:, dead] = 0
    want = np.tensordot(w, bs, axes=(1, 0))
    bs[dead] = np.array([np.inf, -np.inf, np.nan])
    got = parse.block_combine(torch.as_tensor(bs, device="cuda"), w).cpu().numpy()
    np.testing.assert_array_equal(got, want)
