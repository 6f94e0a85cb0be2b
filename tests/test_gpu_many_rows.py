"""Pair counts of more rows than one launch has blocks for in y (65,535 words of 32 rows): rows of
the second round of a block, and the ragged last word.  Whole numbers: exact."""
import numpy as np
import pytest

from pg_gpu_b200 import ld_pipeline

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n_rows", [32 * 65535, 32 * 65535 + 1, 32 * 65535 + 70])
def test_counts(n_rows):
    gen = torch.Generator(device="cuda").manual_seed(n_rows)
    x = torch.randint(0, 2, (n_rows, 5), dtype=torch.int8, device="cuda", generator=gen)
    x[n_rows - 1, 3] = -1
    x[7, 1] = -1
    i, j = np.array([0, 1, 0, 2, 3]), np.array([1, 3, 3, 4, 4])
    got, nv = ld_pipeline.compute_counts_for_pairs(x, i, j)
    a, b = x[:, i], x[:, j]
    want = torch.stack([((a == p) & (b == q)).sum(0) for p, q in ((1, 1), (1, 0), (0, 1), (0, 0))], 1)
    assert (got == want).all() and (nv == ((a >= 0) & (b >= 0)).sum(0)).all()
