"""Pair-list counts through bit planes and the per-SNP call counts, against the oracle: rows
that fill a word exactly, leave one bit or spill into the next, SNP counts around the four-SNP
loads, an unaligned matrix, codes outside {-1, 0, 1} (counted as valid, in no cell), and
populations with and without missing entries.  Whole numbers: exact."""
import numpy as np
import pytest

from oracle import ld_oracle as O
from pg_gpu_b200 import ld_matrix, ld_pipeline

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n_rows", [1, 31, 32, 33, 64, 100])
@pytest.mark.parametrize("m", [2, 5, 127, 130, 515])
def test_counts_match_oracle(n_rows, m):
    rng = np.random.default_rng(n_rows * 1000 + m)
    hap = rng.integers(0, 2, (n_rows + 7, m)).astype(np.int8)
    hap[rng.random(hap.shape) < 0.05] = -1
    hap[rng.random(hap.shape) < 0.02] = 2
    rows = rng.permutation(n_rows + 7)[:n_rows]
    i = rng.integers(0, m, 700)
    j = rng.integers(0, m, 700)
    want, nv = O.hap_counts(hap, i, j, rows)
    X = torch.empty(hap.size + 3, dtype=torch.int8, device="cuda")[3:].view(hap.shape)  # off the word grid
    X.copy_(torch.as_tensor(hap))
    got, n = ld_pipeline.compute_counts_for_pairs(X, i, j, rows)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    assert (n is None) == (not (hap[rows] == -1).any())
    if n is not None:
        x, y = hap[rows][:, i], hap[rows][:, j]
        np.testing.assert_array_equal(n.cpu().numpy(), ((x >= 0) & (y >= 0)).sum(0))


def test_counts_complete_population_and_bad_row():
    hap = np.random.default_rng(1).integers(0, 2, (40, 50)).astype(np.int8)
    hap[39, 3] = -1
    i, j = np.arange(49), np.arange(1, 50)
    assert ld_pipeline.compute_counts_for_pairs(hap, i, j, np.arange(39))[1] is None
    assert ld_pipeline.compute_counts_for_pairs(hap, i, j)[1] is not None
    with pytest.raises(IndexError):
        ld_pipeline.compute_counts_for_pairs(hap, i, j, [0, 40])


@pytest.mark.parametrize("n,m", [(1, 3), (8, 128), (129, 131), (300, 1030)])
@pytest.mark.parametrize("md", ["include", "exclude"])
def test_segregating_sites(n, m, md):
    rng = np.random.default_rng(n + m)
    hap = (rng.random((n, m)) < rng.choice([0.0, 0.3, 1.0], m)).astype(np.int8)
    hap[rng.random(hap.shape) < 0.5 / n] = -1
    np.testing.assert_array_equal(ld_matrix.segregating(hap, md).cpu().numpy(), O.segregating(hap, md))


@pytest.mark.parametrize("P", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 31, 129, 1000])
def test_statistics_rows(P, n):
    """Blocks of 128 (four populations: 32) pairs written as one run: partial last blocks."""
    rng = np.random.default_rng(P * 10 + n)
    c = [rng.multinomial(30, [0.3, 0.2, 0.2, 0.3], size=n).astype(np.int32) for _ in range(P)]
    buf = torch.empty(4 * n + 1, dtype=torch.int32, device="cuda")[1:].view(n, 4)  # off the 16-byte grid
    buf.copy_(torch.as_tensor(c[0]))
    got = ld_pipeline.compute_multi_pop_statistics_batch([buf] + c[1:]).cpu().numpy()
    np.testing.assert_allclose(got, O.hap_stats(c), rtol=1e-11, atol=1e-15)
