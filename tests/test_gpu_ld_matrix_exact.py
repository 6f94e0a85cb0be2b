"""sigma_D^2 of more haplotypes or individuals than the moment form is exact for (5,792), with
rare alleles: pairs whose DD and pi2 numerators are 0 (two singletons on one haplotype) stay 0
or NaN and out of the count, the others agree with the oracle to a few roundings (its numerators and
the kernel's are exact integers there, so 1e-13 is generous)."""
import numpy as np
import pytest

from oracle import ld_oracle as O
from pg_gpu_b200 import haplotype_matrix, ld_matrix, ld_statistics

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


def rare(rng, n, m, top):
    """Two to six carriers a site among the first twelve rows; the first four sites are singletons on
    rows 0, 0, 1 and 2, the next two are 0 and 1 wherever the other has a missing call."""
    x = np.zeros((n, m), np.int8)
    for v in range(m):
        x[rng.choice(12, size=rng.integers(2, 7), replace=False), v] = rng.integers(1, top + 1)
    x[:, :4] = 0
    x[[0, 0, 1, 2], [0, 1, 2, 3]] = 1
    return x


@pytest.mark.parametrize("n,m", [(5792, 70), (5793, 70), (20000, 130), (100003, 20)])
def test_haplotypes(n, m):
    rng = np.random.default_rng(n)
    x = rare(rng, n, m, 1)
    x[12:][rng.random((n - 12, m)) < 1e-3] = -1
    x[:, 4] = 1
    x[:7, 4] = -1  # constant among the called
    M, S = ld_matrix.ld_matrix(x, estimator="sigma_d2", reduce=True)
    want, valid = O.sigma_d2_matrix(x)
    got = M.cpu().numpy()
    assert want[0, 1] == 0 and got[0, 1] == 0 and not got[4].any()
    np.testing.assert_allclose(got, want, rtol=1e-13, atol=0)
    total, count = S.tolist()
    assert count == np.triu(valid, 1).sum()
    np.testing.assert_allclose(total, np.triu(want, 1).sum(), rtol=1e-11)


def test_zns_of_singletons():
    """Kelly's ZnS with the default estimator over sites of which many share their only carrier."""
    n, m = 20000, 40
    x = np.zeros((n, m), np.int8)
    x[np.arange(m) % 5, np.arange(m)] = 1
    x[5, ::2] = 1
    got = ld_statistics.zns(haplotype_matrix.HaplotypeMatrix(x, np.arange(m) * 10))
    np.testing.assert_allclose(got, O.zns(x), rtol=1e-11)


@pytest.mark.parametrize("n,m", [(5792, 70), (5793, 70), (20000, 130), (50001, 20)])
def test_genotypes(n, m):
    rng = np.random.default_rng(n)
    x = rare(rng, n, m, 2)
    M, S = ld_matrix.ld_matrix(x, estimator="sigma_d2_geno", reduce=True)
    want = O.sigma_d2_geno(x)
    got = M.cpu().numpy()[np.triu_indices(m, 1)]
    assert np.isnan(want[0]) and np.isnan(got[0])
    np.testing.assert_allclose(got, want, rtol=1e-13, atol=0, equal_nan=True)
    total, count = S.tolist()
    assert count == np.isfinite(want).sum()
    np.testing.assert_allclose(total, np.nansum(want), rtol=1e-11)
