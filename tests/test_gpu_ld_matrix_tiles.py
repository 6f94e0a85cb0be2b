"""All-pairs LD where the kernel takes another branch: more haplotypes than the 1/n table in
shared memory holds, sets whose 64 x 128 tiles are whole, ragged and on the diagonal, and a
matrix wide enough that the row blocks are cut into several work items.  1e-12 relative
(1e-15 absolute) of the float64 oracle, as for the other matrix tests."""
import numpy as np
import pytest

from oracle import ld_oracle as O
from pg_gpu_b200 import ld_matrix

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


def codes(rng, n, m, top):
    x = rng.binomial(top, rng.uniform(0.05, 0.6, m), size=(n, m)).astype(np.int8)
    x[rng.random(x.shape) < 0.03] = -1
    return x


@pytest.mark.parametrize("n,m", [(8191, 70), (8300, 70), (60, 1), (60, 2), (60, 192), (60, 193), (33, 1500)])
def test_r2_matrix(n, m):
    x = codes(np.random.default_rng(n + m), n, m, 1)
    M, S = ld_matrix.ld_matrix(x, estimator="r2", reduce=True)
    want = O.pairwise_r2_matrix(x)
    np.testing.assert_allclose(M.cpu().numpy(), want, rtol=1e-12, atol=1e-15)
    total, count = S.tolist()
    assert count == m * (m - 1) // 2
    np.testing.assert_allclose(total, np.triu(want, 1).sum(), rtol=1e-11, atol=1e-14)


@pytest.mark.parametrize("m", [1, 2, 65, 192, 500])
def test_dosage_matrix(m):
    x = codes(np.random.default_rng(m), 70, m, 2)
    np.testing.assert_allclose(ld_matrix.diploid_r2_matrix(x).cpu().numpy(), O.diploid_r2_matrix(x), rtol=1e-12, atol=1e-15)
