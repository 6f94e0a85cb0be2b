"""Dosage r^2 and Rogers-Huff r of rare alleles: the covariance of carriers that do not meet is
minus the product of two small sums over n, which a difference of sums near n loses.  Against
rational arithmetic; each value has about a dozen roundings and no cancellation, so 1e-13
relative."""
from fractions import Fraction

import numpy as np
import pytest

from pg_gpu_b200 import ld_matrix

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


def rare(rng, n, m):
    """One to four carriers a site in the lower rows, none of them shared but by every sixth site."""
    x = np.zeros((n, m), np.int8)
    for v in range(m):
        x[5 * v:5 * v + rng.integers(1, 5), v] = rng.integers(1, 3)
    x[:, 5::6] = x[:, 4:-1:6]
    return x


def covariance(x, y, mx, my):
    both = (x >= 0) & (y >= 0)
    a, b = x[both].astype(np.int64), y[both].astype(np.int64)
    return int((a * b).sum()) - my * int(a.sum()) - mx * int(b.sum()) + mx * my * int(both.sum())


def site(x):
    v = x[x >= 0].astype(np.int64)
    m = Fraction(int(v.sum()), len(v))
    return m, int((v * v).sum()) - len(v) * m * m


@pytest.mark.parametrize("n", [330, 20000])
@pytest.mark.parametrize("missing", [False, True])
def test_rare_dosages(n, missing):
    rng = np.random.default_rng(n)
    m = 60
    x = rare(rng, n, m)
    if missing:
        x[300:][rng.random((n - 300, m)) < 0.02] = -1
    M = ld_matrix.ld_matrix(x, estimator="diploid_r2")[0].cpu().numpy()
    R = None if missing else ld_matrix.ld_matrix(x, estimator="rogers_huff_r")[0].cpu().numpy()
    sites = [site(x[:, v]) for v in range(m)]
    for i in range(0, m, 3):
        for j in range(i + 1, m, 2):
            (mi, vi), (mj, vj) = sites[i], sites[j]
            c = covariance(x[:, i], x[:, j], mi, mj)
            want = c * c / (vi * vj)
            assert abs(Fraction(M[i, j]) - want) <= want / 10 ** 13
            if R is not None:
                assert (R[i, j] < 0) == (c < 0) and abs(Fraction(R[i, j]) ** 2 - want) <= 2 * want / 10 ** 13
