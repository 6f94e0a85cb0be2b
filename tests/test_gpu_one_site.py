"""A set of one SNP has no pair: the complete-data estimators give its 1 x 1 NaN whether or not a
call is missing, and refuse the missing call as soon as there are two SNPs."""
import numpy as np
import pytest

from pg_gpu_b200 import _lib, ld_matrix

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


@pytest.mark.parametrize("estimator", ["rogers_huff_r", "sigma_d2_geno"])
def test_missing_call(estimator):
    x = np.array([[0], [1], [-1], [2], [1]], np.int8)
    M, S = ld_matrix.ld_matrix(x, estimator=estimator, reduce=True)
    assert M.shape == (1, 1) and np.isnan(M.cpu().numpy()[0, 0]) and S.tolist() == [0.0, 0.0]
    with pytest.raises(_lib.LdkError):
        ld_matrix.ld_matrix(np.hstack([x, x]), estimator=estimator)
