"""Valid counts handed to the batch statistics in lists that are longer than the populations
(further ones of the right length are not used) or hold None for some of them (the counts' sum)."""
import numpy as np
import pytest

from oracle import ld_oracle as O
from pg_gpu_b200 import ld_pipeline

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


@pytest.mark.parametrize("genotypes", [False, True])
def test_valid_count_lists(genotypes):
    rng = np.random.default_rng(2)
    k = 9 if genotypes else 4
    c = [rng.multinomial(40, np.full(k, 1 / k), size=50).astype(np.int32) for _ in range(2)]
    nv = [x.sum(1, dtype=np.int32) for x in c]
    want = (O.geno_stats if genotypes else O.hap_stats)(c)
    for lists in (nv, nv + [nv[0]], [None, nv[1]], [None, nv[1], nv[1]], [None] * 3, None):
        got = ld_pipeline.compute_multi_pop_statistics_batch(c, lists, genotypes=genotypes).cpu().numpy()
        np.testing.assert_allclose(got, want, rtol=1e-10, atol=1e-14)
    for lists, error in ((nv + [np.zeros(3, np.int32)], RuntimeError), (nv + [None], IndexError),
                         (nv[:1] + [nv[1][:9]], RuntimeError)):
        with pytest.raises(error):
            ld_pipeline.compute_multi_pop_statistics_batch(c, lists, genotypes=genotypes)
