"""The statistic-level forms the tensor-core parse evaluates (spin moments of the jointly
called individuals) against the raw estimator calls they stand for, in rational arithmetic
(no tolerance): random counts of both paths, and haplotype samples of 0 to 5, where the
reciprocals of zero products are 0."""
import pytest

from pg_gpu_b200.csrc import gen_estimators as G


@pytest.mark.parametrize("small", [False, True])
@pytest.mark.parametrize("seed", [1, 2])
def test_spin_forms_equal_raw_calls(seed, small):
    assert G.check_spin(seed=seed, trials=40 if small else 10, small_haplotypes=small)


def test_weights_are_powers_of_two_and_split_separates_pi2():
    """The weights are applied once per staged sum, so they must scale exactly; the two halves
    of the statistics split at the first pi2."""
    for P in (1, 2, 3, 4):
        for geno in (False, True):
            assert all((1 / w).is_integer() and (int(1 / w) & (int(1 / w) - 1)) == 0 for _, w, *_ in G.spin_stats(P, geno))
        names = [n for n, *_ in G.spin_stats(P, False)]
        K = G.spin_split(P)
        assert all(n.startswith("pi2") for n in names[K:]) and not any(n.startswith("pi2") for n in names[:K])
