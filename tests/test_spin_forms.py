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


def test_weights_are_powers_of_two_and_the_order_is_a_permutation():
    """The weights are applied once per staged sum, so they must scale exactly; the staged
    order holds every statistic and r^2 once, the one-population statistics and r^2 first where
    two warps share a pair."""
    for P in (1, 2, 3, 4):
        for geno in (False, True):
            stats = G.spin_stats(P, geno)
            assert all((1 / w).is_integer() and (int(1 / w) & (int(1 / w) - 1)) == 0 for _, w, *_ in stats)
            order, K = G.spin_order(P, geno)
            assert sorted(order) == list(range(len(stats) + 1))
            assert (K > 0) == (not geno and P == 4)
            assert all(k == len(stats) or not stats[k][0].startswith("pi2") or len(set(stats[k][0].split("_")[1:])) == 1
                       for k in order[:K])
