"""The first, tuning call of a shape class reports what every later one does: codes outside the
alphabet, unsorted positions, bootstrap blocks out of range -- and is not taken for a tuning."""
import numpy as np
import pytest

from pg_gpu_b200 import _lib, parse

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


@pytest.mark.parametrize("fault,text", [("code", "alphabet|codes"), ("positions", "unsorted"), ("block", "snp_block")])
def test_first_call_of_a_class(fault, text):
    rng = np.random.default_rng(5)
    m = 300
    hap = (rng.random((50, m)) < 0.4).astype(np.int8)
    pos = np.arange(1, m + 1, dtype=np.float64)
    blocks = np.zeros(m, np.int32)

    def run():
        return parse.ld_parse(hap, pos, [np.arange(50)], np.array([0.0, 20.0, 60.0]), method="tc", max_dist=60.0,
                              snp_block=blocks, n_blocks=2).numpy()

    good = (hap.copy(), pos.copy(), blocks.copy())
    _lib.autotune_clear()
    try:
        _lib.autotune(True)
        if fault == "code":
            hap[17, 123] = 5
        elif fault == "positions":
            pos[[40, 41]] = pos[[41, 40]]
        else:
            blocks[200:] = 2
        for _ in range(2):
            with pytest.raises(_lib.LdkError, match=text):
                run()
        assert _lib.autotune_count()[0] == 0
        hap, pos, blocks = good
        first = run()
        assert _lib.autotune_count()[0] == 1
        again = run()
        for k in first:
            np.testing.assert_array_equal(first[k], again[k])
    finally:
        _lib.autotune(False)
        _lib.autotune_clear()
