"""A tuned choice meets every shape of its class, also those it cannot run: three haplotype
populations of 400 + 400 + 420 and of 1,200 + 20 + 20 pad to the same 1,280 bytes, but the second
keeps its reciprocal table in the workspace, which the narrow tile does not read; a class of so
many bytes that its rows are interleaved has no such tile at all.  Host-only: the width a call
would use."""
import ctypes
import json

import pytest

from pg_gpu_b200 import _lib


def desc(sizes, nb):
    d = _lib.ParseDesc()
    d.n_pops, d.genotypes, d.n_bins, d.n_blocks, d.method, d.max_dist = len(sizes), 0, nb, 1, _lib.METHOD_TC, 1.0
    for k in range(nb + 1):
        d.edges[k] = float(k)
    for k in range(5):
        d.pop_offsets[k] = sum(sizes[:k])
    return d


@pytest.mark.parametrize("k_bytes,shapes,widths", [
    (1280, [(400, 400, 420), (1200, 20, 20)], [16, 32]),
    (4608, [(2300, 2200), (3500, 1000)], [48, 48])])
def test_width_of_a_shape_the_choice_does_not_fit(tmp_path, k_bytes, shapes, widths):
    lib = _lib.load()
    path = tmp_path / "t.json"
    path.write_text('{"format": "ldk-autotune", "version": 1, "entries": [\n' + json.dumps(
        {"pops": len(shapes[0]), "genotypes": 0, "k_bytes": k_bytes, "bins": 16, "cutoff_decade": 0, "window_log2": 0,
         "tile_variant": 1, "tile_partners": 16, "order": 0, "ms": 1.0}) + "\n]}\n")
    try:
        _lib.autotune_load(str(path))
        assert [lib.ldk_tile_width(ctypes.byref(desc(s, 16))) for s in shapes] == widths
    finally:
        _lib.autotune_clear()
