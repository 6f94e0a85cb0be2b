"""Bootstrap blocks outside [0, n_blocks) -- above, below, far below, some SNPs only -- are
reported by the tensor-core parse as by the plain one, and nothing is written for them: what lies
before and behind the outputs and the workspace stays as it was."""
import ctypes

import numpy as np
import pytest

from pg_gpu_b200 import _lib, parse

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("method", ["tc", "plain"])
@pytest.mark.parametrize("bad", [2, 70000, -1, -40, -2 ** 31])
@pytest.mark.parametrize("where", [slice(None), slice(64, 128), slice(199, 200)])
def test_reported_and_not_written(method, bad, where):
    rng = np.random.default_rng(3)
    m = 200
    hap = (rng.random((40, m)) < 0.4).astype(np.int8)
    pos = np.arange(1, m + 1, dtype=np.float64)
    blocks = np.repeat([0, 1], [128, m - 128]).astype(np.int32)
    blocks[where] = bad
    p = parse.Parser(hap, pos, [np.arange(40)], np.array([0.0, 20.0, 60.0]), method=method, max_dist=60.0, snp_block=blocks,
                     n_blocks=2)
    guard = 1 << 16
    need = int(_lib.load().ldk_parse_workspace_size(ctypes.byref(p.desc)))
    room = torch.full((need + 2 * guard,), 0x5A, dtype=torch.uint8, device="cuda")
    assert room.data_ptr() % 256 == 0
    outs = [torch.full((2 * 2 * k + 512,), 7, dtype=torch.int64, device="cuda") for k in (3, 1, 1, 1)]
    out = _lib.ParseOut(*[o.data_ptr() + 256 * 8 for o in outs])
    rc = _lib.load().ldk_parse(ctypes.byref(p.desc), ctypes.byref(out), room.data_ptr() + guard, need, None)
    torch.cuda.synchronize()
    assert rc == _lib.LDK_ERR_DEVICE and b"snp_block" in _lib.load().ldk_last_error()
    assert (room[:guard] == 0x5A).all() and (room[need + guard:] == 0x5A).all()
    for o in outs:
        assert (o[:256] == 7).all() and (o[-256:] == 7).all()
