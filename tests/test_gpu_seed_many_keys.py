"""An index with more keys than the tile pass can number is seeded by the pass
per read, with the same results."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("both", [True, False])
def test_index_beyond_the_tile_pass(monkeypatch, both):
    import ctypes

    import torch

    from graphmambaformer_b200 import _native, seeding, synth

    rng = np.random.default_rng(10)
    ref = synth.random_reference(50_000, rng).astype(np.int8)
    idx = seeding.DeviceMinimizerIndex(ref, device="cuda:0")
    lens = [0, 14, 15, 700, 9_000] + [int(x) for x in rng.integers(20, 2000, 60)]
    off = np.zeros(len(lens) + 1, np.int64)
    np.cumsum(lens, out=off[1:])
    codes = torch.from_numpy(np.concatenate([ref[s: s + n] for s, n in zip(rng.integers(0, 40_000, len(lens)), lens)])).cuda()
    off_d = torch.from_numpy(off).cuda()
    want = idx.seed_device(codes, off_d, len(lens), both)
    monkeypatch.setattr(seeding, "TILE_KEYS", idx.n_keys - 1)
    large = seeding.DeviceMinimizerIndex(ref, device="cuda:0")
    assert large.prefix is None

    def refuse(*args):  # as gmf_seed_scan does for such an index
        raise AssertionError("the tile pass was used")

    monkeypatch.setattr(large, "_seed_tiles", refuse)
    got = large.seed_device(codes, off_d, len(lens), both)
    assert got["n_anchors"] == want["n_anchors"] > 0 and got["max_read_anchors"] == want["max_read_anchors"]
    assert torch.equal(got["read_off"], want["read_off"])
    for name in ("read_pos", "ref_pos", "length", "strand"):
        assert torch.equal(got[name], want[name]), name
    empty = large.seed_device(codes, off_d[:1], 0, both)
    assert empty["n_anchors"] == 0 and empty["read_off"].tolist() == [0]
    big = idx.c()
    big.n_keys = 2 ** 31  # refused before anything is launched
    assert _native.lib().gmf_seed_scan(ctypes.byref(big), None, 0, None, None, 0, 1, ctypes.c_void_p(off_d.data_ptr()),
                                       None, ctypes.c_void_p(off_d.data_ptr()), None, 0, None) == _native.GMF_ERR_LIMIT
