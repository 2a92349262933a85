"""A batch's columns laid side by side for one copy: layout, joined reads,
and the same alignments whichever way the CIGAR words come back."""

from __future__ import annotations

import numpy as np
import pytest
import torch


def test_packed_layout_round_trip():
    from graphmambaformer_b200.device import pack_host, packed_layout

    cols = [np.arange(33, dtype=np.int64), np.zeros(0, np.int32), np.arange(-5, 250, dtype=np.int16).astype(np.int8),
            np.arange((1 << 18) + 3, dtype=np.int32), np.array([2.5])]  # empty, odd, and past 1 MB
    at, n = packed_layout([a.nbytes for a in cols])
    assert all(x % 256 == 0 for x in at) and n >= at[-1] + 8
    host = torch.zeros(n, dtype=torch.uint8)
    pack_host(cols, at, host)
    for a, x in zip(cols, at):
        assert np.array_equal(host.numpy()[x: x + a.nbytes].view(a.dtype), a)
    assert packed_layout([]) == ([], 256)


@pytest.mark.parametrize("dtype", [np.int8, np.int64, np.uint8])
@pytest.mark.parametrize("lens", [[3, 0, 5], [1], [0, 0]])
def test_join_codes_takes_what_concatenate_takes(dtype, lens):
    from graphmambaformer_b200.serving import _join_codes

    rng = np.random.default_rng(len(lens))
    reads = [rng.integers(0, 6, n).astype(dtype) for n in lens]
    total = sum(lens)
    out = np.full(max(total, 1), 77, np.int8)
    _join_codes(reads, out, total)
    assert np.array_equal(out, np.concatenate(reads).astype(np.int8) if total else np.zeros(1, np.int8))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 40])
def test_cigar_words_beside_results_or_after_them(monkeypatch, n):
    from graphmambaformer_b200 import serving, synth
    from graphmambaformer_b200.chaining import ChainingConfig
    from graphmambaformer_b200.config import ExtensionConfig

    pool = synth.mixed_read_pool(n_reads=40, seed=3, ref_len=500_000, max_len=4000)
    reads, anchors = pool.take(np.arange(n))
    al = serving.BatchAligner(torch.from_numpy(pool.ref).to("cuda:0"), "cuda:0", ChainingConfig(), ExtensionConfig())
    got = []
    for limit in (0, 1 << 40):
        monkeypatch.setattr(serving, "CIGAR_WITH_RESULTS", limit)
        got.append([list(x) for x in al.align(reads, anchors)])
    assert got[0] == got[1] and any(got[0])
