"""Seeding in ranges of reads gives what one pass gives, in a bounded amount
of device memory: ranges of many reads, reads above the budget, a code buffer
larger than its reads, no anchors at all, and another stream."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("budget", [1 << 14, 1 << 17, 1 << 20])
@pytest.mark.parametrize("both", [True, False])
def test_ranges_equal_one_pass(monkeypatch, budget, both):
    import torch

    from graphmambaformer_b200 import seeding, synth

    rng = np.random.default_rng(8)
    ref = synth.random_reference(40_000, rng).astype(np.int8)
    idx = seeding.DeviceMinimizerIndex(ref, k=15, w=10, device="cuda:0")
    lens = [0, 9, 600, 12_000, 0, 0] + [int(x) for x in rng.integers(20, 900, 200)] + [0]
    off = np.zeros(len(lens) + 1, np.int64)
    np.cumsum(lens, out=off[1:])
    off += 333  # the buffer begins before the first read and ends beyond the last one
    codes = np.concatenate([ref[:333]] + [ref[s: s + n] for s, n in zip(rng.integers(0, 25_000, len(lens)), lens)]
                           + [ref[:5000]])
    codes_d, off_d = torch.from_numpy(codes).cuda(), torch.from_numpy(off).cuda()
    want = idx.seed_device(codes_d, off_d, len(lens), both)
    monkeypatch.setattr(seeding, "SEED_WORKSPACE", budget)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    for s in (None, stream):
        got = idx.seed_device(codes_d, off_d, len(lens), both, stream=s)
        torch.cuda.synchronize()
        assert got["n_anchors"] == want["n_anchors"] > 1000
        assert got["max_read_anchors"] == want["max_read_anchors"]
        assert torch.equal(got["read_off"], want["read_off"])
        for name in ("read_pos", "ref_pos", "length", "strand"):
            t = want["n_anchors"]
            assert got[name].dtype == want[name].dtype and torch.equal(got[name][:t], want[name][:t]), name
    none = idx.seed_device(torch.full_like(codes_d, 5), off_d, len(lens), both)
    assert none["n_anchors"] == 0 and none["read_pos"].numel() == 1 and int(none["read_off"][-1]) == 0


def test_many_short_reads_take_a_bounded_workspace():
    import torch

    from graphmambaformer_b200 import seeding, synth

    ref = synth.random_reference(300_000, np.random.default_rng(9)).astype(np.int8)
    idx = seeding.DeviceMinimizerIndex(ref, k=15, w=10, device="cuda:0")
    n, L = 400_000, 100
    at = torch.randint(0, 299_000, (n, 1), device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    codes = torch.from_numpy(ref).cuda()[(at + torch.arange(L, device="cuda")).reshape(-1)]
    off = torch.arange(n + 1, device="cuda") * L
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    out = idx.seed_device(codes, off, n)
    results = sum(out[x].numel() * out[x].element_size() for x in ("read_pos", "ref_pos", "length", "strand", "read_off"))
    assert torch.cuda.max_memory_allocated() - before <= seeding.SEED_WORKSPACE + 3 * results
    assert out["n_anchors"] > n  # most reads lie on the reference
