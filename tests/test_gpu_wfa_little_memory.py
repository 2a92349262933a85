"""A device without room for the one-pass history (sized by a guess) still
aligns every pair whose own histories fit, as the two-pass form did."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_alignment_when_the_guessed_history_does_not_fit():
    import torch

    from graphmambaformer_b200 import _native, synth, wfa

    rng = np.random.default_rng(12)
    ref = synth.random_reference(60_000, rng).astype(np.int8)
    qs, ts = [], []
    for n in [int(x) for x in rng.integers(200, 9_000, 60)] + [0, 5]:
        s = int(rng.integers(0, 50_000))
        qs.append(synth.apply_errors(ref[s: s + n], synth.HIFI, rng).astype(np.int8))
        ts.append(ref[s: s + n])
    ts[-2] = ref[:7]
    dp = wfa.upload_wfa_pairs(qs, ts)
    want = wfa.align_device_pairs(dp, 4096)
    f = _native.lib().gmf_wfa_workspace_bytes
    exact = int(((want.distance.astype(np.int64) + 1) ** 2).sum())
    room = f(dp.n, dp.max_len, 4096, exact)
    guess = f(dp.n, dp.max_len, 4096, wfa.direct_entries(dp.h_qlen, dp.h_tlen, 4096))
    assert room < guess
    asked = []

    def workspace(nbytes):
        asked.append(nbytes)
        if nbytes > room:
            raise torch.OutOfMemoryError("no room")
        return torch.empty(nbytes, dtype=torch.uint8, device="cuda")

    got = wfa.align_device_pairs(dp, 4096, workspace=workspace)
    assert asked[0] > room and len(asked) > 1
    assert np.array_equal(got.distance, want.distance) and np.array_equal(got.op_counts, want.op_counts)
    for b in range(dp.n):
        assert got.cigar(b) == want.cigar(b), b
