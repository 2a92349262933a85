"""Batches of as many pairs as there are blocks, one more, twice as many, and
about as many as there are warps, with some long pairs first: every pair is
computed once, whatever the number that a block takes."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 147, 148, 149, 296, 297, 4735, 4737])
@pytest.mark.parametrize("long_pairs,bound", [(0, 4096), (3, 4096), (3, 9000)])
def test_batches_around_the_number_of_blocks(n, long_pairs, bound):
    from graphmambaformer_b200 import synth
    from graphmambaformer_b200.wfa import align_wfa_pairs, upload_wfa_pairs, wfa_distances
    from oracle import oracle

    rng = np.random.default_rng(n)
    ref = synth.random_reference(40_000, rng).astype(np.int8)
    qs, ts = [], []
    for b in range(n):
        L = 9_100 if bound == 9000 and b == 0 and long_pairs else 4_200 if b < long_pairs else int(rng.integers(1, 90))
        s = int(rng.integers(0, 25_000))
        qs.append(synth.apply_errors(ref[s: s + L], synth.ONT, rng).astype(np.int8))
        ts.append(ref[s: s + L])
    dist = wfa_distances(upload_wfa_pairs(qs, ts), bound).cpu().numpy()
    r = align_wfa_pairs(qs, ts, bound)
    assert np.array_equal(dist, r.distance)
    assert np.array_equal(r.op_counts[:, 1:].sum(1), r.distance)
    for b in list(range(min(n, 60))) + [n - 1]:
        d, cigar = oracle.wfa_align(qs[b], ts[b], bound)
        assert int(dist[b]) == d and r.cigar(b) == cigar, b
