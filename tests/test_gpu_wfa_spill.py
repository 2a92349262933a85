"""Pairs whose wavefronts leave shared memory: one-warp pairs (sides up to
3999, 16-bit slots claimed by the warps) and whole-block ones around the
length where they change over, more of them than there are warps in a block,
under bounds of both block sizes -- against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bound", [300, 4096, 9000])
def test_far_pairs_match_oracle(bound):
    from graphmambaformer_b200 import synth
    from graphmambaformer_b200.wfa import align_wfa_pairs, upload_wfa_pairs, wfa_distances
    from oracle import oracle

    rng = np.random.default_rng(bound)
    ref = synth.random_reference(60_000, rng).astype(np.int8)
    qs, ts = [], []
    for n, m in [(3999, 3999), (3999, 3200), (4000, 3999), (4001, 3000), (255, 3999), (3999, 10), (700, 650)] + [
            (int(a), int(b)) for a, b in rng.integers(500, 1300, (60, 2))]:
        s, t = rng.integers(0, 25_000), rng.integers(30_000, 55_000)
        qs.append(ref[s: s + n].copy())
        ts.append(ref[t: t + m].copy())
    ts[10][5:9] = 5
    # as many warps as there are, some of them with several pairs
    qs += [q.copy() for q in qs[7:]] * 3
    ts += [t.copy() for t in ts[7:]] * 3
    if bound == 9000:  # a side beyond the wide block's scores
        qs.append(ref[:9500].copy())
        ts.append(synth.apply_errors(ref[:9500], synth.ONT, rng).astype(np.int8))
    want = [oracle.wfa_align(q, t, bound) for q, t in zip(qs, ts)]
    dist = wfa_distances(upload_wfa_pairs(qs, ts), bound).cpu().numpy()
    r = align_wfa_pairs(qs, ts, bound)
    for b, (d, cigar) in enumerate(want):
        assert int(dist[b]) == d and int(r.distance[b]) == d, b
        if d >= 0:
            assert r.cigar(b) == cigar, b
