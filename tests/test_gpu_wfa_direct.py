"""One-pass wavefront alignment (gmf_wfa_align_direct): distances around the
history's 32-wavefront chunks and the walk's 24-step windows, whole-block and
one-warp pairs, codes that match nothing, runs of one operation across
windows, pairs whose history does not fit, and bounds beyond a wide block's
shared memory -- against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _edit(a, n, kind, rng):
    """n separated edits of one kind (0 substitutions, 1 insertions, 2 deletions, 3 one long insertion, 4 one long
    deletion), so that the distance is about n."""
    if kind == 3:
        at = len(a) // 2
        return np.concatenate([a[:at], rng.integers(1, 5, n).astype(np.int8), a[at:]])
    if kind == 4:
        at = len(a) // 3
        return np.concatenate([a[:at], a[at + n:]])
    at = np.sort(rng.choice(len(a), n, replace=False))
    if kind == 0:
        b = a.copy()
        b[at] = b[at] % 4 + 1
        return b
    return np.insert(a, at, rng.integers(1, 5, n).astype(np.int8)) if kind == 1 else np.delete(a, at)


def _pairs():
    from graphmambaformer_b200 import synth

    rng = np.random.default_rng(91)
    qs, ts = [], []
    for d in (0, 1, 2, 23, 24, 25, 31, 32, 33, 47, 48, 49, 63, 64, 65, 96, 97, 130, 255, 260):
        for kind in range(5):
            for L in (700, 4300):
                a = synth.random_reference(L, rng).astype(np.int8)
                b = _edit(a, d, kind, rng)
                if d % 3 == 1:
                    a[rng.integers(0, L, 2)] = (5, -1)
                    b[rng.integers(0, len(b), 2)] = (5, 0)
                qs.append(a if kind % 2 else b)
                ts.append(b if kind % 2 else a)
    for n, m in ((0, 0), (0, 3), (5, 0), (1, 1), (1, 9), (40, 2)):
        qs.append(synth.random_reference(n, rng).astype(np.int8))
        ts.append(synth.random_reference(m, rng).astype(np.int8))
    return qs, ts


@pytest.mark.parametrize("budget", [1 << 29, 100_000, 2_000])
def test_direct_alignment_matches_oracle(budget):
    from graphmambaformer_b200.wfa import align_wfa_pairs
    from oracle import oracle

    qs, ts = _pairs()
    r = align_wfa_pairs(qs, ts, 4096, history_budget=budget)
    for b in range(len(qs)):
        d, cigar = oracle.wfa_align(qs[b], ts[b], 4096)
        assert int(r.distance[b]) == d and r.cigar(b) == cigar, (budget, b)
        c = r.op_counts[b]
        assert [int(x) for x in c] == [sum(n for op, n in cigar if op == o) for o in "=XID"], b


def test_bounds_beyond_a_wide_block():
    from graphmambaformer_b200 import synth
    from graphmambaformer_b200.wfa import align_wfa_pairs
    from oracle import oracle

    rng = np.random.default_rng(92)
    a = synth.random_reference(9000, rng).astype(np.int8)
    qs = [a, a[:300], a[:2000], a[:5000]]
    ts = [synth.apply_errors(a, synth.ONT, rng).astype(np.int8), synth.random_reference(280, rng).astype(np.int8),
          synth.random_reference(1500, rng).astype(np.int8), _edit(a[:5000], 900, 0, rng)]
    r = align_wfa_pairs(qs, ts, 20_000)
    for b in range(len(qs)):
        d, cigar = oracle.wfa_align(qs[b], ts[b], 20_000)
        assert int(r.distance[b]) == d and r.cigar(b) == cigar, b
