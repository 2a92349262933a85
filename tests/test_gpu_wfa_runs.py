"""Runs of matches around the sizes at which the extension of a diagonal goes
from 4 to 8 codes a step and to a whole warp: single pairs, and many at
once, against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_long", [0, 3])
def test_runs_of_every_length(n_long):
    from graphmambaformer_b200 import synth, wfa
    from oracle import oracle

    rng = np.random.default_rng(9)
    ref = synth.random_reference(60_000, rng).astype(np.int8)
    qs, ts = [], []
    for run in (0, 1, 3, 4, 5, 11, 12, 13, 19, 20, 21, 27, 28, 29, 30, 127, 128, 129, 147, 148, 149, 255, 256, 300):
        for start in range(4):  # every alignment of both sequences
            a = ref[100 + start: 100 + start + run].copy()
            mis = np.array([int(ref[100 + start + run]) % 4 + 1], np.int8)
            tail = ref[5_000: 5_000 + start + run].copy()
            qs += [a, np.concatenate([a, mis, tail]), np.concatenate([a, tail]), np.concatenate([a, [5], tail])]
            ts += [a.copy(), np.concatenate([a, ref[100 + start + run: 101 + start + run], tail]),
                   np.concatenate([a, mis, tail]), np.concatenate([a, [5], tail])]
    for x in range(n_long):  # a block's work: long runs, and an N that ends one
        t = ref[7_000 * x: 7_000 * x + 6_000].copy()
        q = synth.apply_errors(t, synth.HIFI, rng).astype(np.int8)
        q[3_000] = t[3_000] = 5
        qs.append(q)
        ts.append(t)
    qs, ts = [np.asarray(x, np.int8) for x in qs], [np.asarray(x, np.int8) for x in ts]
    got = wfa.align_wfa_pairs(qs, ts, 4096)
    for b in range(len(qs)):
        want = oracle.wfa_align(qs[b], ts[b], 4096)
        assert int(got.distance[b]) == want[0], b
        assert got.cigar(b) == want[1], b
