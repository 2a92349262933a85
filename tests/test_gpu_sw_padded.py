"""Pairs that cooperating warps run with a period longer than their band asks
for: bands around the ranges' ends (the lowest only in small batches), rows
around strip and two-strip sizes, with and without x-drop, against the
oracle; and the same pairs in a batch too large for the lowest range."""

from __future__ import annotations

import numpy as np
import pytest

from helpers import assert_sw_equal

pytestmark = pytest.mark.gpu


def _pairs(repeat):
    from graphmambaformer_b200 import synth

    rng = np.random.default_rng(5)
    ref = synth.random_reference(30_000, rng).astype(np.int8)
    qs, ts, hbs, offs = [], [], [], []
    for hb in (66, 105, 106, 107, 108, 110, 127, 129, 130, 131, 138, 139, 140, 262, 263, 278, 280, 526, 527, 543, 559,
               561):
        for ql in (192, 193, 256, 257, 385, 512, 1030):
            s = int(rng.integers(1000, 25_000))
            q = synth.apply_errors(ref[s: s + ql], synth.ONT, rng).astype(np.int8)
            off, cut = ((0, 40), (30, -60), (hb, hb))[int(rng.integers(3))]
            qs.append(q)
            ts.append(ref[s - off: s + ql + cut].copy())
            hbs.append(hb)
            offs.append(off)
    return synth.PairSet.from_lists(qs * repeat, ts * repeat, np.array(hbs * repeat, np.int32),
                                    np.array(offs * repeat, np.int32))


@pytest.mark.parametrize("repeat", [1, 12])
@pytest.mark.parametrize("params", [(2, 4, 4, 2, 0), (2, 4, 6, 2, 60), (2, 1, 0, 1, 15), (1, 3, 2, 3, 0)])
def test_cooperating_warps_with_a_padded_period(params, repeat):
    from graphmambaformer_b200 import extension as ext
    from oracle import oracle

    ps = _pairs(repeat)
    want = oracle.sw_batch([ps.q(b) for b in range(len(ps))], [ps.t(b) for b in range(len(ps))], ps.half_band,
                           ps.band_offset, *params, threads=8)
    assert_sw_equal(ext.align_pairs(ps, ext.sw_params(*params)), want, label=f"{params}")
    score = ext.align_pairs(ps, ext.sw_params(*params), traceback=False)
    assert np.array_equal(score.score, want.score.astype(np.int32))
