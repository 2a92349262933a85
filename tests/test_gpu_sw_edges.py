"""Band and target edges of the 16x2 SW kernels: half bands around the sizes
where the pipeline's period, the band mask table and the cooperative classes
change, rows and targets around the strip and chunk sizes, bands that lie
left of, right of or across the target's ends, codes that match nothing, and
free gaps and mismatches -- in every lane-group class."""

from __future__ import annotations

import numpy as np
import pytest

from helpers import assert_sw_equal

pytestmark = pytest.mark.gpu

# (l8_max_w, l16_max_w): the default split, everything with 32 lanes, wide bands in 16- and 8-lane groups
SPLITS = [(61, 125), (0, 0), (0, 8193), (8193, 8193)]
SCORINGS = [(2, 4, 4, 2, 0), (2, 4, 6, 2, 60), (3, 0, 0, 0, 0), (2, 1, 0, 1, 15), (1, 3, 2, 3, 9)]


def _edge_pairs():
    from graphmambaformer_b200 import synth

    rng = np.random.default_rng(77)
    ref = synth.random_reference(20_000, rng).astype(np.int8)
    qs, ts, hbs, offs = [], [], [], []
    for hb in (0, 1, 2, 3, 13, 14, 15, 29, 30, 31, 32, 61, 62, 63, 64, 65, 127, 129, 130, 131, 132, 133, 300):
        for ql, cut, off in ((1, 0, 0), (33, 5, 3), (64, -20, hb), (65, 0, hb + 40), (129, 30, -25), (230, -90, 7)):
            s = int(rng.integers(1000, 15_000))
            q = synth.apply_errors(ref[s: s + ql], synth.ONT, rng).astype(np.int8)
            t = ref[s - off if off > 0 else s: s + ql + cut].copy()
            if len(t) and ql > 64:  # codes that match nothing, and a code outside the alphabet that does
                t[rng.integers(0, len(t), 3)] = (5, -1, 0)
                q[rng.integers(0, len(q), 3)] = (5, -1, 0)
            qs.append(q)
            ts.append(t)
            hbs.append(hb)
            offs.append(off)
    return synth.PairSet.from_lists(qs, ts, np.array(hbs, np.int32), np.array(offs, np.int32))


@pytest.mark.parametrize("params", SCORINGS)
def test_band_and_target_edges_in_every_class(params):
    import ctypes

    from graphmambaformer_b200 import _native, extension as ext
    from oracle import oracle

    ps = _edge_pairs()
    want = oracle.sw_batch([ps.q(b) for b in range(len(ps))], [ps.t(b) for b in range(len(ps))], ps.half_band,
                           ps.band_offset, *params, threads=8)
    lib = _native.lib()
    before = _native.GmfSwTuning()
    assert lib.gmf_sw_get_tuning(ctypes.byref(before)) == _native.GMF_OK
    try:
        for l8, l16 in SPLITS:
            t = _native.GmfSwTuning()
            assert lib.gmf_sw_get_tuning(ctypes.byref(t)) == _native.GMF_OK
            t.l8_max_w, t.l16_max_w = l8, l16
            assert lib.gmf_sw_set_tuning(ctypes.byref(t)) == _native.GMF_OK
            assert_sw_equal(ext.align_pairs(ps, ext.sw_params(*params)), want, label=f"{params} {l8} {l16}")
            score = ext.align_pairs(ps, ext.sw_params(*params), traceback=False)
            assert np.array_equal(score.score, want.score.astype(np.int32)), (params, l8, l16)
            assert np.array_equal(score.target_end, want.target_end), (params, l8, l16)
    finally:
        assert lib.gmf_sw_set_tuning(ctypes.byref(before)) == _native.GMF_OK


@pytest.mark.parametrize("form", ["batched", "plain"])
def test_walk_through_gaps_of_every_size(form):
    """The walk copies the traceback words around its path in blocks of 32
    rows and 32 slots and looks at 8 cells of a gap at a time: gaps around
    those sizes, two gaps within one block, alignments that start and end at
    block boundaries, and a score that falls near 0 on the way."""
    from graphmambaformer_b200 import extension as ext, synth
    from oracle import oracle

    rng = np.random.default_rng(78)
    ref = synth.random_reference(20_000, rng).astype(np.int8)
    qs, ts, hbs = [], [], []
    for gap in (1, 2, 7, 8, 9, 15, 16, 17, 18, 31, 32, 33, 40, 63, 64, 120):
        for left in (30, 32, 33, 64, 95, 200):
            for kind in range(3):
                s = int(rng.integers(500, 15_000))
                a, b, c = ref[s: s + left + 60], ref[s + left + 60: s + left + 60 + gap], ref[s + left + 60 + gap:
                                                                                         s + 2 * left + 150 + gap]
                whole, cut = np.concatenate([a, b, c]), np.concatenate([a, c])
                if kind == 2:  # the gap back again some bases later
                    m = len(a) + 20
                    cut = np.concatenate([cut[:m], ref[:gap], cut[m:]])
                qs.append(cut if kind else whole)
                ts.append(whole if kind else cut)
                hbs.append(150 if left % 2 else 40)
    ps = synth.PairSet.from_lists(qs, ts, np.array(hbs, np.int32), np.zeros(len(qs), np.int32))
    for params in ((2, 4, 4, 1, 0), (5, 4, 3, 1, 200)):
        want = oracle.sw_batch(qs, ts, ps.half_band, ps.band_offset, *params, threads=8)
        assert_sw_equal(ext.align_pairs(ps, ext.sw_params(*params), form=form), want, label=str(params))
