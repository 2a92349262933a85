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
