"""One-warp pairs with very wide bands, where fewer warps than asked for make a
block: short pairs around the half bands at which the number changes, against
the oracle, for every number of warps asked for."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from helpers import assert_sw_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("params", [(2, 4, 4, 2, 0), (2, 4, 6, 2, 60)])
@pytest.mark.parametrize("hb", [1087, 2043, 2080, 2111, 4096])
def test_wide_bands_with_fewer_warps_a_block(hb, params):
    from graphmambaformer_b200 import _native, extension as ext, synth
    from oracle import oracle

    rng = np.random.default_rng(hb)
    ref = synth.random_reference(30_000, rng).astype(np.int8)
    qs, ts = [], []
    for ql in [int(x) for x in rng.integers(1, 200, 1500)] + [700, 900]:  # more pairs than one warp of every block
        s = int(rng.integers(5000, 20_000))
        qs.append(synth.apply_errors(ref[s: s + ql], synth.ONT, rng).astype(np.int8))
        ts.append(ref[s - 20: s + ql + 30].copy())
    ps = synth.PairSet.from_lists(qs, ts, np.full(len(qs), hb, np.int32), np.full(len(qs), 20, np.int32))
    want = oracle.sw_batch(qs, ts, ps.half_band, ps.band_offset, *params, threads=8)
    lib, before = _native.lib(), _native.GmfSwTuning()
    assert lib.gmf_sw_get_tuning(ctypes.byref(before)) == _native.GMF_OK
    try:
        for wpb in (4, 3, 1):
            t = _native.GmfSwTuning()
            assert lib.gmf_sw_get_tuning(ctypes.byref(t)) == _native.GMF_OK
            t.warps_per_block = wpb
            assert lib.gmf_sw_set_tuning(ctypes.byref(t)) == _native.GMF_OK
            assert_sw_equal(ext.align_pairs(ps, ext.sw_params(*params)), want, label=f"{hb} {wpb}")
    finally:
        assert lib.gmf_sw_set_tuning(ctypes.byref(before)) == _native.GMF_OK
