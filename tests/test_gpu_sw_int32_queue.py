"""The int32 class with fewer pairs than warps, about as many, and more, alone
in its call and beside 16x2 pairs, for every number of warps a block, against
the oracle."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from helpers import assert_sw_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 147, 149, 593, 2400])
@pytest.mark.parametrize("params", [(2000, 3000, 3001, 1999, 0), (2000, 3000, 3001, 1999, 40_000)])
def test_int32_pairs_against_oracle(n, params):
    from graphmambaformer_b200 import _native, extension as ext, synth
    from oracle import oracle

    rng = np.random.default_rng(n)
    ref = synth.random_reference(30_000, rng).astype(np.int8)
    qs, ts = [], []
    for b in range(n):
        ql = int(rng.integers(1, 12) if b % 5 == 1 else rng.integers(20, 160))  # the shortest stay in 16 bits
        s = int(rng.integers(1000, 25_000))
        qs.append(synth.apply_errors(ref[s: s + ql], synth.ONT, rng).astype(np.int8))
        ts.append(ref[s - 10: s + ql + 12].copy())
    hb = rng.integers(3, 40, n).astype(np.int32)
    ps = synth.PairSet.from_lists(qs, ts, hb, np.full(n, 10, np.int32))
    want = oracle.sw_batch(qs, ts, ps.half_band, ps.band_offset, *params, threads=8)
    lib, before = _native.lib(), _native.GmfSwTuning()
    assert lib.gmf_sw_get_tuning(ctypes.byref(before)) == _native.GMF_OK
    try:
        for wpb in (4, 3, 1):
            t = _native.GmfSwTuning()
            assert lib.gmf_sw_get_tuning(ctypes.byref(t)) == _native.GMF_OK
            t.warps_per_block = wpb
            assert lib.gmf_sw_set_tuning(ctypes.byref(t)) == _native.GMF_OK
            assert_sw_equal(ext.align_pairs(ps, ext.sw_params(*params)), want, label=f"{n} {wpb}")
    finally:
        assert lib.gmf_sw_set_tuning(ctypes.byref(before)) == _native.GMF_OK
