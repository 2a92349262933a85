"""Pairs whose delay line fills a power of two (the widest band of each lane
group among them), with query ends at different places of a strip in one warp,
against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

from helpers import assert_sw_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("params", [(2, 4, 4, 2, 0), (2, 4, 6, 2, 60)])
@pytest.mark.parametrize("hb", [16, 30, 62, 64, 126, 318])
def test_bands_that_fill_the_delay_line(hb, params):
    from graphmambaformer_b200 import extension as ext, synth
    from oracle import oracle

    rng = np.random.default_rng(hb)
    ref = synth.random_reference(30_000, rng).astype(np.int8)
    qs, ts = [], []
    for ql in (1, 15, 16, 17, 31, 33, 63, 65, 100, 127, 150, 190, 257, 500) * 6:
        s = int(rng.integers(1000, 25_000))
        qs.append(synth.apply_errors(ref[s: s + ql], synth.ONT, rng).astype(np.int8))
        ts.append(ref[s - 20: s + ql + 30].copy())
    ps = synth.PairSet.from_lists(qs, ts, np.full(len(qs), hb, np.int32), np.full(len(qs), 20, np.int32))
    want = oracle.sw_batch(qs, ts, ps.half_band, ps.band_offset, *params, threads=8)
    assert_sw_equal(ext.align_pairs(ps, ext.sw_params(*params)), want, label=f"{hb} {params}")
