"""A pair whose band is wider than the call's stated widest one."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widest", [10, 30, 62, 100])
def test_a_band_beyond_the_stated_widest_is_reported(widest):
    """The classes that the widest band rules out are not launched: a pair
    that breaks its word is reported all the same, and harms no other pair."""
    from graphmambaformer_b200 import extension as ext, synth
    from graphmambaformer_b200._native import GMF_SWF_WORKSPACE

    rng = np.random.default_rng(4)
    ref = synth.random_reference(5_000, rng).astype(np.int8)
    qs = [ref[100 * i: 100 * i + 60 + 30 * i].copy() for i in range(12)]
    ps = synth.PairSet.from_lists(qs, [ref[100 * i: 100 * i + 80 + 30 * i].copy() for i in range(12)],
                                  np.full(12, widest, np.int32), np.zeros(12, np.int32))
    p = ext.sw_params(2, 4, 4, 2, 0)
    good = ext.launch_banded_sw(ext.upload_pairs(ps), p)
    dp = ext.upload_pairs(ps)
    dp.half_band[3] = 500
    bad = ext.launch_banded_sw(dp, p)
    assert int(good.error_flags[0]) == 0 and int(bad.error_flags[0]) & GMF_SWF_WORKSPACE
    a, b = good.score.cpu().numpy(), bad.score.cpu().numpy()
    assert b[3] == 0 and np.all(np.delete(a, 3) > 0) and np.array_equal(np.delete(a, 3), np.delete(b, 3))
