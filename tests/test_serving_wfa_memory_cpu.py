"""A batch's memory estimate covers what the wavefront mode takes, and changes
nothing else: not the banded mode, not which requests are taken."""

from __future__ import annotations

import numpy as np
import pytest

from graphmambaformer_b200.config import ChainingConfig, ExtensionConfig
from graphmambaformer_b200.serving import estimate_bytes


@pytest.mark.parametrize("lens", [[150] * 512, [20_000] * 64, [100_000] * 10, [1_000], [150, 40_000]])
@pytest.mark.parametrize("half_band", [16, 512])
@pytest.mark.parametrize("bound", [100, 4096, 60_000])
def test_estimate_covers_the_wavefronts(lens, half_band, bound):
    from graphmambaformer_b200 import _native, wfa

    lens = np.array(lens, np.int64)
    sw = estimate_bytes(lens, 100, ExtensionConfig(max_half_band=half_band), 8)
    got = estimate_bytes(lens, 100, ExtensionConfig(max_half_band=half_band, algorithm="wfa", wfa_max_distance=bound), 8)
    # two chains a read, as the banded estimate counts them
    q = np.repeat(lens, 2)
    md = min(bound, int(q.max()))
    entries = min(wfa.HISTORY_BUDGET, wfa.direct_entries(q, q, md))
    need = _native.lib().gmf_wfa_workspace_bytes(len(q), int(q.max()), md, entries)
    assert got >= max(sw, need)
    assert got <= max(sw, 1.1 * need + (64 << 20))
    W = 2 * half_band + 1
    assert sw == 120 * 100 + int(np.sum((lens + 200) * W)) * 2 // 2 + 64 * len(lens) + (1 << 20)


def test_a_request_above_the_budget_by_its_wavefronts_alone_is_taken():
    from test_serving_cpu import _anchors, _server, _Worker

    cfg = ExtensionConfig(max_half_band=16, algorithm="wfa")
    lens = np.array([20_000])
    most = ChainingConfig().max_chains
    banded, full = (estimate_bytes(lens, 3, cfg, most, wavefronts=x) for x in (False, True))
    assert banded < full
    s = _server([_Worker([])], budget=banded, max_reads=4)
    s.ecfg = cfg
    s.start()
    futs = [s.submit([np.zeros(20_000, np.int8)], _anchors([20_000])) for _ in range(3)]
    assert all(f.result(timeout=30) == [20_000] for f in futs)
    with pytest.raises(ValueError, match="budget"):
        s.submit([np.zeros(60_000, np.int8)], _anchors([60_000]))
    s.stop()
    assert s.in_flight_bytes == 0
