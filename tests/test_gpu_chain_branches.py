"""Reads of one chain with a branch: anchors that leave the chain for another
diagonal and score above the cutoff by the part they share with it.  The pass
for reads with one chain follows a branch back for 64 anchors at most; longer
ones go to the general form, with the same result (the oracle's)."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_chain_near import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("branch", [10, 62, 63, 64, 65, 66, 90, 150])
@pytest.mark.parametrize("strand", [1, -1])
def test_branches_around_the_steps_followed(branch, strand):
    from graphmambaformer_b200.chaining import AnchorCSR
    from graphmambaformer_b200.config import ChainingConfig

    q, t = [np.arange(200) * 20], [np.arange(200) * 20 + 1000]
    for at, shift in ((60, 300), (90, -250)):  # two branches, from different anchors of the chain
        q.append(at * 20 + 10 + np.arange(branch) * 20)
        t.append(q[-1] + 1000 + shift)
    q, t = np.concatenate(q), np.concatenate(t)
    n = len(q)
    b = AnchorCSR(np.array([0, n, 2 * n], np.int64), np.concatenate([q, q[::-1]]).astype(np.int32),
                  np.concatenate([t, t[::-1]]).astype(np.int32), np.full(2 * n, 15, np.int32),
                  np.full(2 * n, strand, np.int8))
    for ratio in (0.6, 0.3, 0.05):
        _check(b, ChainingConfig(max_lookback=50, secondary_score_ratio=ratio))
