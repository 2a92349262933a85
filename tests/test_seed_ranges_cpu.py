"""A large batch is seeded in ranges of reads, each in a bounded workspace."""

from __future__ import annotations

import numpy as np
import pytest


@pytest.mark.parametrize("lens", [[150] * 5000, [0] * 300 + [20_000] * 40, [1_000_000, 3, 2_000_000, 0, 0, 700], [], [5]])
@pytest.mark.parametrize("budget", [1 << 16, 1 << 22, 1 << 30])
def test_ranges_cover_the_reads_within_the_budget(lens, budget):
    from graphmambaformer_b200 import _native
    from graphmambaformer_b200.seeding import workspace_ranges

    off = np.zeros(len(lens) + 1, np.int64)
    np.cumsum(lens, out=off[1:])
    f = _native.lib().gmf_seed_workspace_bytes
    got = workspace_ranges(off + 77, budget)
    assert got[0][0] == 0 and got[-1][1] == len(lens)
    assert all(a[1] == b[0] for a, b in zip(got, got[1:]))
    for r0, r1 in got:
        assert f(r1 - r0, int(off[r1] - off[r0])) <= budget or r1 == r0 + 1
        if r1 < len(lens):  # as many as fit
            assert f(r1 + 1 - r0, int(off[r1 + 1] - off[r0])) > budget


def test_workspace_of_a_batch_within_the_budget_is_one_range():
    from graphmambaformer_b200.seeding import SEED_WORKSPACE, workspace_ranges

    assert workspace_ranges(np.arange(1025, dtype=np.int64) * 2000, SEED_WORKSPACE) == [(0, 1024)]
    assert len(workspace_ranges(np.arange(1_000_001, dtype=np.int64) * 150, SEED_WORKSPACE)) > 4
