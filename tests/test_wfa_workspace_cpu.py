"""Sizes of the WFA workspace: wavefronts beyond shared memory are kept for
the pairs that can be computed at once, not for every warp of every block at
the call's longest side."""

from __future__ import annotations

import pytest


@pytest.mark.parametrize("n,bound,mb", [(1, 4096, 0.2), (8, 4096, 0.6), (64, 4096, 4.3), (148, 4096, 10.1),
                                        (1000, 4096, 66), (10_000, 4096, 156), (64, 8205, 8.5), (10_000, 8205, 312),
                                        (1000, 20_000, 321), (10_000, 20_000, 758)])
def test_fixed_part_of_the_workspace(n, bound, mb):
    """At most what one 32-bit slot of the bound per pair (per warp of a
    256-thread block, two blocks an SM, for large batches) takes."""
    from graphmambaformer_b200 import _native

    f = _native.lib().gmf_wfa_workspace_bytes
    assert f(n, 20_000, bound, 0) <= mb * 1e6
    assert f(n, 20_000, bound, 1000) >= f(n, 20_000, bound, 0) + 4000


def test_short_pairs_and_small_bounds_need_no_slots():
    from graphmambaformer_b200 import _native

    f = _native.lib().gmf_wfa_workspace_bytes
    assert f(10_000, 20_000, 254, 0) <= 256 + 256 + 8 * 10_000
    assert f(10_000, 254, 4096, 0) <= 256 + 256 + 8 * 10_000
    assert f(10_000, 300, 4096, 0) <= 256 + 256 + 8 * 10_000 + 10_000 * 4 * (2 * 300 + 5)
