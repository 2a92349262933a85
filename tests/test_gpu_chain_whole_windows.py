"""Chaining of anchors whose predecessors are not the nearest ones: several
diagonals at once, stretches of them between stretches of one diagonal (so
that blocks change between the two ways of scoring a window), random anchors,
and reads around the sizes at which the sort changes -- against the oracle,
bit for bit, with few and with many reads per call."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_chain_near import _check

pytestmark = pytest.mark.gpu


def _stretch(kind, n, q0, rng):
    q = q0 + np.sort(rng.integers(0, 7 * n + 1, n))
    if kind == "one":
        return q, q + 4000
    if kind == "five":
        return q, q + 4000 + 700 * rng.integers(0, 5, n)
    if kind == "gaps":
        return q, q + 4000 + 40 * (q // 150)
    return q, rng.integers(0, 8000, n)


def _batch(copies):
    from graphmambaformer_b200.chaining import AnchorCSR

    rng = np.random.default_rng(copies)
    shapes = [[("five", 31)], [("five", 33)], [("random", 64)], [("one", 40), ("five", 100), ("one", 130)],
              [("five", 64), ("one", 200), ("random", 90), ("one", 64)], [("gaps", 223)], [("five", 224)], [("random", 225)],
              [("one", 16), ("random", 17), ("gaps", 95), ("five", 160), ("one", 33)], [("five", 700)], [("random", 1)]]
    cols, counts = [], []
    for _ in range(copies):
        for shape in shapes:
            qs, ts, at = [], [], 0
            for kind, n in shape:
                q, t = _stretch(kind, n, at, rng)
                at = int(q.max()) + 30
                qs.append(q)
                ts.append(t)
            q, t = np.concatenate(qs), np.concatenate(ts)
            if len(q) > 100:  # equal anchors and equal ends
                q[5:9], t[5:9] = q[5], t[5]
            order = rng.permutation(len(q)) if rng.random() < 0.5 else np.arange(len(q))
            cols.append((q[order], t[order], np.where(rng.random(len(q)) < 0.8, 15, rng.integers(1, 30, len(q))),
                         np.where(rng.random(len(q)) < 0.75, 1, -1)))
            counts.append(len(q))
    off = np.zeros(len(counts) + 1, np.int64)
    np.cumsum(counts, out=off[1:])
    cat = lambda k, dt: np.concatenate([c[k] for c in cols]).astype(dt)  # noqa: E731
    return AnchorCSR(off, cat(0, np.int32), cat(1, np.int32), cat(2, np.int32), cat(3, np.int8))


@pytest.mark.parametrize("copies", [1, 120])
@pytest.mark.parametrize("lb,max_gap", [(1, 5000), (5, 300), (31, 5000), (64, 5000), (65, 16384), (500, 5000), (1000, 16384)])
def test_windows_of_several_diagonals(copies, lb, max_gap):
    from graphmambaformer_b200.config import ChainingConfig

    _check(_batch(copies), ChainingConfig(max_lookback=lb, max_gap=max_gap, min_chain_score=0.0))


def test_a_single_small_read():
    from graphmambaformer_b200.chaining import AnchorCSR
    from graphmambaformer_b200.config import ChainingConfig

    for n in (0, 1, 2, 31, 32, 33, 96, 223, 224, 225, 300):
        rng = np.random.default_rng(n)
        q = rng.integers(0, 5 * n + 1, n).astype(np.int32)
        b = AnchorCSR(np.array([0, n], np.int64), q, (q + 300 * rng.integers(0, 3, n)).astype(np.int32),
                      np.full(n, 15, np.int32), np.where(rng.random(n) < 0.5, 1, -1).astype(np.int8))
        _check(b, ChainingConfig())
