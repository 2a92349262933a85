"""Overlap limits at and below 0.  The selection drops a chain whose overlap
with the primary one is above the limit, and the first chain's overlap is 0:
a limit below 0 therefore keeps no chain, of reads with one chain too."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [0.0, -0.0, -1e-9, -1.0, float("nan")])
def test_overlap_limit_of_zero_and_below(limit):
    from graphmambaformer_b200 import chaining, synth
    from graphmambaformer_b200.config import ChainingConfig
    from oracle import oracle

    cb = synth.chaining_reads_hifi(n_reads=8, seed=5, ref_len=2_000_000, mean_len=4000)
    cfg = ChainingConfig(max_lookback=50, secondary_overlap=limit)
    got = chaining.chain_anchor_batch(cb, cfg)
    want = oracle.chain_batch(cb.read_off, cb.read_pos, cb.ref_pos, cb.length, cb.strand,
                              oracle.penalty_lut(cfg.max_gap, cfg.gap_open, cfg.gap_extend, cfg.log_coeff),
                              max_lookback=50, max_gap=cfg.max_gap, min_chain_anchors=cfg.min_chain_anchors,
                              max_chains=cfg.max_chains, min_chain_score=cfg.min_chain_score,
                              secondary_overlap=limit, secondary_score_ratio=cfg.secondary_score_ratio, threads=4)
    assert np.array_equal(got.n_chains, want.n_chains)
    assert np.all(got.n_chains == 0) if limit < 0 else np.all(got.n_chains > 0)
