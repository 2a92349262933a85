"""Chaining on anchors that leave the usual shape: dense random anchors (many
equal scores, so that the tie order and the predecessors beyond the nearest
decide), blocks of 16 and 32 anchors and their remainders, windows from 1 to
beyond every ring size, lengths down to 0, free and negative penalties, and
every cut-off of the chain selection -- against the oracle, bit for bit, with
few and with many reads per call."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dense_batch(seed, span, copies=1):
    from graphmambaformer_b200.chaining import AnchorCSR

    rng = np.random.default_rng(seed)
    counts = [0, 1, 2, 3, 4, 5, 6, 15, 16, 17, 31, 32, 33, 34, 63, 64, 65, 70, 130, 300, 700] * copies
    off = np.zeros(len(counts) + 1, np.int64)
    np.cumsum(counts, out=off[1:])
    n = int(off[-1])
    q = rng.integers(0, span, n).astype(np.int32)
    t = np.where(rng.random(n) < 0.6, q + rng.integers(-6, 7, n), rng.integers(0, span, n)).astype(np.int32)
    length = np.where(rng.random(n) < 0.7, 15, rng.integers(0, 41, n)).astype(np.int32)
    return AnchorCSR(off, q, np.maximum(t, 0), length, np.where(rng.random(n) < 0.7, 1, -1).astype(np.int8))


def _check(batch, cfg):
    from graphmambaformer_b200 import chaining
    from oracle import oracle

    got = chaining.chain_anchor_batch(batch, cfg)
    want = oracle.chain_batch(batch.read_off, batch.read_pos, batch.ref_pos, batch.length, batch.strand,
                              oracle.penalty_lut(cfg.max_gap, cfg.gap_open, cfg.gap_extend, cfg.log_coeff),
                              max_lookback=cfg.max_lookback, max_gap=cfg.max_gap,
                              min_chain_anchors=cfg.min_chain_anchors, max_chains=cfg.max_chains,
                              min_chain_score=cfg.min_chain_score, secondary_overlap=cfg.secondary_overlap,
                              secondary_score_ratio=cfg.secondary_score_ratio, threads=8)
    assert np.array_equal(got.n_chains, want.n_chains)
    for r in range(len(batch)):
        for a, b in zip(got.chains(r), want.chains(batch.read_off, r)):
            assert a.score == b["score"] and a.strand == b["strand"] and a.is_primary == b["is_primary"], r
            assert [a.read_start, a.read_end, a.ref_start, a.ref_end] == [
                b["read_start"], b["read_end"], b["ref_start"], b["ref_end"]], r
            assert np.array_equal(a.anchor_idx, b["anchor_idx"]), r


@pytest.mark.parametrize("costs", [(6.0, 0.05, 0.5), (0.0, 0.0, 0.0), (-3.0, 0.1, 0.5)])
@pytest.mark.parametrize("lb", [1, 2, 3, 4, 5, 8, 33, 50, 200, 600])
def test_dense_anchors_match_oracle(lb, costs):
    from graphmambaformer_b200.config import ChainingConfig

    cfg = ChainingConfig(max_lookback=lb, max_gap=300, gap_open=costs[0], gap_extend=costs[1], log_coeff=costs[2])
    for span in (150, 2500):
        _check(_dense_batch(lb, span), cfg)


@pytest.mark.parametrize("kw", [dict(), dict(min_chain_anchors=3), dict(min_chain_score=0.0, secondary_score_ratio=0.0),
                                dict(secondary_score_ratio=1.0), dict(secondary_score_ratio=-0.5, max_chains=64),
                                dict(min_chain_score=1e9), dict(min_chain_anchors=40, secondary_score_ratio=0.3),
                                dict(secondary_overlap=0.0, max_chains=3), dict(min_chain_score=-50.0)])
def test_selection_cutoffs_match_oracle_in_a_large_batch(kw):
    from graphmambaformer_b200.config import ChainingConfig

    _check(_dense_batch(5, 900, copies=75), ChainingConfig(max_lookback=50, max_gap=300, **kw))


@pytest.mark.parametrize("top,shuffle", [(60, True), (3000, False), (200_000, True), (2**31 - 100, True),
                                         (2**31 - 100, False), (2**30 - 40, True)])
def test_sorting_any_order_strand_and_size(top, shuffle):
    """Anchors in read order per strand (as seeding writes them) and in any
    order, strands interleaved and strands that take no part, many equal
    keys, coordinates up to 31 bits, and read sizes around the sort's block
    sizes."""
    from graphmambaformer_b200.chaining import AnchorCSR
    from graphmambaformer_b200.config import ChainingConfig

    rng = np.random.default_rng(top % 1000 + shuffle)
    counts = [0, 1, 2, 31, 32, 33, 255, 256, 257, 511, 513, 4095, 4096, 4097, 8200, 16384, 700, 0, 5]
    off = np.zeros(len(counts) + 1, np.int64)
    np.cumsum(counts, out=off[1:])
    n = int(off[-1])
    t = rng.integers(0, top, n)
    q = np.minimum(np.where(rng.random(n) < 0.5, t % 20_000, rng.integers(0, 20_000, n)), top)
    length = np.full(n, 15)
    strand = rng.choice([1, -1, 0, 2], n, p=[0.5, 0.4, 0.05, 0.05]).astype(np.int8)
    if not shuffle:
        for a, b in zip(off[:-1], off[1:]):
            o = np.lexsort((q[a:b], -strand[a:b].astype(int)))
            q[a:b], t[a:b], strand[a:b] = q[a:b][o], t[a:b][o], strand[a:b][o]
    batch = AnchorCSR(off, q.astype(np.int32), t.astype(np.int32), length.astype(np.int32), strand)
    _check(batch, ChainingConfig(max_lookback=20, max_gap=2000))
