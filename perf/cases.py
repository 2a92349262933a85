"""The work a user of this library has it do, as cases that can be timed.

A case is one call of the alignment path on data the caller already holds:
banded Smith-Waterman of read/target pairs, chaining of a batch's anchors,
minimizer seeding of reads, wavefront alignment, the whole batch pipeline of
the serving loop, and SAM text of finished records.  ``listed()`` holds the
sizes the benchmark, the tests and the stage defaults use, from one read up;
``draw()`` gives others of the same ranges.  Inputs are simulated from the
seed alone (uniform reference, the error profiles of ``synth``).
"""

from __future__ import annotations

import math

import numpy as np
import torch

from graphmambaformer_b200 import chaining, extension, records, seeding, serving, synth, wfa
from graphmambaformer_b200.config import ChainingConfig, ExtensionConfig

FLANK = 32
PROFILES = {"short": synth.SHORT_READ, "illumina": synth.ILLUMINA, "hifi": synth.HIFI, "ont": synth.ONT}
MIX = ("illumina", "hifi", "ont")


# --------------------------------------------------------------------------- #
# Cases
# --------------------------------------------------------------------------- #
def _pairs(name, n, lo, hi, err, band, slope, cap, scoring, x_drop, cigar=True):
    c = dict(kind="pairs", n=n, lo=lo, hi=hi, err=err, band=band, slope=slope, cap=cap, x_drop=x_drop, cigar=cigar)
    c["match"], c["mismatch"], c["open"], c["extend"] = scoring
    return dict(c, name=name) if name else c


def listed() -> list:
    plain, stage = (2, 4, 4, 2), (2, 4, 6, 2)  # the benchmark's scoring, the extension stage's default
    return [
        # a small request's extension step with the stage defaults: launches and latency
        _pairs("pairs_few", 64, 150, 2000, "mix", 64, 0.0, 64, stage, 600),
        # a batch of Illumina reads at their windows, every read as long as the next
        _pairs("pairs_150bp", 10_000, 150, 150, "short", 32, 0.0, 32, plain, 0),
        # the uneven batch: 150 bp to 20 kb of all three technologies, bands growing with the length
        _pairs("pairs_mixed", 20_000, 150, 20_000, "mix", 32, 0.02, 500, plain, 0),
        # gaps of long reads: 8 kb segments with very wide bands
        _pairs("pairs_wide", 400, 7_500, 8_500, "ont", 1_500, 0.05, 2_000, plain, 0),
        # one read of the interactive or single-read call, stage defaults
        dict(name="chain_read", kind="chain", reads=1, lo=15_000, hi=15_000, err="hifi", lookback=64),
        # a batch of HiFi reads, predecessor window 50
        dict(name="chain_hifi", kind="chain", reads=5_000, lo=12_000, hi=18_000, err="hifi", lookback=50),
        # ultra-long ONT reads, about 10k anchors each, predecessor window 200
        dict(name="chain_long", kind="chain", reads=1_000, lo=50_000, hi=100_000, err="ont", lookback=200),
        # seeding of a serving batch against the resident index
        dict(name="seed_reads", kind="seed", reads=1_024, lo=150, hi=20_000, err="mix"),
        # end-to-end (global) alignment of mixed reads by wavefronts, CIGARs included
        dict(name="wfa_mixed", kind="wfa", n=4_000, lo=150, hi=20_000, err="mix"),
        # whole calls of the serving loop's worker: one small request, and a full batch
        dict(name="serve_request", kind="serve", reads=8, lo=150, hi=2_000, err="mix"),
        dict(name="serve_batch", kind="serve", reads=1_024, lo=150, hi=20_000, err="mix"),
        # SAM text of a finished batch, host columns in and text out
        dict(name="sam_text", kind="sam", records=5_000, lo=150, hi=20_000),
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(("pairs", "pairs", "pairs", "chain", "chain", "seed", "wfa", "serve", "sam"))
    if kind == "pairs":
        lo = _log(rng, 100, 8_000)
        hi = min(20_000, int(lo * rng.uniform(1.0, 6.0)))
        band, slope = _log(rng, 16, 1_500), rng.choice((0.0, 0.02))
        cap = min(2_000, max(band, int(band + slope * hi)))
        cells = 0.5 * (lo + hi) * (2 * (band + 0.5 * slope * (lo + hi)) + 1)
        n = _log(rng, 16, max(17, min(20_000, 1.0e10 / cells)))
        scoring, x_drop = rng.choice((((2, 4, 4, 2), 0), ((2, 4, 6, 2), 600), ((1, 4, 6, 1), 100)))
        return _pairs(None, n, lo, hi, rng.choice(("mix", "short", "hifi", "ont")), band, slope, cap, scoring, x_drop,
                      rng.random() < 0.8)
    if kind == "chain":
        lo = _log(rng, 2_000, 60_000)
        hi = int(lo * rng.uniform(1.0, 1.6))
        reads = _log(rng, 1, max(2, min(5_000, 40_000_000 // hi)))
        return dict(kind="chain", reads=reads, lo=lo, hi=hi, err=rng.choice(("hifi", "ont", "mix")),
                    lookback=rng.choice((32, 50, 64, 100, 200)))
    lo = _log(rng, 100, 2_000)
    hi = min(20_000, int(lo * rng.uniform(1.0, 20.0)))
    if kind == "sam":
        return dict(kind="sam", records=_log(rng, 16, min(5_000, 12_000_000 // hi)), lo=lo, hi=hi)
    if kind == "wfa":
        return dict(kind="wfa", n=_log(rng, 16, min(4_000, 9_000_000 // hi)), lo=lo, hi=hi,
                    err=rng.choice(("mix", "hifi", "ont")))
    return dict(kind=kind, reads=_log(rng, 4, min(1_024, 3_000_000 // hi)), lo=lo, hi=hi,
                err=rng.choice(("mix", "hifi", "ont")))


# --------------------------------------------------------------------------- #
# Inputs, simulated on the GPU
# --------------------------------------------------------------------------- #
def _lengths(n: int, lo: int, hi: int) -> np.ndarray:
    """Log-normal read lengths (median about 1.1 kb) where the range is wide,
    else uniform ones; the same lengths for every seed, so that a case is the
    same amount of work and its results have the same sizes."""
    rng = np.random.default_rng([n, lo, hi])
    if hi >= 8 * lo:
        return np.clip(rng.lognormal(7.0, 1.2, size=n), lo, hi).astype(np.int64)
    return rng.integers(lo, hi + 1, size=n)


class _Sim:
    """Reads of a seeded uniform reference: per read its template (start, length), strand and error profile."""

    def __init__(self, seed: int, n: int, lo: int, hi: int, err: str, ref_len: int, margin: int = 0, both=False):
        rng = np.random.default_rng(seed)
        dev = torch.device("cuda")
        g = torch.Generator(dev).manual_seed(int(rng.integers(1 << 62)))
        self.ref = torch.randint(1, 5, (ref_len,), generator=g, device=dev, dtype=torch.int8)
        self.lens = _lengths(n, lo, hi)
        self.starts = rng.integers(margin, ref_len - int(self.lens.max()) - margin, size=n)
        self.strand = np.where(rng.random(n) < 0.5, 1, -1) if both else np.ones(n, np.int64)
        prof = rng.integers(0, 3, size=n) if err == "mix" else np.zeros(n, np.int64)
        table = torch.tensor([[PROFILES[e].p_del, PROFILES[e].p_sub, PROFILES[e].p_ins]
                              for e in (MIX if err == "mix" else (err,))], device=dev)
        up = lambda a: torch.from_numpy(np.asarray(a, np.int64)).to(dev)  # noqa: E731
        lens, starts, strand = up(self.lens), up(self.starts), up(self.strand)
        row = torch.repeat_interleave(lens)
        col = torch.arange(row.numel(), device=dev) - (torch.cumsum(lens, 0) - lens)[row]
        rev = strand[row] < 0
        base = self.ref[starts[row] + torch.where(rev, lens[row] - 1 - col, col)]
        base = torch.where(rev, 5 - base, base)
        p = table[up(prof)[row]]
        u = torch.rand(row.numel(), generator=g, device=dev)
        shift = torch.randint(1, 4, (row.numel(),), generator=g, device=dev, dtype=torch.int8)
        extra = torch.randint(1, 5, (row.numel(),), generator=g, device=dev, dtype=torch.int8)
        gone = u < p[:, 0]
        base = torch.where(~gone & (u < p[:, 0] + p[:, 1]), (base - 1 + shift) % 4 + 1, base)
        ins = torch.rand(row.numel(), generator=g, device=dev) < p[:, 2]
        keep = torch.stack([ins, ~gone], 1).reshape(-1)  # an inserted base, then the template's
        self.codes = torch.stack([extra, base], 1).reshape(-1)[keep].contiguous()
        n_out = torch.zeros(n, dtype=torch.int64, device=dev)
        n_out.index_add_(0, row, ins.long() + (~gone).long())
        self.off = np.zeros(n + 1, np.int64)
        np.cumsum(n_out.cpu().numpy(), out=self.off[1:])

    def targets(self, flank: int) -> tuple:
        """Every read's template with ``flank`` bases to each side, as CSR codes on the host."""
        dev = self.ref.device
        lens = self.lens + 2 * flank
        off = np.zeros(len(lens) + 1, np.int64)
        np.cumsum(lens, out=off[1:])
        ld = torch.from_numpy(lens).to(dev)
        row = torch.repeat_interleave(ld)
        col = torch.arange(row.numel(), device=dev) - (torch.cumsum(ld, 0) - ld)[row]
        return self.ref[torch.from_numpy(self.starts - flank).to(dev)[row] + col].cpu().numpy(), off


def _ref_len(hi: int) -> int:
    return max(1_000_000, 12 * hi)


def _room(lens: np.ndarray) -> int:
    """Entries that hold any of a case's variable-size results (CIGAR words, anchors, text beside the bases)."""
    return int(0.5 * lens.sum()) + 512 * len(lens)


def _chain_config(case) -> ChainingConfig:
    return ChainingConfig(max_lookback=int(case["lookback"]))


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "pairs":
        sim = _Sim(seed, case["n"], case["lo"], case["hi"], case["err"], _ref_len(case["hi"]), margin=FLANK + 1)
        t, toff = sim.targets(FLANK)
        hb = np.clip(case["band"] + case["slope"] * sim.lens, case["band"], case["cap"]).astype(np.int32)
        ps = synth.PairSet(sim.codes.cpu().numpy(), sim.off, t, toff, hb, np.full(case["n"], FLANK, np.int32))
        dp = extension.upload_pairs(ps)
        return dict(kind=kind, dp=dp, cigar=case["cigar"], room=_room(sim.lens), out=extension.SWOutputs.allocate(dp, case["cigar"]),
                    params=extension.sw_params(case["match"], case["mismatch"], case["open"], case["extend"],
                                               case["x_drop"]))
    if kind == "wfa":
        sim = _Sim(seed, case["n"], case["lo"], case["hi"], case["err"], _ref_len(case["hi"]))
        t, toff = sim.targets(0)
        batch = wfa.WfaBatch(sim.codes.cpu().numpy(), sim.off, t, toff)
        return dict(kind=kind, dp=wfa.upload_wfa_batch(batch), room=_room(sim.lens))
    if kind == "sam":
        batch = _sam_columns(case, seed)
        return dict(kind=kind, batch=batch, room=2 * int(batch.seq_off[-1]) + _room(np.diff(batch.seq_off)))
    sim = _Sim(seed, case["reads"], case["lo"], case["hi"], case["err"], _ref_len(case["hi"]), both=True)
    n = case["reads"]
    index = seeding.DeviceMinimizerIndex(sim.ref.cpu().numpy(), k=15, w=10)
    if kind == "serve":
        al = serving.BatchAligner(sim.ref, sim.ref.device, ChainingConfig(), ExtensionConfig(), index=index)
        codes = sim.codes.cpu().numpy()
        torch.cuda.synchronize()
        return dict(kind=kind, aligner=al, reads=[codes[sim.off[r]: sim.off[r + 1]].copy() for r in range(n)],
                    room=_room(sim.lens))
    off_d = torch.from_numpy(sim.off).to(sim.ref.device)
    if kind == "seed":
        return dict(kind=kind, index=index, codes=sim.codes, off=off_d, n=n, room=_room(sim.lens))
    a = index.seed_device(sim.codes, off_d, n)  # the anchors, as the seed stage hands them over
    da = chaining.DeviceAnchors(n, a["n_anchors"], a["read_off"], a["read_pos"], a["ref_pos"], a["length"],
                                a["strand"], sim.ref.device)
    cfg = _chain_config(case)
    return dict(kind=kind, da=da, cfg=cfg, out=chaining.ChainOutputs.allocate(da, cfg.max_chains),
                room=_room(sim.lens))


def _sam_columns(case, seed) -> records.SamBatch:
    """Finished records as a service holds them: the reads' bases and qualities in page-locked memory."""
    rng = np.random.default_rng(seed)
    n = case["records"]
    lens = _lengths(n, case["lo"], case["hi"])
    off = np.zeros(n + 1, np.int64)
    np.cumsum(lens, out=off[1:])
    total = int(off[-1])

    def pinned(a):
        return torch.from_numpy(a).pin_memory().numpy()

    seq = pinned(np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, total, dtype=np.uint8)])
    qual = pinned(rng.integers(0, 60, total, dtype=np.uint8))
    # a CIGAR per record: '=' runs of about 200 bases that fill the read, one-base deletions between them
    words, clen = [], np.zeros(n, np.int32)
    for r in range(n):
        k = max(1, int(lens[r]) // 200)
        cut = np.unique(rng.integers(1, lens[r], size=k))
        runs = np.diff(np.concatenate([[0], cut, [lens[r]]])).astype(np.uint32)
        w = np.empty(2 * len(runs) - 1, np.uint32)
        w[0::2] = runs << 4  # '=' over the bases
        w[1::2] = (np.uint32(1) << 4) | np.uint32(3)  # a one-base deletion between them
        words.append(w)
        clen[r] = len(w)
    cstart = np.zeros(n, np.int64)
    np.cumsum(clen[:-1], out=cstart[1:])
    names = [f"read{r}".encode() for r in range(n)]
    name_off = np.zeros(n + 1, np.int64)
    np.cumsum([len(x) for x in names], out=name_off[1:])
    start = rng.integers(0, 9_000_000, size=n)
    tag = np.frombuffer(b"RG:Z:ont\tXM:Z:ont", np.uint8)
    return records.SamBatch(
        np.frombuffer(b"".join(names), np.uint8).copy(), name_off, seq, off, qual, np.zeros(n, np.int32),
        np.frombuffer(b"ref0", np.uint8).copy(), np.array([0, 4], np.int64), start, start + lens,
        np.where(rng.random(n) < 0.5, 1, -1).astype(np.int8), rng.integers(0, 61, size=n).astype(np.int32),
        np.concatenate(words), cstart, clen, np.tile(tag, n), np.arange(n + 1, dtype=np.int64) * len(tag), ["ont"])


# --------------------------------------------------------------------------- #
# One pass
# --------------------------------------------------------------------------- #
class Results(dict):
    """A call's result buffers.  CIGAR words lie in the order in which the
    pairs finished, a read's chain slots beyond its chain count hold nothing,
    and the sizes of the results depend on the data: such an entry is a
    function that gives what a reader takes from the buffers, pair by pair
    and read by read in an array of fixed size, when it is looked at."""

    def __getitem__(self, key):
        v = super().__getitem__(key)
        return v() if callable(v) else v


def _fill(a, n: int) -> torch.Tensor:
    """The rows of ``a``, followed by zeros up to ``n`` rows."""
    t = a if isinstance(a, torch.Tensor) else torch.from_numpy(np.array(a))
    out = torch.zeros((max(n, len(t)),) + tuple(t.shape[1:]), dtype=t.dtype, device=t.device)
    out[: len(t)] = t
    return out


def _by_pair(words, start, count, n: int) -> torch.Tensor:
    """Variable-length entries (``count`` words from ``start``) one pair after another."""
    t = [x if isinstance(x, torch.Tensor) else torch.from_numpy(np.array(x)) for x in
         (words.view(np.int32) if isinstance(words, np.ndarray) else words, start, count)]
    count = t[2].long().clamp(min=0)
    row = torch.repeat_interleave(count)
    at = torch.arange(row.numel(), device=count.device) - (torch.cumsum(count, 0) - count)[row]
    return _fill(t[0][t[1].long()[row] + at], n)


def run(state: dict):
    kind, room = state["kind"], state["room"]
    if kind == "pairs":
        o = extension.launch_banded_sw(state["dp"], state["params"], state["cigar"], out=state["out"])
        r = Results(score=o.score, query_end=o.query_end, target_end=o.target_end, error_flags=o.error_flags)
        if state["cigar"]:
            r.update(query_start=o.query_start, target_start=o.target_start, op_counts=o.op_counts,
                     cigar_len=o.cigar_len, cigar=lambda: _by_pair(o.cigar, o.cigar_start, o.cigar_len, room))
        return r
    if kind == "chain":
        da = state["da"]
        o = chaining.launch_chain_batch(da, state["cfg"], out=state["out"])
        mc = o.max_chains

        def slots(t, width=1):
            kept = torch.arange(mc, device=t.device)[None, :, None] < o.n_chains[:, None, None]
            return torch.where(kept, t.reshape(da.n_reads, mc, width), torch.zeros_like(t[:1]))

        return Results(n_chains=o.n_chains, score=lambda: slots(o.score), strand=lambda: slots(o.strand),
                       span=lambda: slots(o.span, 4), is_primary=lambda: slots(o.is_primary),
                       n_members=lambda: slots(o.n_members),
                       members=lambda: _by_pair(o.members, da.read_off[:-1], slots(o.n_members).sum((1, 2)), room))
    if kind == "seed":
        a = state["index"].seed_device(state["codes"], state["off"], state["n"])
        cols = {x: (lambda x=x: _fill(a[x][: a["n_anchors"]], room)) for x in ("read_pos", "ref_pos", "length", "strand")}
        return Results(read_off=a["read_off"], max_read_anchors=a["max_read_anchors"], **cols)
    if kind == "wfa":
        r = wfa.align_device_pairs(state["dp"], 4096)
        return Results(distance=r.distance, op_counts=r.op_counts, cigar_len=r.cigar_len,
                       cigar=lambda: _by_pair(r.cigar_words, r.cigar_start, r.cigar_len, room))
    if kind == "serve":
        b = state["aligner"].align(state["reads"])
        k, most = b.cols, 8 * len(state["reads"])  # at most max_chains chains of a read
        named = dict(chain_score=b.chains["score"], strand=b.chains["strand"], score=k["score"], read_start=k["qs"],
                     read_end=k["qe"], ref_start=k["ts"], ref_end=k["te"], op_counts=k["counts"], cigar_len=k["clen"])
        return Results({x: (lambda v=v: _fill(v, most)) for x, v in named.items()}, chain_off=b.chain_off,
                       cigar=lambda: _by_pair(b.words, k["cstart"], k["clen"], room))
    text = records.render_sam_array(state["batch"])
    return Results(text=lambda: _fill(text, room))


# --------------------------------------------------------------------------- #
# What a pass cannot do without
# --------------------------------------------------------------------------- #
def _mean_len(case) -> float:
    lo, hi = case["lo"], case["hi"]
    return min(max(2_100.0, lo), hi) if hi >= 8 * lo else 0.5 * (lo + hi)


def work(case: dict) -> dict:
    L, kind = _mean_len(case), case["kind"]
    if kind == "pairs":  # codes in, results out; 11 integer operations per in-band cell
        W = 2 * min(case["band"] + case["slope"] * L, case["cap"]) + 1
        n = case["n"]
        return {"bytes": n * (2 * L + 64 + (60 if case["cigar"] else 12)), "flops": 11.0 * n * L * min(W, L + 2 * FLANK)}
    if kind == "chain":  # 13 bytes of an anchor in, its membership out; one candidate is 10 operations
        a = case["reads"] * L * (0.18 if case["err"] == "hifi" else 0.13)
        return {"bytes": a * 17 + case["reads"] * 200.0, "flops": 10.0 * a}
    if kind == "seed":  # codes in, 13 bytes per anchor out; hash and window minimum of both orientations
        b = case["reads"] * L
        return {"bytes": b * (1 + 0.15 * 13), "flops": 2 * 30.0 * b}
    if kind == "wfa":  # both sequences in, CIGARs out; diagonals of the wavefronts
        n, d = case["n"], 0.03 * L
        return {"bytes": n * (2 * L + 4 * d + 40), "flops": n * (10.0 * d * d + 2 * L)}
    if kind == "serve":  # reads and windows in, results out; the extension's cells
        n = case["reads"]
        return {"bytes": n * (3 * L + 0.15 * L * 30 + 100), "flops": 11.0 * n * L * 130}
    n = case["records"]
    return {"bytes": n * (4 * L + 120.0), "flops": 2.0 * n * L}


# --------------------------------------------------------------------------- #
# Chain scores in plain numpy
# --------------------------------------------------------------------------- #
def _chain_scores(re, fe, w, cfg) -> list:
    """Scores of the chains of one strand's sorted anchors, in the order in which they are peeled off."""
    n = len(re)
    f, par = np.zeros(n), np.full(n, -1, np.int64)
    for i in range(n):
        j = np.arange(max(0, i - cfg.max_lookback), i)
        dq, dr = re[i] - re[j], fe[i] - fe[j]
        ok = (dq > 0) & (dr > 0) & (dq <= cfg.max_gap) & (dr <= cfg.max_gap)
        f[i] = w[i]
        if ok.any():
            j, dq, dr = j[ok], dq[ok], dr[ok]
            gap = np.abs(dr - dq)
            pen = np.where(gap > 0, cfg.gap_open + cfg.gap_extend * gap + cfg.log_coeff * np.log2(gap + 1.0), 0.0)
            s = f[j] + np.minimum(np.minimum(dq, dr), w[i]) - pen
            b = int(np.argmax(s))
            if s[b] > f[i]:
                f[i], par[i] = s[b], j[b]
    taken, out = np.zeros(n, bool), []
    for i in np.argsort(-f, kind="stable"):
        if taken[i]:
            continue
        x, members = int(i), 0
        while x >= 0 and not taken[x]:
            taken[x] = True
            members += 1
            x = int(par[x])
        s = f[i] - (f[x] if x >= 0 else 0.0)
        if members >= cfg.min_chain_anchors and s >= cfg.min_chain_score:
            out.append(s)
    return out


def exact(case: dict, seed: int):
    """Chain scores in 64 bits where a read or a few are chained (a read's
    best chain alone where it has only one above the secondary cutoff);
    every other output is a whole number or text."""
    if case["kind"] != "chain" or case["reads"] * case["hi"] > 400_000:
        return None
    st = prepare(case, seed)
    da, cfg = st["da"], st["cfg"]
    off = da.read_off.cpu().numpy()
    cols = [t.cpu().numpy()[: da.n_anchors].astype(np.int64) for t in (da.read_pos, da.ref_pos, da.length, da.strand)]
    scores = []
    for r in range(da.n_reads):
        rp, fp, ln, sd = (c[off[r]: off[r + 1]] for c in cols)
        found = []
        for strand in (1, -1):
            x = np.flatnonzero(sd == strand)
            x = x[np.lexsort((rp[x] + ln[x], fp[x] + ln[x]))]
            found += _chain_scores((rp + ln)[x], (fp + ln)[x], ln[x].astype(np.float64), cfg)
        found.sort(reverse=True)
        if len(found) > 1 and found[1] >= cfg.secondary_score_ratio * found[0]:
            return None  # a secondary chain: its selection depends on the spans
        scores.append(found[:1] + [0.0] * (cfg.max_chains - len(found[:1])))
    return dict(n_chains=None, score=np.array(scores).reshape(da.n_reads, -1, 1), strand=None, span=None,
                is_primary=None, n_members=None, members=None)
