"""Minimizer seeding on the device.

The index is the reference's (w, k) minimizer table (alignment/seeding.py
L524-538: pack_kmers, hash64, minimizer_mask, KmerTable.build with
max_occ), built once on the host by the same functions
(``synth.MinimizerSketch`` restates them) and kept on the device with a
prefix table over its keys.  Reads are seeded by ``gmf_seed_scan`` /
``gmf_seed_emit``: both orientations, forward
anchors first, reverse-complement anchors in the reverse-complemented read's
coordinates -- what SeedingEngine.seed_read (L1056-1101) collects from
MinimizerIndex.query before merging diagonals.
"""

from __future__ import annotations

import ctypes
from typing import Optional, Sequence

import numpy as np
import torch

from . import _native
from .chaining import AnchorCSR
from .device import bind, require_cuda, to_device


# Workspace of one seeding pass.  It takes about 12 bytes a base, and 8 KB for
# a read shorter than a tile: 1,000,000 reads of 150 bp took 8.3 GB and 21.5 ms
# at once, 1.4 GB and 22.2 ms in ranges of this size (0.9 GB and 22.5 ms, 0.6 GB
# and 24.2 ms in ranges of a half and a quarter of it).
SEED_WORKSPACE = 1 << 30


# Keys of an index that the tile pass can hold (it keeps 32-bit key numbers).
TILE_KEYS = 2 ** 31 - 1


def workspace_ranges(read_off: np.ndarray, budget: int) -> list:
    """Consecutive ranges [r0, r1) of reads whose seeding workspaces are at
    most ``budget`` bytes each; a read above it forms a range of its own."""
    off = np.asarray(read_off, np.int64)
    f, n, out, r0 = _native.lib().gmf_seed_workspace_bytes, len(off) - 1, [], 0
    while r0 < n:
        lo, hi = r0 + 1, n  # the most reads that fit
        while lo < hi:
            mid = (lo + hi + 1) // 2
            if f(mid - r0, int(off[mid] - off[r0])) <= budget:
                lo = mid
            else:
                hi = mid - 1
        out.append((r0, lo))
        r0 = lo
    return out or [(0, 0)]


class DeviceMinimizerIndex:
    def __init__(self, ref_codes: np.ndarray, k: int = 15, w: int = 10, max_occ: int = 0, device=None):
        from .synth import MinimizerSketch

        if not 1 <= k <= 31 or not 1 <= w <= 256:
            raise ValueError("k must be within [1, 31] and w within [1, 256]")
        self.device = require_cuda(device)
        self.k, self.w = int(k), int(w)
        sk = MinimizerSketch(np.asarray(ref_codes, np.int8), k=k, w=w, max_occ=max_occ)
        pad = lambda x, dt: x.astype(dt) if len(x) else np.zeros(1, dt)  # noqa: E731
        self.n_keys = len(sk.keys)
        self.keys = to_device(pad(sk.keys, np.int64), self.device)
        self.offsets = to_device(sk.offsets.astype(np.int64), self.device)
        self.positions = to_device(pad(sk.positions, np.int32), self.device)
        self.bytes = int(self.keys.numel() * 8 + self.offsets.numel() * 8 + self.positions.numel() * 4)
        # about one key per bucket, so a lookup is one load of the table and one or two of keys
        self.prefix = None
        if 0 < self.n_keys <= TILE_KEYS:
            self.prefix_bits = min(2 * self.k, 24, max(1, self.n_keys.bit_length()))
            self.prefix = torch.empty((1 << self.prefix_bits) + 1, dtype=torch.int32, device=self.device)
            s = torch.cuda.current_stream(self.device)
            bind(self.device, int(s.cuda_stream))
            idx = self.c()
            _native.check("gmf_seed_prefix_fill", _native.lib().gmf_seed_prefix_fill(
                ctypes.byref(idx), self.prefix_bits, ctypes.c_void_p(self.prefix.data_ptr()),
                ctypes.c_void_p(int(s.cuda_stream))))
            s.synchronize()  # other streams read it
            self.bytes += int(self.prefix.numel() * 4)

    def c(self) -> _native.GmfMinimizerIndex:
        return _native.GmfMinimizerIndex(self.k, self.w, self.n_keys, self.keys.data_ptr(), self.offsets.data_ptr(),
                                         self.positions.data_ptr())

    def seed_device(self, codes_d: torch.Tensor, read_off_d: torch.Tensor, n_reads: int, both_strands: bool = True,
                    stream: Optional[torch.cuda.Stream] = None) -> dict:
        """Seed reads already on the device (codes CSR).  Returns device
        tensors read_off (n_reads + 1, per read: forward then reverse
        anchors), read_pos, ref_pos, length, strand, the anchor count and the
        largest read's anchor count."""
        s = stream or torch.cuda.current_stream(self.device)
        bind(self.device, int(s.cuda_stream))
        # every allocation and torch op on the caller's stream: the library's
        # kernels run there, and a worker's stream is not ordered with the
        # thread's default stream
        with torch.cuda.stream(s):
            if self.n_keys > TILE_KEYS:
                return self._seed_reads(codes_d, read_off_d, n_reads, both_strands, s)
            need = int(_native.lib().gmf_seed_workspace_bytes(n_reads, int(codes_d.numel())))
            if need <= SEED_WORKSPACE:
                return self._seed_tiles(codes_d, read_off_d, n_reads, both_strands, s, need)
            # a batch whose workspace would be larger is seeded in ranges of reads
            h_off = read_off_d[: n_reads + 1].cpu().numpy()
            parts = []
            for r0, r1 in workspace_ranges(h_off, SEED_WORKSPACE):
                c0, c1 = int(h_off[r0]), int(h_off[r1])
                at = min(c0, codes_d.numel() - 1)  # a range of empty reads still has an address
                codes = codes_d[at: max(c1, at + 1)]
                need = int(_native.lib().gmf_seed_workspace_bytes(r1 - r0, int(codes.numel())))
                parts.append(self._seed_tiles(codes, read_off_d[r0: r1 + 1] - c0, r1 - r0, both_strands, s, need))
            if len(parts) == 1:
                return parts[0]
            n = [p["n_anchors"] for p in parts]
            out = dict(n_anchors=sum(n), max_read_anchors=max(p["max_read_anchors"] for p in parts))
            base = np.cumsum([0] + n)
            out["read_off"] = torch.cat([p.pop("read_off")[: None if k == len(n) - 1 else -1] + int(base[k])
                                         for k, p in enumerate(parts)])
            for name in ("read_pos", "ref_pos", "length", "strand"):
                out[name] = torch.cat([p.pop(name)[:t] for p, t in zip(parts, n)])
                if out["n_anchors"] == 0:
                    out[name] = out[name].new_empty(1)
        return out

    def _seed_tiles(self, codes_d: torch.Tensor, read_off_d: torch.Tensor, n_reads: int, both_strands: bool,
                    s: torch.cuda.Stream, need: int) -> dict:
        """seed_device in one workspace of ``need`` bytes, on the current stream ``s``."""
        sp, vp, lib = int(s.cuda_stream), ctypes.c_void_p, _native.lib()
        idx = self.c()
        total_codes = int(codes_d.numel())
        pre = _native.GmfSeedPrefix(self.prefix_bits, self.prefix.data_ptr()) if self.prefix is not None else None
        both = 1 if both_strands else 0
        ws = torch.empty(max(need, 256), dtype=torch.uint8, device=self.device)
        off = torch.empty(3 * n_reads + 4, dtype=torch.int64, device=self.device)
        aoff, roff, totals = off[: 2 * n_reads + 1], off[2 * n_reads + 1: 3 * n_reads + 2], off[3 * n_reads + 2:]
        _native.check("gmf_seed_scan", lib.gmf_seed_scan(
            ctypes.byref(idx), ctypes.byref(pre) if pre is not None else None, n_reads, vp(codes_d.data_ptr()),
            vp(read_off_d.data_ptr()), total_codes, both, vp(aoff.data_ptr()), vp(roff.data_ptr()),
            vp(totals.data_ptr()), vp(ws.data_ptr()), ws.numel(), vp(sp)))
        # the total sizes the outputs; the largest read is checked against the chaining limit (one
        # host round trip for both)
        total, most = (int(x) for x in totals.cpu().tolist())
        i32 = dict(dtype=torch.int32, device=self.device)
        out = dict(read_pos=torch.empty(max(total, 1), **i32), ref_pos=torch.empty(max(total, 1), **i32),
                   length=torch.empty(max(total, 1), **i32),
                   strand=torch.empty(max(total, 1), dtype=torch.int8, device=self.device))
        _native.check("gmf_seed_emit", lib.gmf_seed_emit(
            ctypes.byref(idx), n_reads, vp(read_off_d.data_ptr()), total_codes, both, vp(aoff.data_ptr()),
            vp(out["read_pos"].data_ptr()), vp(out["ref_pos"].data_ptr()), vp(out["length"].data_ptr()),
            vp(out["strand"].data_ptr()), vp(ws.data_ptr()), ws.numel(), vp(sp)))
        out.update(read_off=roff, n_anchors=total, max_read_anchors=most)
        return out

    def _seed_reads(self, codes_d: torch.Tensor, read_off_d: torch.Tensor, n_reads: int, both_strands: bool,
                    s: torch.cuda.Stream) -> dict:
        """seed_device by one block per read and orientation, for an index of
        any size, on the current stream ``s``."""
        sp, vp, lib = int(s.cuda_stream), ctypes.c_void_p, _native.lib()
        idx, both = self.c(), 1 if both_strands else 0
        counts = torch.empty(max(2 * n_reads, 1), dtype=torch.int64, device=self.device)
        _native.check("gmf_seed_count", lib.gmf_seed_count(
            ctypes.byref(idx), n_reads, vp(codes_d.data_ptr()), vp(read_off_d.data_ptr()), both,
            vp(counts.data_ptr()), vp(sp)))
        aoff = torch.zeros(2 * n_reads + 1, dtype=torch.int64, device=self.device)
        if n_reads:
            torch.cumsum(counts[: 2 * n_reads], 0, out=aoff[1:])
        per_read = (counts[0: 2 * n_reads: 2] + counts[1: 2 * n_reads: 2]).max() if n_reads else counts[0] * 0
        total, most = (int(x) for x in torch.stack([aoff[-1], per_read]).cpu().tolist())
        i32 = dict(dtype=torch.int32, device=self.device)
        out = dict(read_pos=torch.empty(max(total, 1), **i32), ref_pos=torch.empty(max(total, 1), **i32),
                   length=torch.empty(max(total, 1), **i32),
                   strand=torch.empty(max(total, 1), dtype=torch.int8, device=self.device))
        _native.check("gmf_seed_fill", lib.gmf_seed_fill(
            ctypes.byref(idx), n_reads, vp(codes_d.data_ptr()), vp(read_off_d.data_ptr()), both, vp(aoff.data_ptr()),
            vp(out["read_pos"].data_ptr()), vp(out["ref_pos"].data_ptr()), vp(out["length"].data_ptr()),
            vp(out["strand"].data_ptr()), vp(sp)))
        out.update(read_off=aoff[::2].contiguous(), n_anchors=total, max_read_anchors=most)
        return out

    def seed(self, reads: Sequence[np.ndarray], both_strands: bool = True) -> AnchorCSR:
        """Host reads in, host anchors (CSR, per read forward then reverse) out."""
        n = len(reads)
        off = np.zeros(n + 1, np.int64)
        np.cumsum([len(r) for r in reads], out=off[1:])
        codes = np.concatenate([np.asarray(r, np.int8) for r in reads]) if off[-1] else np.zeros(1, np.int8)
        d = self.seed_device(to_device(codes, self.device), to_device(off, self.device), n, both_strands)
        torch.cuda.synchronize(self.device)
        t = d["n_anchors"]
        return AnchorCSR(d["read_off"].cpu().numpy(), d["read_pos"][:t].cpu().numpy(), d["ref_pos"][:t].cpu().numpy(),
                         d["length"][:t].cpu().numpy(), d["strand"][:t].cpu().numpy())
