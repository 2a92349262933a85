"""gmf_seed_scan / gmf_seed_emit with fewer total codes than the reads have:
a read that goes on beyond them is cut there, later ones are empty, and no
code beyond is read."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scan_emit(idx, codes, off, n, total, both):
    import torch

    from graphmambaformer_b200 import _native

    lib, vp, c = _native.lib(), ctypes.c_void_p, idx.c()
    sp = vp(int(torch.cuda.current_stream().cuda_stream))
    ws = torch.empty(lib.gmf_seed_workspace_bytes(n, total), dtype=torch.uint8, device="cuda")
    aoff = torch.zeros(2 * n + 1, dtype=torch.int64, device="cuda")
    totals = torch.zeros(2, dtype=torch.int64, device="cuda")
    _native.check("scan", lib.gmf_seed_scan(ctypes.byref(c), None, n, vp(codes.data_ptr()), vp(off.data_ptr()), total,
                                            both, vp(aoff.data_ptr()), None, vp(totals.data_ptr()), vp(ws.data_ptr()),
                                            ws.numel(), sp))
    t = int(totals[0])
    out = [torch.empty(max(t, 1), dtype=d, device="cuda") for d in (torch.int32, torch.int32, torch.int32, torch.int8)]
    _native.check("emit", lib.gmf_seed_emit(ctypes.byref(c), n, vp(off.data_ptr()), total, both, vp(aoff.data_ptr()),
                                            *[vp(x.data_ptr()) for x in out], vp(ws.data_ptr()), ws.numel(), sp))
    return aoff.cpu().numpy(), [x[:t].cpu().numpy() for x in out]


@pytest.mark.parametrize("both", [0, 1])
@pytest.mark.parametrize("first", [0, 700])
def test_reads_are_cut_at_the_total_codes(first, both):
    import torch

    from graphmambaformer_b200 import synth
    from graphmambaformer_b200.seeding import DeviceMinimizerIndex

    rng = np.random.default_rng(3)
    ref = synth.random_reference(30_000, rng).astype(np.int8)
    idx = DeviceMinimizerIndex(ref, k=15, w=10, device="cuda:0")
    lens = np.array([600, 0, 14, 2100, 5000, 300])
    off = np.zeros(len(lens) + 1, np.int64)
    np.cumsum(lens, out=off[1:])
    off += first
    codes = np.concatenate([ref[:first], *[ref[s: s + n] for s, n in zip(rng.integers(0, 20_000, len(lens)), lens)]])
    codes_d, off_d = torch.from_numpy(codes).cuda(), torch.from_numpy(off).cuda()
    for total in (len(codes), len(codes) - 1, int(off[4]) + 1030, int(off[4]) + 3, int(off[1]) - 88, first, first // 2):
        got_off, got = _scan_emit(idx, codes_d, off_d, len(lens), total, both)
        cut = torch.from_numpy(np.minimum(off, total)).cuda()
        want_off, want = _scan_emit(idx, codes_d, cut, len(lens), len(codes), both)
        assert np.array_equal(got_off, want_off), total
        for a, b in zip(got, want):
            assert np.array_equal(a, b), total
