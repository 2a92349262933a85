"""The tiled seeding pass (gmf_seed_scan / gmf_seed_emit) against the
one-block-per-read passes (gmf_seed_count / gmf_seed_fill): read lengths
around the 512-position tile, window and k-mer sizes from the smallest to the
largest, N runs, repeated keys, more reads than one search level holds, one
orientation only, and no prefix table."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _count_fill(idx, codes, off, n, both):
    import torch

    from graphmambaformer_b200 import _native

    lib, vp, c = _native.lib(), ctypes.c_void_p, idx.c()
    sp = vp(int(torch.cuda.current_stream().cuda_stream))
    counts = torch.empty(2 * n, dtype=torch.int64, device="cuda")
    _native.check("count", lib.gmf_seed_count(ctypes.byref(c), n, vp(codes.data_ptr()), vp(off.data_ptr()), both,
                                              vp(counts.data_ptr()), sp))
    aoff = torch.zeros(2 * n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(counts, 0, out=aoff[1:])
    t = int(aoff[-1])
    out = [torch.empty(max(t, 1), dtype=d, device="cuda") for d in (torch.int32, torch.int32, torch.int32, torch.int8)]
    _native.check("fill", lib.gmf_seed_fill(ctypes.byref(c), n, vp(codes.data_ptr()), vp(off.data_ptr()), both,
                                            vp(aoff.data_ptr()), *[vp(x.data_ptr()) for x in out], sp))
    return aoff[::2].cpu().numpy(), [x[:t].cpu().numpy() for x in out]


@pytest.mark.parametrize("k,w", [(15, 10), (4, 1), (5, 2), (31, 19), (11, 256), (7, 33)])
def test_tiled_pass_equals_the_pass_per_read(k, w):
    import torch

    from graphmambaformer_b200 import synth
    from graphmambaformer_b200.seeding import DeviceMinimizerIndex

    rng = np.random.default_rng(1000 * k + w)
    ref = synth.random_reference(30_000, rng).astype(np.int8)
    ref[20_000:20_600] = ref[1_000:1_600]
    idx = DeviceMinimizerIndex(ref, k=k, w=w, device="cuda:0")
    lens = [0, 1, k - 1, k, k + 1, 511 + k - 1, 512 + k - 1, 513 + k - 1, 1024 + k - 1, 1025 + k, 2000, 5000]
    lens += [int(x) for x in rng.integers(k, 120, 1100)]
    reads = []
    for n in lens:
        s = int(rng.integers(0, len(ref) - n))
        r = synth.apply_errors(ref[s: s + n], synth.ONT, rng).astype(np.int8)
        if n > 1000:
            r[700:760] = 5
        reads.append(synth.reverse_complement(r) if n % 2 else r)
    off = np.zeros(len(reads) + 1, np.int64)
    np.cumsum([len(r) for r in reads], out=off[1:])
    codes = torch.from_numpy(np.concatenate(reads)).cuda()
    off_d = torch.from_numpy(off).cuda()
    table = idx.prefix
    for both in (1, 0):
        want_off, want = _count_fill(idx, codes, off_d, len(reads), both)
        for prefix in (table, None):
            idx.prefix = prefix
            got = idx.seed_device(codes, off_d, len(reads), bool(both))
            t = got["n_anchors"]
            assert np.array_equal(got["read_off"].cpu().numpy(), want_off)
            assert got["max_read_anchors"] == int(np.diff(want_off).max())
            for name, x in zip(("read_pos", "ref_pos", "length", "strand"), want):
                assert np.array_equal(got[name][:t].cpu().numpy(), x), (name, both, prefix is None)
    idx.prefix = table
