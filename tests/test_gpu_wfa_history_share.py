"""gmf_wfa_align_direct in a workspace of the pairs' own shares of history:
unrelated pairs, which need many times theirs, leave the other pairs room."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_unrelated_pairs_leave_the_others_their_share():
    import torch

    from graphmambaformer_b200 import _native, synth, wfa

    rng = np.random.default_rng(6)
    ref = synth.random_reference(40_000, rng).astype(np.int8)
    # more long unrelated pairs than the GPU runs at once, longest first, so all of them start before the others
    qs = [ref[s: s + 4_100] for s in rng.integers(0, 15_000, 160)]
    ts = [ref[s: s + 4_100] for s in rng.integers(20_000, 35_000, 160)]
    for s in rng.integers(0, 30_000, 64):
        qs.append(synth.apply_errors(ref[s: s + 300], synth.ONT, rng).astype(np.int8))
        ts.append(ref[s: s + 300])
    dp = wfa.upload_wfa_pairs(qs, ts)
    lib, n, md = _native.lib(), dp.n, 4096
    need = int(lib.gmf_wfa_workspace_bytes(n, dp.max_len, md, wfa.direct_entries(dp.h_qlen, dp.h_tlen, md)))
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    cap = int(dp.h_qlen.sum() + dp.h_tlen.sum()) + n
    i32 = dict(dtype=torch.int32, device="cuda")
    counts, cigar, clen, dist = torch.empty(4 * n, **i32), torch.empty(cap, **i32), torch.empty(n, **i32), torch.empty(n, **i32)
    start, used = torch.empty(n, dtype=torch.int64, device="cuda"), torch.empty(1, dtype=torch.int64, device="cuda")
    err = torch.empty(1, **i32)
    order = torch.arange(n, **i32)
    res = _native.GmfWfaResults(counts.data_ptr(), cigar.data_ptr(), cap, start.data_ptr(), clen.data_ptr(),
                                used.data_ptr(), err.data_ptr())
    pairs = dp.c(order)
    sp = ctypes.c_void_p(int(torch.cuda.current_stream().cuda_stream))
    _native.check("direct", lib.gmf_wfa_align_direct(ctypes.byref(pairs), md, ctypes.c_void_p(dist.data_ptr()),
                                                     ctypes.byref(res), ctypes.c_void_p(ws.data_ptr()), need, sp))
    got = clen.cpu().numpy()
    assert int(err[0]) == 0 and np.all(dist.cpu().numpy() >= 0)
    assert np.all(got[160:] >= 0) and np.any(got[:160] == -2)
    # and the call that replays what did not fit gives every pair its CIGAR
    r = wfa.align_device_pairs(dp, md)
    assert np.array_equal(r.distance, dist.cpu().numpy())
    assert np.array_equal(r.op_counts[:, 1:].sum(1), r.distance)
    assert np.array_equal(r.op_counts[:, :3].sum(1), dp.h_qlen)
