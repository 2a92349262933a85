"""The delay line of the one-warp SW classes: its ring holds the delay and one
chunk of 4 steps more, whatever the band, so that the entries a chunk stores
are never those it reads (nothing orders the two within a chunk)."""

from __future__ import annotations

import ctypes

import pytest


@pytest.mark.parametrize("lanes", [8, 16, 32])
def test_a_chunk_never_stores_what_it_reads(lanes):
    from graphmambaformer_b200 import _native

    lib = _native.lib()
    d, n = ctypes.c_int32(), ctypes.c_int32()
    full = set()
    for hb in range(4097):
        assert lib.gmf_sw_test_delay_ring(hb, lanes, ctypes.byref(d), ctypes.byref(n)) == _native.GMF_OK
        ring = n.value
        assert ring & (ring - 1) == 0 and d.value % 4 == 0
        reads = {(-d.value + u) % ring for u in range(4)}
        stores = {u % ring for u in range(4)}
        assert d.value == 0 or not reads & stores, (lanes, hb, d.value, ring)
        if d.value and d.value & (d.value - 1) == 0:
            full.add(d.value)
    assert {4, 32, 128, 1024, 4096} <= full  # delays that fill a power of two
    assert lib.gmf_sw_test_delay_ring(5, 4, ctypes.byref(d), ctypes.byref(n)) == _native.GMF_ERR_INVALID_ARGUMENT
