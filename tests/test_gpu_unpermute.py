"""The reverse permutation (layout -> sorted order) through the C ABI.

The reference has no reverse permutation; its forward layouts, as the oracle
restates them, are the inputs: bit-exact on seeded keys at sizes the oracle
finishes in seconds (every size 1..300, tile and unit boundaries, both key
widths), and at the benchmark's sizes a round trip permute -> unpermute that
must give back the input exactly.
"""
import numpy as np
import pytest

import oracle as O
import tree_layouts as T
from gpu_util import from_dev, to_dev
from tree_layouts import data

pytestmark = pytest.mark.gpu

CASES = [("bst", 1), ("btree", 2), ("btree", 3), ("btree", 8), ("btree", 16), ("btree", 32), ("mveb", 0), ("veb", 0)]
EDGE = [511, 4095, 4096, 4097, 8191, 8192, 8193, 65535, 65537, 83521, 262143, 300001, 1048575, 3000017]


@pytest.mark.parametrize("layout,b", CASES)
@pytest.mark.parametrize("dtype", [np.uint64, np.uint32])
def test_oracle_layouts_back_to_sorted(layout, b, dtype):
    for n in list(range(1, 301, 7)) + EDGE:
        keys = data.sorted_keys_np(n, 1, 3, 13 + n, dtype)
        t = to_dev(O.permute(layout, keys, b or 16))
        T.unpermute(layout, t, b or 16)
        assert np.array_equal(from_dev(t), keys), (layout, b, n)


def test_caller_workspace_timing_and_too_small():
    import torch
    n = 1_000_003
    keys = data.sorted_keys_np(n, 1, 16, 3)
    t = to_dev(O.permute("btree", keys, 16))
    need = T.lib().tl_unpermute_workspace_bytes
    import ctypes as C
    out = C.c_uint64()
    assert need(1, n, 16, 8, C.byref(out)) == 0
    ws = torch.empty(out.value, dtype=torch.uint8, device="cuda")
    assert T.unpermute("btree", t, 16, workspace=ws, timed=True) > 0
    assert np.array_equal(from_dev(t), keys)
    small = torch.empty(out.value - 256, dtype=torch.uint8, device="cuda")
    with pytest.raises(T.TreeLayoutError) as e:
        T.unpermute("btree", t, 16, workspace=small)
    assert e.value.status == T.ERROR_WORKSPACE_TOO_SMALL
    assert np.array_equal(from_dev(t), keys)  # rejected before any device work


@pytest.mark.parametrize("layout,b,n,kb,gap", [
    ("btree", 16, 500_000_000, 8, 16),
    ("bst", 1, 2**28 - 1, 8, 16),
    ("btree", 8, 60_000_000, 8, 16),
    ("mveb", 0, 2**30 - 1, 4, 3),
    ("veb", 0, 300_000_000, 4, 3),
])
def test_full_size_round_trip(layout, b, n, kb, gap):
    import torch
    keys = data.sorted_keys_torch(n, 1, gap, 17, kb)
    t = keys.clone()
    T.permute(layout, t, b)
    assert not torch.equal(t, keys)
    T.unpermute(layout, t, b)
    assert torch.equal(t, keys)


@pytest.mark.parametrize("layout,b,n,kb,skip", [
    # either side of each form's line (8, 32, 192 MB), ragged sizes, arrays that
    # start off a 16- or 128-byte boundary (no vector stores, shifted stretches)
    ("btree", 16, (8 << 17) - 1, 8, 1), ("btree", 16, (8 << 17) + 1, 8, 0), ("btree", 3, 2_100_001, 4, 3),
    ("btree", 16, 25_165_824, 8, 0), ("btree", 16, 25_165_825, 8, 1), ("btree", 2, 60_000_001, 4, 5),
    ("btree", 1000, 30_000_001, 8, 3), ("btree", 100_000, 50_331_777, 4, 1),
    ("bst", 1, 2**25 + 5, 8, 1), ("bst", 1, 2**26 - 1, 8, 0), ("bst", 1, 3 * 2**25 + 1, 8, 1),
    ("mveb", 0, 2**22, 8, 1), ("mveb", 0, 2**22 + 1, 8, 0), ("mveb", 0, 2**23 - 1, 8, 1), ("mveb", 0, 2**24 + 7, 4, 3),
    ("veb", 0, 2**23 + 1, 4, 1), ("veb", 0, 2**19 - 1, 8, 1), ("veb", 0, 12_345_679, 8, 1), ("veb", 0, 2**25 - 1, 4, 0),
])
def test_reverse_forms_round_trip(layout, b, n, kb, skip):
    import torch
    keys = data.sorted_keys_torch(n, 1, 3, 5, kb)
    buf = torch.full((n + skip + 64,), -1, dtype=keys.dtype, device="cuda")
    t = buf[skip:skip + n]
    t.copy_(keys)
    T.permute(layout, t, b or 16)
    T.unpermute(layout, t, b or 16)
    assert torch.equal(t, keys)
    assert bool((buf[:skip] == -1).all()) and bool((buf[skip + n:] == -1).all())


def test_expired_reverse_wait_reports_timeout_and_context_survives():
    import torch
    n = 30_000_001
    keys = data.sorted_keys_torch(n, 1, 16, 9, 8)
    t = keys.clone()
    T.permute("btree", t, 16)
    lay = t.clone()
    T.set_wait(spin_limit=64, force_timeout=True)
    try:
        with pytest.raises(T.TreeLayoutError) as e:
            T.unpermute("btree", t, 16)
        assert e.value.status == T.ERROR_TIMEOUT
    finally:
        T.set_wait(0, False)
    T.unpermute("btree", lay, 16)
    assert torch.equal(lay, keys)


def test_restores_from_a_copy_build_no_tile_tables():
    """B-trees that go back from a copy use no ordered-tile tables and take no
    place in the library's cache of them (64 geometries): after 70 such restores a
    permutation of a new size still has the ordered schedule.  In a process of its
    own, as the cache is the process's."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = f"""
import ctypes as C
import sys
sys.path.insert(0, {os.path.join(root, "tree-layouts_b200")!r})
import torch
import tree_layouts as T
plan = T.lib().tl_debug_permute_plan
plan.argtypes = [C.c_int, C.c_uint64, C.c_uint64, C.c_uint32]
words = torch.arange(2_000_000, device="cuda", dtype=torch.int64)
for x in range(70):
    T.unpermute("btree", words[:1_700_000 + 4321 * x].clone(), 16)
assert plan(1, 3_000_000, 16, 8) == 2
"""
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300)


@pytest.mark.parametrize("layout", ["mveb", "veb"])
@pytest.mark.parametrize("n,kb", [(7 << 20, 8), ((7 << 20) + 1, 8), ((14 << 20) - 1, 4), ((14 << 20) + 5, 4)])
def test_veb_forms_round_trip_at_their_line(layout, n, kb):
    """vEB arrays of 56 MB go back from a copy, larger ones in place."""
    import torch
    keys = data.sorted_keys_torch(n, 1, 3, 5, kb)
    buf = torch.full((n + 65,), -1, dtype=keys.dtype, device="cuda")
    t = buf[1:n + 1]
    t.copy_(keys)
    T.permute(layout, t)
    assert not torch.equal(t, keys)
    T.unpermute(layout, t)
    assert torch.equal(t, keys)
    assert int(buf[0]) == -1 and bool((buf[n + 1:] == -1).all())


@pytest.mark.parametrize("b", [1, 2, 3, 8, 16, 17, 32])
@pytest.mark.parametrize("kb", [4, 8])
@pytest.mark.parametrize("mb", [13, 200])
def test_reverse_by_tiles_round_trip_at_tile_edges(b, kb, mb):
    """B-trees and BSTs just above the sizes that go back key by key (12 MB) and
    from a copy (192 MB), around whole tiles of 32 KB and off a line."""
    import torch
    tile = 32768 // kb
    for tiles, extra in ((mb * 32, 0), (mb * 32, 1), (mb * 32 + 1, -1), (mb * 32 + 3, 1000)):
        n = tiles * tile + extra
        keys = data.sorted_keys_torch(n, 1, 3, 5, kb)
        buf = torch.full((n + 3,), -1, dtype=keys.dtype, device="cuda")
        t = buf[3:]
        t.copy_(keys)
        layout = "bst" if b == 1 else "btree"
        T.permute(layout, t, b)
        T.unpermute(layout, t, b)
        assert torch.equal(t, keys), (b, kb, n)
        assert bool((buf[:3] == -1).all())
