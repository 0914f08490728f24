"""Parity of the sm_100a query kernels with the oracle (and, through the golden
fixtures, with the reference's own query code), through the C ABI."""
import hashlib
import json
import os

import numpy as np
import pytest

import oracle as O
import tree_layouts as T
from gpu_util import from_dev, to_dev
from tree_layouts import data

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")


def sha(a):
    return hashlib.sha256(np.ascontiguousarray(a, dtype=np.uint64).tobytes()).hexdigest()[:24]


def gpu_answers(layout, tree, Q, b=16):
    import torch
    ans = torch.empty(len(Q), dtype=torch.int64, device="cuda")
    T.query(layout, to_dev(tree), to_dev(Q), ans, b)
    return ans.cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("layout,b", [("bst", 1), ("btree", 16), ("btree", 8), ("btree", 3), ("btree", 32),
                                      ("btree", 1), ("btree", 64), ("mveb", 0), ("veb", 0)])
@pytest.mark.parametrize("dtype", [np.uint64, np.uint32])
def test_queries_match_oracle(layout, b, dtype):
    for n in [1, 2, 3, 5, 16, 17, 100, 255, 1000, 4097, 65535, 70001, 1048575, 3000017]:
        keys = data.sorted_keys_np(n, 1, 16 if dtype == np.uint64 else 3, n, dtype)
        tree = O.permute(layout, keys, b or 16)
        Q = data.queries_np(keys, 5000, 0.5, n + 1)
        Q = np.concatenate([Q, keys[:1] - 1 if keys[0] > 0 else keys[:1], keys[-1:] + 1]).astype(dtype)
        exp = O.search(layout, tree, Q, b or 16)
        got = gpu_answers(layout, tree, Q, b or 16)
        assert np.array_equal(got, exp), (layout, b, n)


@pytest.mark.parametrize("dtype", [np.uint64, np.uint32])
def test_sorted_binary_search_matches_oracle(dtype):
    for n in [1, 2, 3, 4, 5, 7, 8, 100, 4095, 4096, 8191, 8192, 8193, 65537, 1048575, 3000017]:
        keys = data.sorted_keys_np(n, 1, 16 if dtype == np.uint64 else 3, n + 7, dtype)
        Q = data.queries_np(keys, 5000, 0.5, n + 8)
        edge = [keys[0] - 1 if keys[0] > 0 else keys[0], keys[0], keys[-1], keys[-1] + 1]
        Q = np.concatenate([Q, np.array(edge, dtype=dtype)]).astype(dtype)
        exp = O.search_sorted(keys, Q)
        got = gpu_answers("sorted", keys, Q)
        assert np.array_equal(got, exp), (n, dtype)


def test_queries_match_reference_golden():
    with open(os.path.join(GOLD, "golden_cpu.json")) as f:
        g = json.load(f)
    for e in g["query_btree"]:
        keys = data.sorted_keys_np(e["n"], 1, 16, e["seed"])
        Q = data.queries_np(keys, e["q"], 0.5, e["seed"] + 1)
        assert sha(gpu_answers("btree", O.permute("btree", keys, e["b"]), Q, e["b"])) == e["sha"]
    for e in g["query_bst"]:
        keys = data.sorted_keys_np(e["n"], 1, 16, e["seed"])
        Q = data.queries_np(keys, e["q"], 0.5, e["seed"] + 1)
        assert sha(gpu_answers("bst", O.permute("bst", keys), Q)) == e["sha"]


def test_standard_veb_queries_match_reference_golden():
    with open(os.path.join(GOLD, "golden_cpu.json")) as f:
        g = json.load(f)
    for e in g["query_veb_std"]:
        keys = data.sorted_keys_np(e["n"], 1, 16, e["seed"])
        Q = data.queries_np(keys, e["q"], 1.0, e["seed"] + 1)
        assert sha(gpu_answers("veb", O.permute("veb", keys), Q)) == e["sha"], e["n"]


def test_benchmark_query_shapes_small():
    # config shapes at reduced n: BST 2^20-1 u64 with q=2^20, mvEB non-perfect u32 tables
    keys = data.sorted_keys_np(2**20 - 1, 1, 16, 1)
    Q = data.queries_np(keys, 2**20, 0.5, 2)
    tree = O.permute("bst", keys)
    assert np.array_equal(gpu_answers("bst", tree, Q), O.search("bst", tree, Q))
    keys = data.sorted_keys_np(3_000_000, 1, 3, 5, np.uint32)
    Q = data.queries_np(keys, 200_000, 0.5, 6)
    tree = O.permute("mveb", keys)
    assert np.array_equal(gpu_answers("mveb", tree, Q), O.search("mveb", tree, Q))


@pytest.mark.parametrize("layout,b", [("btree", 16), ("btree", 8), ("btree", 2), ("btree", 32), ("btree", 5),
                                      ("bst", 1), ("mveb", 0)])
@pytest.mark.parametrize("dtype", [np.uint64, np.uint32])
def test_queries_on_an_unaligned_layout(layout, b, dtype):
    """A layout that starts one key past a 16-byte boundary takes the kernels'
    scalar node reads; answers are unchanged."""
    import torch
    for n in [17, 1000, 70001, 1_048_575]:
        keys = data.sorted_keys_np(n, 1, 16 if dtype == np.uint64 else 3, n + 3, dtype)
        tree = O.permute(layout, keys, b or 16)
        Q = data.queries_np(keys, 20_000, 0.5, n + 4)
        buf = to_dev(np.concatenate([np.zeros(1, dtype), tree]))
        view = buf[1:]
        assert view.data_ptr() % 16 != 0
        ans = torch.empty(len(Q), dtype=torch.int64, device="cuda")
        T.query(layout, view, to_dev(Q), ans, b or 16)
        assert np.array_equal(ans.cpu().numpy().view(np.uint64), O.search(layout, tree, Q, b or 16)), (layout, b, n)


@pytest.mark.parametrize("b", [1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 64, 100])
def test_btree_queries_every_node_width(b):
    """Every node width: 16-byte rows, one key per lane (b <= 32), and the
    scalar group kernel (b > 32 without 16-byte rows)."""
    for dtype in (np.uint64, np.uint32):
        for n in [b, b + 1, 5 * b + 3, 100_003]:
            keys = data.sorted_keys_np(n, 1, 16 if dtype == np.uint64 else 3, n + b, dtype)
            tree = O.permute("btree", keys, b)
            Q = data.queries_np(keys, 10_000, 0.5, b)
            Q = np.concatenate([Q, keys[:1] - 1 if keys[0] > 0 else keys[:1], keys[-1:] + 1]).astype(dtype)
            assert np.array_equal(gpu_answers("btree", tree, Q, b), O.search("btree", tree, Q, b)), (b, n, dtype)


@pytest.mark.parametrize("variant", [0, 2, 5, 6])
def test_btree_query_kernel_forms(variant):
    """Each B-tree node-read form gives the oracle's answers: a group of
    b*w/32 lanes with one 32-byte load each (the default for 64-, 128- and
    256-byte nodes), a thread per query with 32-byte loads (variant 6, and with
    the top levels in shared memory, 5) and with 16-byte loads (2); the partial
    last leaf and queries past both ends included."""
    import ctypes as C
    L = T.lib()
    L.tl_debug_set_query_variant.argtypes = [C.c_int]
    L.tl_debug_set_query_variant(variant)
    try:
        for b, dtype in [(4, np.uint64), (8, np.uint64), (16, np.uint64), (32, np.uint64), (8, np.uint32),
                         (16, np.uint32), (32, np.uint32), (64, np.uint32)]:
            for n in [1, b - 1, b, b + 1, 7 * b + 5, 65_537, 1_000_003]:
                if n < 1:
                    continue
                keys = data.sorted_keys_np(n, 1, 16 if dtype == np.uint64 else 3, n + b, dtype)
                tree = O.permute("btree", keys, b)
                Q = data.queries_np(keys, 20_000, 0.5, n + 2)
                Q = np.concatenate([Q, keys[:1] - 1 if keys[0] > 0 else keys[:1], keys[-1:] + 1]).astype(dtype)
                assert np.array_equal(gpu_answers("btree", tree, Q, b), O.search("btree", tree, Q, b)), \
                    (variant, b, n, dtype)
    finally:
        L.tl_debug_set_query_variant(0)


@pytest.mark.parametrize("variant", [0, 3, 4])
@pytest.mark.parametrize("layout", ["mveb", "veb"])
def test_veb_query_kernel_forms(variant, layout):
    """Each vEB descent form gives the oracle's answers, perfect and
    non-perfect trees, u32 and u64: one descent per thread (default), two or
    four in lock-step (3, 4)."""
    import ctypes as C
    L = T.lib()
    L.tl_debug_set_query_variant.argtypes = [C.c_int]
    L.tl_debug_set_query_variant(variant)
    try:
        for dtype in (np.uint32, np.uint64):
            for n in [1, 2, 3, 7, 100, 4095, 65536, 1_000_003, 2**21 - 1]:
                keys = data.sorted_keys_np(n, 1, 3, n + 11, dtype)
                tree = O.permute(layout, keys, 16)
                Q = data.queries_np(keys, 20_000, 0.5, n + 12)
                Q = np.concatenate([Q, keys[:1] - 1 if keys[0] > 0 else keys[:1], keys[-1:] + 1]).astype(dtype)
                assert np.array_equal(gpu_answers(layout, tree, Q), O.search(layout, tree, Q, 16)), \
                    (variant, layout, n, dtype)
    finally:
        L.tl_debug_set_query_variant(0)


@pytest.mark.parametrize("layout,n,kb,q", [("mveb", 2**24 - 1, 4, 2**23), ("bst", 2**23 - 1, 8, 2**23),
                                           ("bst", 2**25 - 1, 8, 2**23), ("mveb", 2**24 - 1, 4, 2**27)])
def test_grouped_queries_at_16_and_20_bucket_bits(layout, n, kb, q):
    """Batches large enough for 16 bucket bits (2^23 queries: four passes) and
    for 20 (2^27: five passes), grouped by default, equal the same batches
    searched as given (variant 19); the 256 MB BST takes the grouped shape
    with the smaller pinned prefix."""
    import ctypes as C

    import torch
    L = T.lib()
    L.tl_debug_set_query_variant.argtypes = [C.c_int]
    keys = data.sorted_keys_torch(n, 1, 3 if kb == 4 else 16, n % 1000 + 3, kb)
    tree = keys.clone()
    T.permute(layout, tree, 16)
    tabs = T.VebTablesDevice(n, "cuda", standard=layout == "veb") if layout != "bst" else None
    Q = data.queries_torch(keys, q, 0.5, 11)
    got = torch.empty(q, dtype=torch.int64, device="cuda")
    exp = torch.empty_like(got)
    T.query(layout, tree, Q, got, 16, tables=tabs)  # default: grouped at these sizes
    try:
        L.tl_debug_set_query_variant(19)
        T.query(layout, tree, Q, exp, 16, tables=tabs)
    finally:
        L.tl_debug_set_query_variant(0)
    assert torch.equal(got, exp), (layout, n, q)
    hit = got != n
    assert torch.equal(tree[got[hit]], Q[hit])


@pytest.mark.parametrize("layout,n,kb", [("mveb", 2**24 - 1, 4), ("mveb", 20_000_003, 4), ("veb", 2**22 - 1, 8),
                                         ("bst", 2**23 - 1, 8), ("bst", 9_000_001, 4)])
def test_partitioned_queries_match_unpartitioned(layout, n, kb):
    """A batch searched grouped by value (a partition of the batch's value
    range into up to 2^20 buckets, 4 bits a pass, answers written back through the carried
    index, vEB descents in 256-thread blocks; variant 20 forces it at any
    size) equals the batch searched as
    given (variant 19) for batch lengths around the partition's 4096-entry
    tiles, with duplicates and a batch of one value; every hit names its key's
    slot and every miss is a key absent from the sorted keys."""
    import ctypes as C

    import torch
    L = T.lib()
    L.tl_debug_set_query_variant.argtypes = [C.c_int]
    keys = data.sorted_keys_torch(n, 1, 3 if kb == 4 else 16, n % 1000 + 1, kb)
    tree = keys.clone()
    T.permute(layout, tree, 16)
    tabs = T.VebTablesDevice(n, "cuda", standard=layout == "veb") if layout != "bst" else None
    Qall = data.queries_torch(keys, 2**21, 0.5, 7)
    Qall[:3] = keys[0]  # duplicates and the smallest key
    for q in [1, 2, 4095, 4096, 4097, 100_003, 2**21]:
        Q = Qall[:q].clone()
        got = torch.empty(q, dtype=torch.int64, device="cuda")
        exp = torch.empty_like(got)
        try:
            L.tl_debug_set_query_variant(20)
            T.query(layout, tree, Q, got, 16, tables=tabs)
            L.tl_debug_set_query_variant(19)
            T.query(layout, tree, Q, exp, 16, tables=tabs)
        finally:
            L.tl_debug_set_query_variant(0)
        assert torch.equal(got, exp), (layout, n, q)
        hit = got != n
        assert torch.equal(tree[got[hit]], Q[hit])
        pos = torch.searchsorted(keys, Q).clamp_max(n - 1)
        assert torch.equal(keys[pos] == Q, hit)
    Q = torch.full((5000,), int(keys[n // 2].item()), dtype=keys.dtype, device="cuda")  # one value
    got = torch.empty(5000, dtype=torch.int64, device="cuda")
    try:
        L.tl_debug_set_query_variant(20)
        T.query(layout, tree, Q, got, 16, tables=tabs)
    finally:
        L.tl_debug_set_query_variant(0)
    assert torch.equal(tree[got], Q)


def _check_answers(tree, sorted_keys, Q, ans):
    """Hits name a position that holds the key, misses (answer n) are absent;
    unsigned values."""
    import torch
    n = tree.numel()
    mask = (1 << (8 * tree.element_size())) - 1 if tree.element_size() == 4 else -1
    ks, q = sorted_keys.to(torch.int64) & mask, Q.to(torch.int64) & mask
    at = torch.searchsorted(ks, q).clamp_max(n - 1)
    present = ks[at] == q
    hit = ans != n
    assert torch.equal(hit, present)
    assert bool(((ans >= 0) & (ans <= n)).all())
    assert torch.equal(tree[ans[hit]], Q[hit])


@pytest.mark.parametrize("layout", ["mveb", "veb"])
@pytest.mark.parametrize("kb", [4, 8])
@pytest.mark.parametrize("n,skip", [(1, 0), (2, 1), (15, 3), (16, 5), (31, 0), (255, 1), (256, 7), (4095, 0), (4096, 3),
                                    (65535, 1), (65536, 6), (1_000_003, 1), (2**22 - 1, 5)])
def test_veb_pieces_unaligned_layouts(layout, kb, n, skip):
    """Descents piece by piece: sizes around the recursion's splits, a layout
    that starts `skip` keys into its allocation (pieces cross 32-byte sectors at
    every phase and may not be read past either end), batches of one query, of
    one value, around a block's chunk and over several rounds of chunks."""
    import torch
    dt = torch.int64 if kb == 8 else torch.int32
    keys = data.sorted_keys_torch(n, 1, 3, n + skip, kb)
    buf = torch.empty(n + skip, dtype=dt, device="cuda")
    tree = buf[skip:]
    tree.copy_(keys)
    T.permute(layout, tree)
    tabs = T.VebTablesDevice(n, "cuda", standard=layout == "veb")
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    top = int(keys[-1].item())
    for q in [1, 147, 149, 16385, 148 * 16384 + 5]:
        Q = torch.randint(0, top + 3, (q,), generator=g, device="cuda", dtype=torch.int64).to(dt)
        ans = torch.full((q,), -7, dtype=torch.int64, device="cuda")
        T.query(layout, tree, Q, ans, tables=tabs)
        _check_answers(tree, keys, Q, ans)
    Q = torch.full((20_000,), top, dtype=dt, device="cuda")
    Q[::1000] = 0
    ans = torch.empty(20_000, dtype=torch.int64, device="cuda")
    T.query(layout, tree, Q, ans, tables=tabs)
    _check_answers(tree, keys, Q, ans)


def test_veb_pieces_with_64_bit_positions():
    """2^31 + 3 keys: positions and path indices past 32 bits."""
    import torch
    n = 2**31 + 3
    keys = torch.arange(n, device="cuda", dtype=torch.int64).to(torch.int32)  # 0 .. n - 1 as uint32
    T.permute("mveb", keys)
    tabs = T.VebTablesDevice(n, "cuda")
    Q64 = torch.randint(0, n + 1000, (1 << 20,), device="cuda", dtype=torch.int64)
    Q64[:3] = torch.tensor([0, n - 1, n], device="cuda")
    ans = torch.empty(1 << 20, dtype=torch.int64, device="cuda")
    T.query("mveb", keys, Q64.to(torch.int32), ans, tables=tabs)
    hit = ans != n
    assert torch.equal(hit, Q64 < n)
    assert torch.equal(keys[ans[hit]], Q64[hit].to(torch.int32))


@pytest.mark.parametrize("kb,b", [(8, 8), (8, 16), (8, 32), (4, 16), (4, 32), (4, 64)])
def test_btree_top_levels_in_shared_memory(kb, b):
    """The B-tree form with its top levels in shared memory (variant 9 at any
    size; the default from 2^20 queries): trees with one level up to several
    below the top, a partial last leaf, evenly spread and skewed keys (most top
    keys in one bin), all keys equal in their high bits, queries for every key
    of the top, below the first, past the last."""
    import ctypes as C

    import torch
    L = T.lib()
    L.tl_debug_set_query_variant.argtypes = [C.c_int]
    g = torch.Generator(device="cuda")
    g.manual_seed(b + kb)
    dt = torch.int64 if kb == 8 else torch.int32
    for n in [b, b + 1, (b + 1) ** 2 - 1, (b + 1) ** 2 + b // 2, 50_021, 1_000_003]:
        even = data.sorted_keys_torch(n, 1, 3, n, kb).to(torch.int64)
        rank = torch.arange(n, device="cuda", dtype=torch.float64)
        skew = even + (torch.exp2(rank / n * 24 + 6)).to(torch.int64) if kb == 4 else \
            even + (torch.exp2(rank / n * 60)).to(torch.int64)
        for keys in (even, skew.clamp_max(2**31 - n) + torch.arange(n, device="cuda") if kb == 4 else skew):
            tree = keys.to(dt).clone()
            T.permute("btree", tree, b)
            Q = torch.cat([tree[:min(n, 5000)].to(torch.int64), keys[torch.randint(0, n, (20_000,), generator=g,
                                                                                   device="cuda")],
                           keys[torch.randint(0, n, (20_000,), generator=g, device="cuda")] + 1, keys[:1] - 1,
                           keys[-1:] + 1, torch.zeros(1, dtype=torch.int64, device="cuda")]).to(dt)
            got = torch.full((Q.numel(),), -7, dtype=torch.int64, device="cuda")
            L.tl_debug_set_query_variant(9)
            try:
                T.query("btree", tree, Q, got, b)
            finally:
                L.tl_debug_set_query_variant(0)
            _check_answers(tree, keys.to(dt), Q, got)
    q = (1 << 20) + 77  # the default route
    Q = keys[torch.randint(0, n, (q,), generator=g, device="cuda")].to(dt) + 1
    got = torch.full((q,), -7, dtype=torch.int64, device="cuda")
    T.query("btree", tree, Q, got, b)
    _check_answers(tree, keys.to(dt), Q, got)


@pytest.mark.parametrize("kb", [4, 8])
@pytest.mark.parametrize("n,skip", [(1, 0), (2, 1), (3, 0), (4094, 1), (4095, 0), (4096, 3), (8191, 0), (8192, 1),
                                    (65_537, 1), (2**20 - 1, 0), (2_000_003, 3)])
def test_bst_ordered_chunks(kb, n, skip):
    """BST descents over chunks ordered by value: trees within, just past and well
    past the levels in shared memory, unaligned layouts, batches of one query, of
    one value, around a block's chunk and over several rounds; the grouped route
    (variant 20) on the same batches."""
    import ctypes as C

    import torch
    L = T.lib()
    L.tl_debug_set_query_variant.argtypes = [C.c_int]
    dt = torch.int64 if kb == 8 else torch.int32
    keys = data.sorted_keys_torch(n, 1, 3, n + skip, kb)
    buf = torch.empty(n + skip, dtype=dt, device="cuda")
    tree = buf[skip:]
    tree.copy_(keys)
    T.permute("bst", tree)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    top = int(keys[-1].item())
    for q in [1, 295, 297, 4097, 296 * 4096 + 5]:
        Q = torch.randint(0, top + 3, (q,), generator=g, device="cuda", dtype=torch.int64).to(dt)
        for variant in (0, 20):
            ans = torch.full((q,), -7, dtype=torch.int64, device="cuda")
            L.tl_debug_set_query_variant(variant)
            try:
                T.query("bst", tree, Q, ans)
            finally:
                L.tl_debug_set_query_variant(0)
            _check_answers(tree, keys, Q, ans)
    Q = torch.full((20_000,), top, dtype=dt, device="cuda")
    Q[::1000] = 0
    ans = torch.empty(20_000, dtype=torch.int64, device="cuda")
    T.query("bst", tree, Q, ans)
    _check_answers(tree, keys, Q, ans)


def test_bst_with_64_bit_nodes():
    """2^31 + 3 keys: node numbers past 32 bits, in chunks and grouped."""
    import torch
    n = 2**31 + 3
    keys = torch.arange(n, device="cuda", dtype=torch.int64).to(torch.int32)  # 0 .. n - 1 as uint32
    T.permute("bst", keys)
    for q in (1 << 20, (1 << 22) + 1):
        Q64 = torch.randint(0, n + 1000, (q,), device="cuda", dtype=torch.int64)
        Q64[:3] = torch.tensor([0, n - 1, n], device="cuda")
        ans = torch.empty(q, dtype=torch.int64, device="cuda")
        T.query("bst", keys, Q64.to(torch.int32), ans)
        hit = ans != n
        assert torch.equal(hit, Q64 < n)
        assert torch.equal(keys[ans[hit]], Q64[hit].to(torch.int32))


@pytest.mark.parametrize("kb", [4, 8])
@pytest.mark.parametrize("n,skip", [(1, 0), (2, 1), (3, 0), (31, 3), (4096, 1), (4097, 0), (8193, 1), (1_000_003, 5)])
def test_sorted_array_ordered_chunks(kb, n, skip):
    """Binary search over chunks ordered by value: arrays within and past the
    pinned probes, unaligned arrays, batches on either side of the form's line and
    over several rounds of chunks, a batch of one value."""
    import torch
    dt = torch.int64 if kb == 8 else torch.int32
    keys = data.sorted_keys_torch(n, 1, 3, n + skip, kb)
    buf = torch.empty(n + skip, dtype=dt, device="cuda")
    arr = buf[skip:]
    arr.copy_(keys)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    top = int(keys[-1].item())
    for q in [1, (1 << 16) - 1, 1 << 16, 296 * 4096 + 5]:
        Q = torch.randint(0, top + 3, (q,), generator=g, device="cuda", dtype=torch.int64).to(dt)
        ans = torch.full((q,), -7, dtype=torch.int64, device="cuda")
        T.query("sorted", arr, Q, ans)
        _check_answers(arr, keys, Q, ans)
    Q = torch.full((70_000,), top, dtype=dt, device="cuda")
    ans = torch.empty(70_000, dtype=torch.int64, device="cuda")
    T.query("sorted", arr, Q, ans)
    _check_answers(arr, keys, Q, ans)


@pytest.mark.parametrize("layout", ["mveb", "veb"])
@pytest.mark.parametrize("dtype", [np.uint64, np.uint32])
@pytest.mark.parametrize("n", [(1 << 22) - 1, 1 << 22, 5_000_011])
def test_duplicate_keys_on_either_side_of_the_veb_forms(layout, dtype, n):
    """The same for the two forms of the vEB search, which meet equal keys in the
    pieces (from 2^22 keys) or at the path's left turns."""
    keys = _with_duplicates(n, n, dtype)
    tree = O.permute(layout, keys, 16)
    for q in (1000, (1 << 17) + 77):
        Q = data.queries_np(keys, q, 0.7, 3)
        Q[:3] = keys[0], keys[-1], keys[-1] + 1
        assert np.array_equal(gpu_answers(layout, tree, Q), O.search(layout, tree, Q)), q


def _with_duplicates(n, seed, dtype):
    """n sorted keys, runs of one value geometrically long."""
    rng = np.random.default_rng(seed)
    return np.repeat(np.cumsum(rng.integers(1, 5, n)).astype(dtype), rng.geometric(0.3, n))[:n].copy()


@pytest.mark.parametrize("layout,b", [("bst", 1), ("btree", 8), ("btree", 16), ("btree", 32), ("btree", 5), ("mveb", 0),
                                      ("veb", 0)])
@pytest.mark.parametrize("dtype", [np.uint64, np.uint32])
def test_duplicate_keys_answer_the_first_on_the_path(layout, b, dtype):
    """Equal keys: the answer is the one that the search from the root meets
    first, as the oracle's, for small batches and for those whose top levels are
    searched in shared memory; one value all over, and several divisions."""
    for n in (2, 31, 100, 4095, 65_537, 1_000_003):
        for keys in (_with_duplicates(n, n, dtype), np.full(n, 7, dtype)):
            tree = O.permute(layout, keys, b or 16)
            for q in (5000, (1 << 20) + 77):
                Q = data.queries_np(keys, q, 0.7, 3)
                Q[:3] = keys[0], keys[-1], keys[-1] + 1
                assert np.array_equal(gpu_answers(layout, tree, Q, b or 16), O.search(layout, tree, Q, b or 16)), \
                    (layout, b, n, q)


@pytest.mark.parametrize("layout", ["mveb", "bst"])
def test_threads_query_with_different_batches(layout):
    """Host threads whose launches of one kernel ask for different amounts of
    shared memory, in tight loops through the C entry: none refuses another's."""
    import ctypes as C
    import threading

    import torch
    n, L = 2**20 + 5, T.lib()
    keys = data.sorted_keys_torch(n, 1, 16, 3, 8)
    batches = [keys[torch.randint(0, n, (q,), device="cuda")] for q in (1 << 20, 1 << 10, 1 << 10, 1 << 10)]
    answers = [torch.empty_like(Q) for Q in batches]
    streams = [torch.cuda.Stream() for _ in batches]
    T.permute(layout, keys)
    tabs = T.VebTablesDevice(n)
    calls = []
    for Q, ans, st in zip(batches, answers, streams):
        tail = (C.c_void_p(Q.data_ptr()), C.c_uint64(Q.numel()), C.c_void_p(ans.data_ptr()), C.c_void_p(st.cuda_stream),
                None)
        calls.append((C.c_void_p(keys.data_ptr()), C.c_uint64(n)) + tail if layout == "bst" else
                     (C.c_void_p(keys.data_ptr()), C.c_void_p(tabs.tables.data_ptr()), C.c_void_p(tabs.idx.data_ptr()),
                      C.c_void_p(tabs.table_idx.data_ptr()), C.c_uint64(n), C.c_uint32(tabs.d),
                      C.c_uint32(tabs.num_tables)) + tail)
    fn = L.tl_query_bst_u64 if layout == "bst" else L.tl_query_veb_nonperfect_u64
    torch.cuda.synchronize()
    refused, done = [0] * len(calls), threading.Event()

    def work(w):
        for _ in range(200):
            if done.is_set():
                break
            for _ in range(100):
                refused[w] += fn(*calls[w]) != 0
            streams[w].synchronize()
        if w == 0:
            done.set()

    threads = [threading.Thread(target=work, args=(w,)) for w in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert refused == [0] * len(calls)
    for Q, ans in zip(batches, answers):
        assert torch.equal(keys[ans], Q)


@pytest.mark.parametrize("layout", ["mveb", "veb", "bst"])
@pytest.mark.parametrize("dtype", [np.uint64, np.uint32])
@pytest.mark.parametrize("last", [0, 1])
def test_small_layouts_and_the_largest_key(layout, dtype, last):
    """Layouts held whole in shared memory, perfect and of several divisions, on
    either side of what is held at each batch size; with and without the type's
    largest value among the keys, queried for it."""
    top = int(np.iinfo(dtype).max)
    for n in (1, 2, 3, 5, 30, 31, 255, 1000, 2047, 2048, 4101, 8191, 8192, 16383, 16384):
        keys = data.sorted_keys_np(n, 1, 5, n, dtype)
        if last:
            keys[-1] = top
        tree = O.permute(layout, keys, 16)
        for q in (1500, (1 << 17) + 3):
            Q = data.queries_np(keys, q, 0.5, n + 1)
            Q[:5] = 0, top, top - 1, keys[0], keys[-1]
            Q[5:40] = top
            assert np.array_equal(gpu_answers(layout, tree, Q), O.search(layout, tree, Q)), (layout, n, q)


def test_bst_grouping_line_over_4_gb():
    """Either side of the batch size from which a 4 GB BST's queries are grouped."""
    import torch
    n = 2**30 - 1
    keys = torch.arange(1, n + 1, device="cuda", dtype=torch.int32) * 2
    tree = keys.clone()
    T.permute("bst", tree)
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    for q in ((3 << 20) - 1, 3 << 20):
        Q = torch.randint(0, 2**31 - 1, (q,), generator=g, device="cuda", dtype=torch.int32)
        ans = torch.full((q,), -7, dtype=torch.int64, device="cuda")
        T.query("bst", tree, Q, ans)
        hit = ans != n
        assert torch.equal(hit, (Q % 2 == 0) & (Q > 0))
        assert torch.equal(tree[ans[hit]], Q[hit])
