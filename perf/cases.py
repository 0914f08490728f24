"""The calls a program makes of this library, as timed cases: building a layout
from sorted keys, taking a layout back to sorted order, answering query batches,
and the batched and learned modes, each through the Python entry points of
tree_layouts.

A case is a dict of plain values:

- do "build": tree_layouts.permute of n sorted keys into `layout`;
- do "restore": tree_layouts.unpermute of a layout of n keys;
- do "lookup": tree_layouts.query of q queries over a layout (or the sorted keys);
- do "batch-build" / "batch-lookup": a BatchPlan's permute and query over `num`
  arrays of log-uniform sizes in [2^lo, 2^hi];
- do "learned": the learned-start B-tree query over skewed keys, Zipf queries.

The outputs are words moved and integer positions, so there is no rounding and
no exact() here: two correct programs give equal outputs.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tree-layouts_b200"))

import tree_layouts as T  # noqa: E402
from tree_layouts import batched, data, learned  # noqa: E402


def listed():
    return [
        # a small index rebuilt in a serving loop: latency and launches count
        dict(name="build-bst-1m-u64", do="build", layout="bst", n=2**20 - 1, b=1, kb=8),
        # the benchmark's index: half a billion 8-byte keys, 128-byte nodes
        dict(name="build-btree-500m-u64", do="build", layout="btree", n=500_000_000, b=16, kb=8),
        # a cache-oblivious index whose size is no power of two, 4-byte keys
        dict(name="build-mveb-300m-u32", do="build", layout="mveb", n=300_000_000, b=1, kb=4),
        # indexes taken apart again, to merge new keys in or to scan in order
        dict(name="restore-btree-60m-u64", do="restore", layout="btree", n=60_000_000, b=8, kb=8),
        dict(name="restore-mveb-300m-u32", do="restore", layout="mveb", n=300_000_000, b=1, kb=4),
        # one request's lookups against a small index
        dict(name="lookup-btree-16k-of-1m", do="lookup", layout="btree", n=1_000_003, b=16, kb=8, q=16384),
        # bulk joins: a large batch against the benchmark's index
        dict(name="lookup-btree-128m-of-500m", do="lookup", layout="btree", n=500_000_000, b=16, kb=8, q=2**27),
        # a perfect BST and a ragged vEB probed by medium and large batches
        dict(name="lookup-bst-16m-of-134m", do="lookup", layout="bst", n=2**27 - 1, b=1, kb=4, q=2**24),
        dict(name="lookup-mveb-64m-of-300m", do="lookup", layout="mveb", n=300_000_000, b=1, kb=4, q=2**26),
        # many independent indexes of uneven sizes (one per tenant or partition)
        dict(name="batch-build-1024", do="batch-build", num=1024, lo=10.0, hi=22.0, b=8),
        dict(name="batch-lookup-16m-in-1024", do="batch-lookup", num=1024, lo=10.0, hi=22.0, b=8, q=2**24),
        # popular keys of a skewed key set through the learned start
        dict(name="learned-64m-of-134m", do="learned", n=2**27, b=16, q=2**26, leaves=2**18),
    ]


def _log_uniform(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    do = rng.choice(["build"] * 4 + ["restore"] * 2 + ["lookup"] * 5 + ["batch-build", "batch-lookup", "learned"])
    if do in ("batch-build", "batch-lookup"):
        lo = rng.uniform(6.0, 12.0)
        hi = lo + rng.uniform(2.0, 10.0)
        c = dict(do=do, num=_log_uniform(rng, 16, 1025), lo=lo, hi=hi, b=rng.choice([4, 8, 8, 16]))
        if do == "batch-lookup":
            c["q"] = _log_uniform(rng, 2**12, 2**24)
        return c
    if do == "learned":
        n = _log_uniform(rng, 2**20, 2**27)
        return dict(do=do, n=n, b=rng.choice([8, 16, 16]), q=_log_uniform(rng, 2**14, 2**26),
                    leaves=2 ** max(12, n.bit_length() - 10))
    kb = rng.choice([4, 8])
    layout = rng.choice(["bst", "btree", "btree", "mveb", "veb"] + (["sorted"] if do == "lookup" else []))
    n = _log_uniform(rng, 2**12, 500_000_001)
    if layout in ("bst", "mveb", "veb") and rng.random() < 0.4:
        n = 2 ** (n.bit_length() - 1) - 1  # a perfect tree
    b = rng.choice([3, 4, 8, 16, 16, 32]) if layout == "btree" else 1
    c = dict(do=do, layout=layout, n=n, b=b, kb=kb)
    if do == "lookup":
        c["q"] = _log_uniform(rng, 2**10, 2**25)
    return c


def _sorted_keys(n, kb, seed):
    # 4-byte keys: the widest uniform gaps whose sum stays below 2^32
    gap = 64 if kb == 8 else max(1, min(64, int(1.98 * 2**32 / n) - 2))
    return data.sorted_keys_torch(n, 1, gap, seed, kb)


def _batch_sizes(case):
    # the sizes belong to the case; the keys in the arrays come from the seed
    return batched.batch_sizes_np(case["num"], case["lo"], case["hi"], case["num"])


def prepare(case, seed):
    do = case["do"]
    if do in ("batch-build", "batch-lookup"):
        keys, offsets = data.batch_keys_torch(_batch_sizes(case), 64, seed)
        plan = batched.BatchPlan(offsets, b=case["b"], key_bytes=8)
        s = dict(do=do, plan=plan, keys=keys)
        if do == "batch-lookup":
            s["queries"], s["inst"] = data.batch_queries_torch(keys, offsets, case["q"], 0.5, seed + 1)
            plan.permute(keys)
            s["answers"] = torch.empty(case["q"], dtype=torch.int64, device="cuda")
        return s
    if do == "learned":
        keys = data.skewed_keys_torch(case["n"], seed, oversample=1.12)
        model, leaves = learned.train(keys, num_leaves=case["leaves"], steps=300, seed=1 + seed)
        queries = data.zipf_queries_torch(keys, case["q"], seed + 1)
        T.permute("btree", keys, case["b"])
        return dict(do=do, keys=keys, model=model, leaves=leaves, queries=queries, b=case["b"],
                    answers=torch.empty(case["q"], dtype=torch.int64, device="cuda"))
    layout, b, n = case["layout"], case["b"], case["n"]
    keys = _sorted_keys(n, case["kb"], seed)
    s = dict(do=do, layout=layout, b=b, keys=keys)
    if do == "lookup":
        s["queries"] = data.queries_torch(keys, case["q"], 0.5, seed + 1)
        s["answers"] = torch.empty(case["q"], dtype=torch.int64, device="cuda")
        s["tables"] = T.VebTablesDevice(n, standard=layout == "veb") if layout in ("mveb", "veb") else None
    if do == "restore" or do == "lookup" and layout != "sorted":
        T.permute(layout, keys, b)
    return s


def run(s):
    do = s["do"]
    if do == "build":  # words moved in place: every pass moves the same words, sorted or not
        T.permute(s["layout"], s["keys"], s["b"])
        return s["keys"]
    if do == "restore":
        T.unpermute(s["layout"], s["keys"], s["b"])
        return s["keys"]
    if do == "lookup":
        T.query(s["layout"], s["keys"], s["queries"], s["answers"], s["b"], tables=s["tables"])
        return s["answers"]
    if do == "batch-build":
        s["plan"].permute(s["keys"])
        return s["keys"]
    if do == "batch-lookup":
        s["plan"].query(s["keys"], s["queries"], s["inst"], s["answers"])
        return s["answers"]
    learned.query(s["keys"], s["model"], s["leaves"], s["queries"], s["answers"], s["b"])
    return s["answers"]


def work(case):
    """Bytes of one pass.  A build or restore reads and writes each key once; a
    lookup reads its queries, writes its 8-byte answers and reads at least one
    32-byte sector of the layout per query, or the whole layout once where that
    is less."""
    do = case["do"]
    if do in ("batch-build", "batch-lookup"):
        keys = int(_batch_sizes(case).sum())
        if do == "batch-build":
            return {"bytes": 2 * 8 * keys, "flops": 0}
        return {"bytes": case["q"] * (8 + 4 + 8) + min(keys * 8, case["q"] * 32), "flops": 0}
    kb = case.get("kb", 8)
    if do in ("build", "restore"):
        return {"bytes": 2 * case["n"] * kb, "flops": 0}
    return {"bytes": case["q"] * (kb + 8) + min(case["n"] * kb, case["q"] * 32), "flops": 0}
