"""Workloads of the batched B+tree, for timing and for comparing outputs.

Each case is one call (or one write epoch) that a program makes on a loaded
tree: point searches from a thousand keys to a headline batch, batch sets in a
captured plan, host-buffer searches, both range forms, write epochs of serving
and of bulk size, and the bulk load itself.  Keys are 63-bit and either
scattered over the key space (hashes, the generator's default) or dense
(auto-increment ids); values are arbitrary non-negative integers; inputs come
from the seed alone and are made on the GPU.
"""
import math

import torch

from harmonia_b200 import BPlusTree

MAX_KEY = 2**63 - 1
MASK63 = 2**63 - 1


def listed():
    return [
        # one small request of a latency-bound caller on a small index
        dict(name="search_1k", kind="search", n_keys=1 << 20, n=1000, hit=0.9, dist="uniform", fanout=64, leaf_cap=16,
             keys="scattered"),
        # an ordinary ragged batch: too small for any grouping of the queries to pay
        dict(name="search_100k", kind="search", n_keys=1 << 24, n=100_003, hit=0.9, dist="uniform", fanout=64,
             leaf_cap=16, keys="scattered"),
        # a large ragged batch against a much larger tree (fewer queries than leaves)
        dict(name="search_1m", kind="search", n_keys=1 << 26, n=1_048_583, hit=0.9, dist="uniform", fanout=64,
             leaf_cap=16, keys="scattered"),
        # the benchmark's batch: 2^24 uniform queries, 90 % hits, 2^26 keys, fanout 64
        dict(name="search_16m", kind="search", n_keys=1 << 26, n=1 << 24, hit=0.9, dist="uniform", fanout=64,
             leaf_cap=16, keys="scattered"),
        # skewed reads on the other node shape: fanout 128, 64-key leaves
        dict(name="search_zipf_wide", kind="search", n_keys=1 << 24, n=6_000_011, hit=1.0, dist="zipf", fanout=128,
             leaf_cap=64, keys="scattered"),
        # 64 batches of uneven size, half uniform and half Zipf, replayed as one captured plan
        dict(name="plan_uneven", kind="plan", n_keys=1 << 25, n=12_000_000, batches=64, hit=0.9, fanout=64,
             leaf_cap=16, keys="scattered"),
        # a program with its queries in page-locked host memory
        dict(name="search_host", kind="host", n_keys=1 << 24, n=4_000_037, hit=0.9, dist="uniform", fanout=64,
             leaf_cap=16, keys="scattered", pinned=True),
        # the benchmark's scans: the first 1-256 records from each start key
        dict(name="range_1m", kind="range", n_keys=1 << 26, n=1 << 20, longest=256, fanout=64, leaf_cap=16,
             keys="scattered"),
        # inclusive [start, end] windows of about 40 records, result size not known beforehand
        dict(name="between_50k", kind="between", n_keys=1 << 22, n=50_021, mean=40, fanout=64, leaf_cap=16,
             keys="scattered"),
        # one request's writes in a serving loop: expire a few keys, then store a few hundred
        dict(name="write_256", kind="write", n_keys=1 << 22, n=256, new=0.25, leaf_fill=12, fanout=64, leaf_cap=16,
             keys="scattered"),
        # the benchmark's update epoch: 4096K keys, 5 % of them new; the expired ones go first
        dict(name="write_4m", kind="write", n_keys=1 << 26, n=4096 * 1000, new=0.05, leaf_fill=12, fanout=64,
             leaf_cap=16, keys="scattered"),
        # building an index from unsorted pairs
        dict(name="load_16m", kind="load", n_keys=1 << 24, leaf_fill=16, fanout=64, leaf_cap=16, keys="scattered"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "search", "search", "plan", "host", "range", "between", "write", "write", "load"])
    c = dict(kind=kind, n_keys=_log_int(rng, 1 << 17, 1 << 26), fanout=rng.choice([64, 64, 128]),
             leaf_cap=rng.choice([16, 16, 16, 64]), keys=rng.choice(["scattered", "scattered", "dense"]))
    if kind in ("search", "host"):
        c.update(n=_log_int(rng, 500, 1 << 24) if kind == "search" else _log_int(rng, 1 << 15, 1 << 22),
                 hit=rng.choice([0.5, 0.9, 1.0]), dist=rng.choice(["uniform", "uniform", "zipf"]))
        if kind == "host":
            c.update(pinned=rng.choice([True, False]))
    elif kind == "plan":
        c.update(n=_log_int(rng, 1 << 17, 12_000_000), batches=rng.randint(3, 100), hit=rng.choice([0.5, 0.9, 1.0]))
    elif kind == "range":
        c.update(n=_log_int(rng, 1000, 1 << 20), longest=rng.randint(2, 256))
    elif kind == "between":
        c.update(n=_log_int(rng, 1000, 1 << 19), mean=rng.randint(2, 128))
    elif kind == "write":
        most = min(4096 * 1000, c["n_keys"] // 8)
        c.update(n=_log_int(rng, 32, most), new=rng.choice([0.05, 0.1, 0.25]), leaf_fill=c["leaf_cap"] * 3 // 4)
    else:
        c.update(n_keys=_log_int(rng, 1 << 17, 1 << 24), leaf_fill=rng.choice([c["leaf_cap"], c["leaf_cap"] * 3 // 4]))
    return c


# ---- inputs -----------------------------------------------------------------


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _mix63(x):
    """A bijection of [0, 2^63): multiplications by odd numbers and xor-shifts modulo 2^63."""
    x = (x * -7046029254386353131) & MASK63
    x = x ^ (x >> 31)
    x = (x * -4658895280553007687) & MASK63
    return x ^ (x >> 29)


def _gen(seed, salt):
    g = torch.Generator(device=_device())
    g.manual_seed((seed * 1_000_003 + salt) % (1 << 62))
    return g


def _key_of(case, seed, i):
    """Key number i: numbers below n_keys are loaded, the ones from n_keys on are not (until they are upserted)."""
    if case["keys"] == "dense":
        # loaded ids are even, the others odd
        n = case["n_keys"]
        return torch.where(i < n, 2 * i, 2 * (i - n) + 1) + 1_000_000 * (seed % 1000)
    return _mix63(i + (seed % 1000) * (1 << 40))


def _values(g, n):
    return torch.randint(0, MASK63, (n,), generator=g, device=_device(), dtype=torch.int64)


def _loaded(case, seed):
    """The pairs a program loads, in no order."""
    n = case["n_keys"]
    keys = _key_of(case, seed, torch.arange(n, device=_device(), dtype=torch.int64))
    g = _gen(seed, 1)
    if case["keys"] == "dense":
        keys = keys[torch.randperm(n, generator=g, device=_device())]
    return keys, _values(g, n)


def _numbers(g, n, dist, n_keys):
    """n key numbers below n_keys: uniform, or Zipf-like with exponent 0.99 (rank = number)."""
    u = torch.rand(n, generator=g, device=_device(), dtype=torch.float64)
    if dist == "zipf":
        e = 1.0 - 0.99
        u = ((u * (float(n_keys) ** e - 1.0) + 1.0) ** (1.0 / e) - 1.0) / n_keys
    return (u * n_keys).to(torch.int64).clamp_(0, n_keys - 1)


def _queries(case, seed, n, dist, salt):
    g = _gen(seed, salt)
    i = _numbers(g, n, dist, case["n_keys"])
    miss = torch.rand(n, generator=g, device=_device()) >= case["hit"]
    return _key_of(case, seed, torch.where(miss, i + case["n_keys"], i))


def _batch_sizes(case, seed):
    """`batches` sizes that add up to n, spread over a factor of about a thousand."""
    b = case["batches"]
    w = torch.rand(b, generator=torch.Generator().manual_seed(seed + 17)).double()
    w = torch.exp(w * math.log(1000.0))
    sizes = (w / w.sum() * case["n"] * 0.999).to(torch.int64).clamp_(min=1)
    sizes[0] += case["n"] - int(sizes.sum())
    return sizes.tolist()


def _range_inputs(case, seed):
    """Starts (a stored key, or one just below it) and lengths or ends; the lengths of any seed are the same ones in another order."""
    g = _gen(seed, 3)
    n, d = case["n"], _device()
    keys = torch.sort(_loaded(case, seed)[0])[0]
    longest = case["longest"] if case["kind"] == "range" else 2 * case["mean"] - 1
    length = (torch.arange(n, device=d) % longest + 1)[torch.randperm(n, generator=g, device=d)]
    first = _numbers(g, n, "uniform", case["n_keys"] - longest)
    start = keys[first] - torch.randint(0, 2, (n,), generator=g, device=d)
    if case["kind"] == "range":
        return start, length.to(torch.int32)
    return start, keys[first + length - 1] + torch.randint(0, 2, (n,), generator=g, device=d)


def _write_batch(case, seed):
    """(new keys, all keys, their values): new keys once, the others drawn from the loaded ones, in no order."""
    g = _gen(seed, 4)
    n = case["n"]
    fresh_n = max(1, int(n * case["new"]))
    # dense ids: the new ones spread over the whole range of ids
    pick = torch.randperm(case["n_keys"], generator=g, device=_device())[:fresh_n]
    fresh = _key_of(case, seed, pick + case["n_keys"])
    old = _key_of(case, seed, _numbers(g, n - fresh_n, "uniform", case["n_keys"]))
    keys = torch.cat([fresh, old])[torch.randperm(n, generator=g, device=_device())]
    return fresh, keys, _values(g, n)


def _tree(case, seed):
    keys, vals = _loaded(case, seed)
    return BPlusTree.bulk_load(keys, vals, fanout=case["fanout"], leaf_cap=case["leaf_cap"],
                               leaf_fill=case.get("leaf_fill"))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "load":
        keys, vals = _loaded(case, seed)
        return dict(case=case, keys=keys, vals=vals)
    s = dict(case=case, tree=_tree(case, seed))
    if kind == "search":
        s["q"] = _queries(case, seed, case["n"], case["dist"], 2)
    elif kind == "host":
        q = _queries(case, seed, case["n"], case["dist"], 2).cpu()
        if case["pinned"]:
            s["q"], s["out"] = q.pin_memory(), torch.empty(case["n"], dtype=torch.int64).pin_memory()
        else:
            s["q"], s["out"] = q.numpy(), None
    elif kind == "plan":
        sizes = _batch_sizes(case, seed)
        q = torch.cat([_queries(case, seed, m, "zipf" if b % 2 else "uniform", 100 + b) for b, m in enumerate(sizes)])
        s["out"] = torch.empty_like(q)
        s["plan"] = s["tree"].plan(list(zip(q.split(sizes), s["out"].split(sizes))))
    elif kind in ("range", "between"):
        s["start"], s["to"] = _range_inputs(case, seed)
    else:
        s["fresh"], s["keys"], s["vals"] = _write_batch(case, seed)
        s["tree"].upsert(s["keys"], s["vals"])  # the rows that the first epoch will expire
    return s


class _DeviceArray:
    """One of the tree's device arrays (hm_tree_info), as torch takes it; keeps the tree."""

    def __init__(self, tree, ptr, count, typestr):
        self.tree = tree
        self.__cuda_array_interface__ = dict(shape=(count,), typestr=typestr, data=(ptr, False), version=3, strides=None)


def _contents(tree):
    """The stored records where they lie: leaf rows, records per leaf, records before each leaf."""
    i = tree.info()
    parts = ((i.leaf_rows, i.n_leaf * i.leaf_row_words, "<i8"), (i.leaf_cnt, i.n_leaf, "<i4"),
             (i.leaf_base, i.n_leaf, "<i8"))
    return [torch.as_tensor(_DeviceArray(tree, p, n, t), device="cuda") for p, n, t in parts]


def run(s):
    kind = s["case"]["kind"]
    if kind == "search":
        return s["tree"].search(s["q"])
    if kind == "host":
        return s["tree"].search(s["q"], out=s["out"])
    if kind == "plan":
        s["plan"].launch()
        return s["out"]
    if kind == "range":
        return s["tree"].range_search(s["start"], s["to"])
    if kind == "between":
        return s["tree"].range_between(s["start"], s["to"])
    if kind == "write":
        removed = s["tree"].delete(s["fresh"])
        s["tree"].upsert(s["keys"], s["vals"])
        return [removed] + _contents(s["tree"])
    c = s["case"]
    tree = BPlusTree.bulk_load(s["keys"], s["vals"], fanout=c["fanout"], leaf_cap=c["leaf_cap"],
                               leaf_fill=c["leaf_fill"])
    return _contents(tree)


# ---- work -------------------------------------------------------------------


def _leaf_words(case):
    return 2 * case["leaf_cap"] + (case["leaf_cap"] // 8 if case["leaf_cap"] >= 32 else 0)


def work(case):
    """Bytes one pass cannot do without: inputs and outputs once, and the tree's records once or the touched ones."""
    kind, n, nk = case["kind"], case.get("n", 0), case["n_keys"]
    if kind == "load":
        return dict(bytes=16.0 * nk + 8.0 * _leaf_words(case) * nk / case["leaf_fill"], flops=0.0)
    if kind in ("search", "host", "plan"):
        # distinct records touched by n uniform queries, 16 B each, and at least the keys of a miss
        touched = nk * -math.expm1(-n / nk)
        return dict(bytes=16.0 * n + 16.0 * touched, flops=0.0)
    if kind in ("range", "between"):
        mean = (case["longest"] + 1) / 2 if kind == "range" else case["mean"]
        touched = nk * -math.expm1(-n * mean / nk)
        return dict(bytes=n * (12.0 if kind == "range" else 16.0) + 8.0 * n + 16.0 * n * mean + 16.0 * touched, flops=0.0)
    # write: the batch, each touched leaf record read and written, and both rank updates of leaf_base
    leaves = nk / case["leaf_fill"]
    row = 8.0 * _leaf_words(case)
    fresh = n * case["new"]
    touched = leaves * (-math.expm1(-n / leaves) - math.expm1(-fresh / leaves))
    return dict(bytes=16.0 * n + 8.0 * fresh + 2 * row * touched + 2 * 12.0 * leaves, flops=0.0)


# ---- what the outputs are, by plain torch -----------------------------------


def _search_sorted(keys, vals, q):
    i = torch.searchsorted(keys, q).clamp_(max=len(keys) - 1)
    return torch.where(keys[i] == q, vals[i], torch.full_like(q, -1))


def _sorted_pairs(keys, vals):
    """In key order, the last of equal keys."""
    keys, order = torch.sort(keys, stable=True)
    vals = vals[order]
    last = torch.ones_like(keys, dtype=torch.bool)
    last[:-1] = keys[1:] != keys[:-1]
    return keys[last], vals[last]


def _rows(case, keys, vals, leaf, n_leaf):
    """Leaf rows, counts and bases of sorted pairs whose leaf numbers are given; None if a leaf overflows."""
    lc, row = case["leaf_cap"], _leaf_words(case)
    li = row - 2 * lc
    cnt = torch.bincount(leaf, minlength=n_leaf)
    if int(cnt.max()) > lc:
        return None
    base = torch.cumsum(cnt, 0) - cnt
    slot = torch.arange(len(keys), device=keys.device) - base[leaf]
    rows = torch.full((n_leaf, row), MAX_KEY, dtype=torch.int64, device=keys.device)
    rows[:, li + lc:] = -1
    rows[leaf, li + slot] = keys
    rows[leaf, li + lc + slot] = vals
    for w in range(li):
        rows[:, w] = rows[:, li + 8 * (w + 1)] if 8 * (w + 1) < lc else MAX_KEY
    return [rows.reshape(-1), cnt.to(torch.int32), base]


def _even_leaves(case):
    """First loaded record of each leaf of a fresh load, records spread evenly."""
    n = case["n_keys"]
    n_leaf = -(-n // case["leaf_fill"])
    j = torch.arange(n_leaf, device=_device(), dtype=torch.int64)
    return j * (n // n_leaf) + torch.clamp(j, max=n % n_leaf), n_leaf


def exact(case, seed):
    kind = case["kind"]
    keys, vals = _sorted_pairs(*_loaded(case, seed))
    if kind in ("search", "host"):
        r = _search_sorted(keys, vals, _queries(case, seed, case["n"], case["dist"], 2))
        return r if kind == "search" else r.cpu()
    if kind == "plan":
        sizes = _batch_sizes(case, seed)
        q = [_queries(case, seed, m, "zipf" if b % 2 else "uniform", 100 + b) for b, m in enumerate(sizes)]
        return _search_sorted(keys, vals, torch.cat(q))
    if kind in ("range", "between"):
        start, to = _range_inputs(case, seed)
        first = torch.searchsorted(keys, start)
        if kind == "range":
            count = torch.minimum(to.to(torch.int64), len(keys) - first)
        else:
            count = (torch.searchsorted(keys, to, right=True) - first).clamp_(min=0)
        offsets = torch.zeros(len(start) + 1, dtype=torch.int64, device=start.device)
        offsets[1:] = torch.cumsum(count, 0)
        at = torch.repeat_interleave(first - offsets[:-1], count)
        at += torch.arange(len(at), device=at.device)
        return offsets, keys[at], vals[at]
    first, n_leaf = _even_leaves(case)
    if kind == "load":
        leaf = torch.searchsorted(first, torch.arange(len(keys), device=keys.device), right=True) - 1
        return _rows(case, keys, vals, leaf, n_leaf)
    fresh, bk, bv = _write_batch(case, seed)
    fences = keys[first]
    ak, av = _sorted_pairs(torch.cat([keys, bk]), torch.cat([vals, bv]))
    leaf = (torch.searchsorted(fences, ak, right=True) - 1).clamp_(min=0)
    rows = _rows(case, ak, av, leaf, n_leaf)
    return None if rows is None else [len(fresh)] + rows
