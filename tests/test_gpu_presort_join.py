"""GPU parity of the query pre-sort and the bucket join where their kernels can
go wrong: counters of one hot bucket, tiles and steps with remainders, first
keys whose 31-bit images coincide, and batches that lie in one bucket."""
import numpy as np
import pytest

from harmonia_b200 import BPlusTree, datagen as dg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _tree_keys(kind):
    n = 60_000
    i = np.arange(n, dtype=np.int64)
    if kind == "scattered":
        return dg.gen_keys(n, seed=12)
    if kind == "dense":
        return i * 3 - 50_000
    # 100 neighbours every so often over all 64 bits: whole leaves share an image
    return np.unique((i // 100 - 300) * np.int64(2**54 + 12345) + (i % 100) * 2)


def _queries(kind, keys, n, rng):
    q = np.where(rng.random(n) < 0.8, rng.choice(keys, n), rng.choice(keys, n) + 1)
    if kind == "hot":  # one key for most of the batch
        q = np.where(rng.random(n) < 0.7, keys[len(keys) // 3], q)
    elif kind == "sorted":
        q = np.sort(q)
    q[:1] = 2**63 - 1
    q[-1:] = -(2**63)
    return q


@pytest.mark.parametrize("tree", ["scattered", "dense", "groups"])
@pytest.mark.parametrize("leaf_cap", [16, 64])
def test_against_the_oracle(tree, leaf_cap):
    keys = _tree_keys(tree)
    sk = np.sort(keys)
    rng = np.random.default_rng(1)
    exp = po.PortTree(sk, dg.values_for(sk))
    with BPlusTree.bulk_load(keys, dg.values_for(keys), leaf_cap=leaf_cap) as t:
        for cfg in (dict(join=1), dict(join=2, sort_bits=3), dict(join=2, sort_bits=8), dict(join=2, sort_bits=13)):
            t.set_search_config(**cfg)
            for n in (2, 319, 321, 8192, 8193, 300_001):
                for kind in ("mixed", "hot", "sorted"):
                    q = _queries(kind, keys, n, rng)
                    assert (t.search(cuda(q)).cpu().numpy() == exp.search(q)).all(), (cfg, n, kind)


def test_counters_past_their_halves():
    """Millions of queries of one bucket: its 16-bit counters spill many times."""
    keys = dg.gen_keys(200_000, seed=2)
    sk = np.sort(keys)
    with BPlusTree.bulk_load(keys, dg.values_for(keys)) as t:
        t.set_search_config(join=1)
        q = np.full(20_000_003, sk[1234], np.int64)
        q[::1000] = np.resize(sk, len(q[::1000]))
        out = t.search(cuda(q)).cpu().numpy()
        assert (out == dg.values_for(q)).all()


@pytest.mark.parametrize("sizes", [[1, 8191, 8192, 8193, 0, 100_000], [3] * 1500])
def test_batch_sets(sizes):
    keys = dg.gen_keys(60_000, seed=12)
    sk = np.sort(keys)
    exp = po.PortTree(sk, dg.values_for(sk))
    rng = np.random.default_rng(5)
    with BPlusTree.bulk_load(keys, dg.values_for(keys)) as t:
        t.set_search_config(join=1)
        qs = [_queries("hot", keys, m, rng) if m else np.zeros(0, np.int64) for m in sizes]
        pairs = [(cuda(q), torch.empty(len(q), dtype=torch.int64, device="cuda")) for q in qs]
        t.search_batches(pairs)
        assert all((o.cpu().numpy() == exp.search(q)).all() for q, (_, o) in zip(qs, pairs))
        with t.plan(pairs) as plan:
            for _, o in pairs:
                o.zero_()
            plan.launch()
            torch.cuda.synchronize()
            assert all((o.cpu().numpy() == exp.search(q)).all() for q, (_, o) in zip(qs, pairs))
