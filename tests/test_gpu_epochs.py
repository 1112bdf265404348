"""GPU parity of write epochs at the edges of their kernels: batches around a
word of 32 keys and around the one-CTA sort, leaf runs that reach over words,
repeated keys, overflowing leaves and batches that crowd a sort bucket."""
import numpy as np
import pytest

from harmonia_b200 import BPlusTree, datagen as dg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _batch(kind, keys, n, rng):
    old = rng.choice(keys, n)
    new = dg.gen_keys(n, seed=n + 77)
    if kind == "scattered":  # a quarter new
        return np.where(rng.random(n) < 0.25, new, old)
    if kind == "near":  # neighbours of a few stored keys: long runs on few leaves, most without room
        return rng.choice(keys, max(1, n // 40))[rng.integers(0, max(1, n // 40), n)] + rng.integers(-20, 20, n)
    if kind == "repeated":  # about eight times each, stored and new
        return rng.choice(np.concatenate([old[: n // 16 + 1], new[: n // 16 + 1]]), n)
    if kind == "hot":  # half of the batch one key, past what a sort bucket holds in the larger batches
        return np.where(rng.random(n) < 0.5, keys[len(keys) // 2], np.where(rng.random(n) < 0.5, new, old))
    raise ValueError(kind)


@pytest.mark.parametrize("n", [1, 31, 33, 1024, 2048, 2049, 9000])
@pytest.mark.parametrize("kind", ["scattered", "near", "repeated", "hot"])
@pytest.mark.parametrize("cfg", [dict(leaf_fill=12), dict(fanout=128, leaf_cap=64, leaf_fill=40)])
def test_upsert_then_delete(n, kind, cfg):
    rng = np.random.default_rng(n)
    keys = dg.gen_keys(30_000, seed=4)
    sk = np.sort(keys)
    sv = dg.values_for(sk)
    ref_rule = n % 2 == 1
    with BPlusTree.bulk_load(keys, dg.values_for(keys), **cfg) as t:
        for epoch in range(2):
            bk = _batch(kind, keys, n, rng)
            bv = rng.integers(0, 2**62, n)
            t.upsert(cuda(bk), cuda(bv), ref_rule=ref_rule)
            sk, sv = po.upsert_set(sk, sv, bk, bv, ref_rule)
            assert t.size == len(sk)
            dk = np.concatenate([bk[: n // 2], dg.gen_keys(n // 2 + 1, seed=n + epoch), [2**63 - 1]])
            gone = t.delete(cuda(dk))
            before = len(sk)
            sk, sv = po.delete_set(sk, sv, dk)
            assert gone == before - len(sk)
        xk, xv = t.export()
        assert (xk == sk).all() and (xv == sv).all()
        q = np.concatenate([bk, sk[::7]])
        tree = po.PortTree(sk, sv)
        assert (t.search(cuda(q)).cpu().numpy() == tree.search(q)).all()
        st, ln = dg.gen_ranges(200, 1, 100, seed=n)
        got = t.range_search(cuda(st), cuda(ln.astype(np.int32)))
        assert all((a.cpu().numpy() == b).all() for a, b in zip(got, tree.range(st, ln)))


def test_larger_batches_sorted_in_one_and_two_passes():
    keys = dg.gen_keys(1_000_000, seed=8)
    sk = np.sort(keys)
    sv = dg.values_for(sk)
    with BPlusTree.bulk_load(keys, dg.values_for(keys), leaf_fill=12) as t:
        for m in (300_000, 500_001):  # 256 buckets, then 512
            bk, bv = dg.gen_upserts(sk, m, 0.1, seed=m)
            t.upsert(cuda(bk), cuda(bv))
            sk, sv = po.upsert_set(sk, sv, bk, bv)
            dk = bk[::3]
            assert t.delete(cuda(dk)) == len(np.unique(dk))
            sk, sv = po.delete_set(sk, sv, dk)
        xk, xv = t.export()
        assert (xk == sk).all() and (xv == sv).all()
