"""GPU parity of the bucket sort under the bulk loader: its size and bucket
edges, key spacings that take its counting, bitonic and fallback paths, and
its error cases, against the oracle's layout."""
import numpy as np
import pytest

from harmonia_b200 import BPlusTree, HarmoniaError, datagen as dg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _keys(kind, n):
    i = np.arange(n, dtype=np.int64)
    rng = np.random.default_rng(n)
    if kind == "scattered":
        return dg.gen_keys(n, seed=n)
    if kind == "dense":
        return rng.permutation(i)
    if kind == "descending":  # range of all 64 bits
        return np.int64(2**63 - 2) - i * np.int64((2**64 - 4) // max(n, 2) // 2) * 2
    if kind == "ends":  # INT64_MIN and the largest key that can be stored beside a dense middle: falls back to LSD
        k = rng.permutation(i)
        k[:2] = [-(2**63), 2**63 - 2]
        return k
    if kind == "groups":  # scattered groups of 30 neighbours: crowded bins inside evenly filled buckets
        return rng.permutation(dg.gen_keys(n // 30 + 1, seed=n)[i // 30] // 64 * 64 + i % 30)
    raise ValueError(kind)


def _same_layout(t, keys, vals, **cfg):
    order = np.argsort(keys, kind="stable")
    exp = po.PortTree(keys[order], vals[order], **cfg).layout()
    got = t.layout()
    for k in ("inner", "prefix", "leaf_rows", "leaf_cnt", "leaf_base"):
        assert (got[k] == exp[k]).all(), k


# one bucket up to 2048 pairs, one pass up to 2^18, then two; 4096-pair tiles
@pytest.mark.parametrize("n", [3, 2047, 2048, 2049, 4096, 4097, 1 << 18, (1 << 18) + 1, 700_001])
@pytest.mark.parametrize("kind", ["scattered", "dense", "descending", "ends", "groups"])
def test_layout(kind, n):
    keys = _keys(kind, n)
    vals = dg.values_for(keys)
    cfg = dict(fanout=128, leaf_cap=64, leaf_fill=49) if n % 2 else dict(fanout=64, leaf_cap=16, leaf_fill=13)
    dev = kind in ("scattered", "ends")  # device inputs are read in place, host inputs are copied
    put = (lambda a: torch.from_numpy(a).cuda()) if dev else (lambda a: a)
    with BPlusTree.bulk_load(put(keys), put(vals), **cfg) as t:
        _same_layout(t, keys, vals, **cfg)
        q = np.concatenate([keys[:: max(1, n // 5000)], dg.gen_point_queries(keys, 1000, 0.5, seed=3)])
        exp = po.PortTree(np.sort(keys), dg.values_for(np.sort(keys)), **cfg).search(q)
        assert (t.search(torch.from_numpy(q).cuda()).cpu().numpy() == exp).all()


@pytest.mark.parametrize("n", [100, 5000, 300_000])
@pytest.mark.parametrize("kind", ["scattered", "groups"])
def test_errors(kind, n):
    keys = _keys(kind, n)
    twice, top = keys.copy(), keys.copy()
    twice[n // 2] = keys[n // 3]
    top[n // 4] = 2**63 - 1
    both = twice.copy()
    both[n // 4] = 2**63 - 1
    many = np.where(np.arange(n) < n // 2, keys[0], keys)  # one key for half of the batch
    for bad, code in ((twice, -3), (top, -4), (both, -4), (many, -3)):
        with pytest.raises(HarmoniaError) as e:
            BPlusTree.bulk_load(bad, bad)
        assert e.value.code == code
    with BPlusTree.bulk_load(keys, keys) as t:
        assert t.size == n
