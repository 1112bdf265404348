"""Bulk loads whose keys crowd a bucket of the bucket sort, which then leaves
the load to the LSD sort: every placement of the inputs, at the sizes where the
number of partition passes changes, against the oracle's layout."""
import numpy as np
import pytest

from harmonia_b200 import BPlusTree, datagen as dg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CFG = dict(fanout=64, leaf_cap=16, leaf_fill=13)


def _keys(kind, n):
    rng = np.random.default_rng(n)
    if kind == "outlier":  # a dense range and one key far above it
        k = np.arange(n, dtype=np.int64)
        k[-1] = 2**62
    elif kind == "clusters":  # two dense ranges far apart
        k = np.arange(n, dtype=np.int64)
        k[n // 3:] += 2**60
    else:  # log-normal
        x = np.exp(rng.normal(0, 6, 2 * n + 100)) * 1e9
        k = rng.permutation(np.unique(np.minimum(x, 2.0**62).astype(np.int64)))[:n]
        assert len(k) == n
        k[0] = 2**62 + 1
    k = rng.permutation(k)
    far = int(np.argmax(k))
    k[[0, far]] = k[[far, 0]]  # the first key is always in the sort's sample of the range
    return k


def _put(a, where):
    return torch.from_numpy(a).cuda() if where == "device" else a


# one bucket up to 2048 pairs, one partition pass up to 393215, then two
@pytest.mark.parametrize("n", [2049, 2051, 5000, 70_000, 393_215, 393_216, 393_217])
@pytest.mark.parametrize("kind", ["outlier", "clusters", "lognormal"])
def test_layout_for_every_placement(kind, n):
    keys = _keys(kind, n)
    vals = dg.values_for(keys)
    order = np.argsort(keys, kind="stable")
    exp = po.PortTree(keys[order], vals[order], **CFG).layout()
    for kw, vw in (("host", "host"), ("device", "device"), ("host", "device"), ("device", "host")):
        k, v = _put(keys, kw), _put(vals, vw)
        with BPlusTree.bulk_load(k, v, **CFG) as t:
            got = t.layout()
            for name in ("inner", "prefix", "leaf_rows", "leaf_cnt", "leaf_base"):
                assert (got[name] == exp[name]).all(), (kw, vw, name)
        for a, b in ((k, keys), (v, vals)):  # the caller's arrays stay as they are
            assert (a.cpu().numpy() == b).all() if torch.is_tensor(a) else (a == b).all()


@pytest.mark.parametrize("n", [5000, 70_000])
def test_snapshot_of_crowded_keys(tmp_path, n):
    keys = _keys("outlier", n)
    vals = dg.values_for(keys)
    order = np.argsort(keys)
    path = str(tmp_path / "t.hmb")
    with BPlusTree.bulk_load(_put(keys, "device"), _put(vals, "device"), **CFG) as t:
        t.save(path)
    with BPlusTree.load(path) as t:
        k, v = t.export()
        assert (k == keys[order]).all() and (v == vals[order]).all()
