"""Loads and write epochs just above one bucket of the bucket sort: keys that are
spread evenly take it wherever their range ends between two powers of two (the
other sort takes some twenty launches more), and the results are the oracle's."""
import numpy as np
import pytest

from harmonia_b200 import BPlusTree, datagen as dg, launch_count
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("n", [2049, 2600, 3000, 3071, 3072, 6000, 6143, 12_287])
def test_even_keys_take_the_bucket_sort(n):
    rng = np.random.default_rng(n)
    for i in range(16):  # ranges of 1 to 2 times 2^40
        sk = np.arange(n, dtype=np.int64) * ((1 << 40) * (16 + i) // 16 // n)
        keys = rng.permutation(sk)
        vals = dg.values_for(keys)
        k, v = cuda(keys), cuda(vals)
        before = launch_count()
        with BPlusTree.bulk_load(k, v, leaf_fill=12) as t:
            assert launch_count() - before <= 12, i
            before = launch_count()
            t.upsert(k, v + 1)
            assert launch_count() - before <= 12, i
            xk, xv = t.export()
            assert (xk == sk).all() and (xv == dg.values_for(sk) + 1).all()
            q = np.concatenate([keys, keys + 1])
            assert (t.search(cuda(q)).cpu().numpy() == po.PortTree(xk, xv).search(q)).all()
