"""The bucket join over keys in dense groups: many leaves of a bucket then share
one image, and buckets with more leaves than a stage holds look their queries
up one by one, two at a time where an item has more than one a thread."""
import numpy as np
import pytest

from harmonia_b200 import BPlusTree, datagen as dg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# 2^18 keys make 16384 leaves and 512 buckets of 32; from 768 queries a bucket on
# the join is the one with a directory
@pytest.mark.parametrize("n_q", [40_000, 160_000, 390_000])
@pytest.mark.parametrize("group", [16, 64, 300, 700, 5000])
@pytest.mark.parametrize("span", [30, 61])
def test_grouped_keys(group, span, n_q):
    n = 1 << 18
    rng = np.random.default_rng(group * n_q + span)
    start = np.arange(-(-n // group), dtype=np.int64) * ((1 << span) * group // n) + rng.integers(0, 50, -(-n // group))
    sk = np.unique((start[:, None] + np.arange(group)).ravel())
    sv = dg.values_for(sk)
    near = rng.choice(sk, n_q) + rng.choice(np.array([0, 0, 0, 0, 1, -1, 40, group], np.int64), n_q)
    q = np.concatenate([near, sk[:3] - 1, sk[-3:] + 2, np.full(50, 2**63 - 1), np.full(5, -(2**63))])
    rng.shuffle(q)
    with BPlusTree.bulk_load(torch.from_numpy(sk).cuda(), torch.from_numpy(sv).cuda()) as t:
        t.set_search_config(join=1)
        assert (t.search(torch.from_numpy(q).cuda()).cpu().numpy() == po.PortTree(sk, sv).search(q)).all()


def test_pairs_of_sentinels_in_a_crowded_bucket():
    # one bucket past any stage, all queries in it, Max_Key among them
    sk = np.concatenate([np.arange(200_000, dtype=np.int64), [2**62]])
    sv = dg.values_for(sk)
    q = np.random.default_rng(3).integers(-5, 200_050, 100_000)
    q[::3] = 2**63 - 1
    q[5000:9000] = 2**63 - 1
    with BPlusTree.bulk_load(torch.from_numpy(sk).cuda(), torch.from_numpy(sv).cuda()) as t:
        t.set_search_config(join=1)
        assert (t.search(torch.from_numpy(q).cuda()).cpu().numpy() == po.PortTree(sk, sv).search(q)).all()
