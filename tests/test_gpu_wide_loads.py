"""GPU parity of the point search's 32-byte loads: every slot of full, ragged and
nearly empty rows, hit and missed by one, with each group width."""
import numpy as np
import pytest

from harmonia_b200 import BPlusTree
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

HI, LO = 2**63 - 1, -(2**63)


@pytest.mark.parametrize("fanout", [64, 128])
@pytest.mark.parametrize("n", [1, 15, 17, 1040, 20_011])
def test_every_slot(n, fanout):
    keys = np.arange(n, dtype=np.int64) * 3 - n
    vals = np.arange(n, dtype=np.int64)[::-1] * 7 + 1
    q = np.concatenate([keys, keys + 1, keys - 1, [HI, HI - 1, LO, LO + 1]])
    exp = po.PortTree(keys, vals).search(q)
    with BPlusTree.bulk_load(keys, vals, fanout=fanout) as t:
        for w in (1, 2, 4, 8, 16, 32):
            t.set_search_config(group_width=w, sort_bits=0, join=2)
            got = t.search(torch.from_numpy(q).cuda()).cpu().numpy()
            assert (got == exp).all(), w
