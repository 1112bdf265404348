"""A staging budget that a caller sets on a loaded tree is taken at its word;
the default one leaves levels beyond 16 KiB to L1."""
import numpy as np
import pytest

from harmonia_b200 import BPlusTree
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_levels_follow_the_budget_that_was_set():
    n = 3457  # inner levels of 1 and 28 rows: 592 and 16848 bytes with their child ids
    keys = np.arange(n, dtype=np.int64) * 5 - 7 * n
    vals = np.arange(n, dtype=np.int64) * 3 + 1
    q = torch.from_numpy(np.concatenate([keys, keys + 1])).cuda()
    exp = po.PortTree(keys, vals).search(q.cpu().numpy())
    with BPlusTree.bulk_load(keys, vals, leaf_fill=2) as t:
        assert t.info().smem_levels == 1
        for smem, levels in ((40_000, 2), (16_000, 1), (20_000, 2), (49_152, 1), (200 * 1024, 2), (700, 1)):
            t.set_search_config(smem_bytes=smem, join=2)
            assert t.info().smem_levels == levels, smem
            assert (t.search(q).cpu().numpy() == exp).all()
            t.set_search_config(group_width=8)  # other settings leave it as it is
            assert t.info().smem_levels == levels, smem
            t.set_search_config(group_width=4)
        t.set_search_config(smem_bytes=40_000)
        t.upsert(torch.from_numpy(keys[:5]).cuda(), torch.from_numpy(vals[:5]).cuda())
        assert t.info().smem_levels == 2  # and after an epoch
