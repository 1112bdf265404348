"""Which top levels are staged in shared memory, at the edge of the 16 KiB that
the default budget gives them, and point and range results on either side."""
import numpy as np
import pytest

from harmonia_b200 import BPlusTree
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# inner levels of 1 and 27 rows (16256 bytes), of 1 and 28 (16848 bytes), of 1 and 63
@pytest.mark.parametrize("n,smem,levels", [(3456, None, 2), (3457, None, 1), (3457, 40_000, 1), (3457, 200 * 1024, 2),
                                           (8000, None, 1), (8000, 49_153, 2)])
def test_levels_and_results(n, smem, levels):
    keys = np.arange(n, dtype=np.int64) * 5 - 7 * n
    vals = np.arange(n, dtype=np.int64) * 3 + 1
    q = np.concatenate([keys, keys + 1, [2**63 - 1, -(2**63)]])
    with BPlusTree.bulk_load(keys, vals, leaf_fill=2, smem_bytes=smem) as t:
        assert (t.info().height, t.info().smem_levels) == (2, levels)
        t.set_search_config(join=2, sort_bits=0)
        got = t.search(torch.from_numpy(q).cuda()).cpu().numpy()
        assert (got == po.PortTree(keys, vals).search(q)).all()
        off, rk, rv = (torch.as_tensor(x).cpu().numpy() for x in t.range_between(
            torch.from_numpy(keys[::7].copy()).cuda(), torch.from_numpy(keys[::7] + 11).cuda())[:3])
        first = np.arange(0, n, 7)
        count = np.minimum(3, n - first)
        assert (off == np.concatenate([[0], np.cumsum(count)])).all()
        at = np.concatenate([np.arange(f, f + c) for f, c in zip(first, count)])
        assert (rk == keys[at]).all() and (rv == vals[at]).all()
