"""Write epochs, range scans and hm_sync on one stream while the thread
captures another: they neither fail nor end the capture, also where the
library's page-locked result slots have to be made first."""
import numpy as np
import pytest

from harmonia_b200 import BPlusTree, datagen as dg
from harmonia_b200.tree import trim_memory
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
def test_epoch_beside_a_capture(mode):
    keys = dg.gen_keys(20_000, seed=9)
    sk = np.sort(keys)
    sv = dg.values_for(sk)
    bk, bv = dg.gen_upserts(keys, 300, 0.2, seed=10)
    with BPlusTree.bulk_load(keys, dg.values_for(keys), leaf_fill=8) as t:
        s = torch.cuda.Stream()
        t.upsert(cuda(bk), cuda(bv), stream=s)  # the tree's scratch for this stream
        sk, sv = po.upsert_set(sk, sv, bk, bv)
        dk, dv = cuda(bk), cuda(bv + 1)
        x = torch.zeros(8, device="cuda")
        g = torch.cuda.CUDAGraph()
        trim_memory()
        with torch.cuda.graph(g, capture_error_mode=mode):
            y = x + 1
            t.upsert(dk, dv, stream=s)
            t.sync(stream=s)
            y = y + 1
        sk, sv = po.upsert_set(sk, sv, bk, bv + 1)
        assert t.size == len(sk)
        g.replay()
        torch.cuda.synchronize()
        assert (y == 2).all()
        xk, xv = t.export()
        assert (xk == sk).all() and (xv == sv).all()
