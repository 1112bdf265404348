"""Replays of a captured plan over the bucket join after write epochs that
raised the tree's largest key in place (no rebuild, so no re-capture)."""
import numpy as np
import pytest

from harmonia_b200 import BPlusTree, datagen as dg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# 2^17 keys in 10923 leaves make 512 buckets, so their images are the offset's
# bits from shift - 31 on: span 2^36 gives shift 27 (whole offsets), 2^50 41
# (ten bits dropped), 2^62 53; from 768 queries a bucket on the join is the one
# with a directory.
@pytest.mark.parametrize("n_q", [20_000, 400_000])
@pytest.mark.parametrize("span", [36, 50, 62])
@pytest.mark.parametrize("how", ["spread", "replaced"])
def test_keys_past_the_captured_end(span, how, n_q):
    n, fill = 1 << 17, 12
    step = np.int64(1) << (span - 17)
    sk = np.arange(n, dtype=np.int64) * step
    sv = dg.values_for(sk)
    end = np.int64(1) << span
    # spread: enough keys to re-spread the last leaves over keys past the old
    # end; replaced: the last leaf keeps only such keys
    count = 150 if how == "spread" else 4
    new = end + np.arange(1, count + 1, dtype=np.int64) * (end >> 9)
    q = np.concatenate([new, new + 1, sk[-40:], dg.gen_point_queries(sk, n_q, 0.9, seed=5)])
    with BPlusTree.bulk_load(cuda(sk), cuda(sv), leaf_fill=fill) as t:
        t.set_search_config(join=1)
        dq, dout = cuda(q), torch.empty(len(q), dtype=torch.int64, device="cuda")
        with t.plan([(dq[:777], dout[:777]), (dq[777:], dout[777:])]) as plan:
            plan.launch()
            torch.cuda.synchronize()
            assert (dout.cpu().numpy() == po.PortTree(sk, sv).search(q)).all()
            rows = t.info().leaf_rows
            nv = new * 3 + 1
            t.upsert(cuda(new), cuda(nv))
            sk, sv = po.upsert_set(sk, sv, new, nv)
            if how == "replaced":
                last = int(t.layout()["leaf_cnt"][-1]) - count
                old = sk[len(sk) - count - last: len(sk) - count]
                assert t.delete(cuda(old)) == last
                sk, sv = po.delete_set(sk, sv, old)
            assert t.info().leaf_rows == rows  # no rebuild
            oracle = po.PortTree(sk, sv)
            plan.launch()
            torch.cuda.synchronize()
            assert (dout.cpu().numpy() == oracle.search(q)).all()
            assert (t.search(dq).cpu().numpy() == oracle.search(q)).all()


@pytest.mark.parametrize("n_q", [20_000, 400_000])
@pytest.mark.parametrize("leaf_cap,fill", [(16, 12), (64, 48)])
def test_keys_between_the_captured_end_and_the_last_bucket(leaf_cap, fill, n_q):
    # the captured range ends a little past the middle of the buckets
    n = 1 << 17
    sk = np.arange(n, dtype=np.int64) * (1 << 20) * 9 // 8
    sv = dg.values_for(sk)
    new = sk[-1] + np.arange(1, 15 * leaf_cap, dtype=np.int64) * (1 << 29)
    q = np.concatenate([new, new + 1, sk[-40:], dg.gen_point_queries(sk, n_q, 0.9, seed=6)])
    with BPlusTree.bulk_load(cuda(sk), cuda(sv), leaf_cap=leaf_cap, leaf_fill=fill) as t:
        t.set_search_config(join=1)
        dq, dout = cuda(q), torch.empty(len(q), dtype=torch.int64, device="cuda")
        with t.plan([(dq, dout)]) as plan:
            rows = t.info().leaf_rows
            t.upsert(cuda(new), cuda(new - 5))
            sk, sv = po.upsert_set(sk, sv, new, new - 5)
            assert t.info().leaf_rows == rows  # no rebuild
            oracle = po.PortTree(sk, sv)
            plan.launch()
            torch.cuda.synchronize()
            assert (dout.cpu().numpy() == oracle.search(q)).all()
            assert (t.search(dq).cpu().numpy() == oracle.search(q)).all()
