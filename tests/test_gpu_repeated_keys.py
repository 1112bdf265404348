"""Write epochs in which one key fills a long run of the batch: the leaf's
other keys on either side of the run, run lengths around the words of marks
that a step looks at, and the time of a run of a million."""
import time

import numpy as np
import pytest

from harmonia_b200 import BPlusTree, datagen as dg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


N = 3000
STEP = np.int64(1) << 40


@pytest.mark.parametrize("run", [1, 30, 32, 33, 64, 127, 129, 1000, 4095, 4097, 8160, 8192, 8225, 16_383, 16_390, 33_000,
                                 70_001])
@pytest.mark.parametrize("cfg", [dict(leaf_fill=8), dict(fanout=128, leaf_cap=64, leaf_fill=40)])
def test_run_between_the_keys_of_its_leaf(run, cfg):
    fill = cfg["leaf_fill"]
    sk = np.arange(N, dtype=np.int64) * STEP
    sv = dg.values_for(sk)
    rng = np.random.default_rng(run)
    with BPlusTree.bulk_load(cuda(sk), cuda(sv), **cfg) as t:
        for epoch, at in enumerate((5 * fill + 3, 20 * fill)):  # inside a leaf, and its first key
            hot = sk[at] + (epoch == 0)  # a new key, then a stored one
            near = sk[at] + np.array([-3, -2, 7, 9], np.int64)
            far = sk[1000:1300:13] + 5
            bk = rng.permutation(np.concatenate([np.full(run, hot), near, far, sk[40:50]]))
            bv = rng.integers(0, 2**62, len(bk))
            t.upsert(cuda(bk), cuda(bv))
            sk, sv = po.upsert_set(sk, sv, bk, bv)
            xk, xv = t.export()
            assert (xk == sk).all() and (xv == sv).all()
            dk = rng.permutation(np.concatenate([np.full(run, hot + 1), near[1:], far[::2], np.full(run, near[2])]))
            before = len(sk)
            gone = t.delete(cuda(dk))
            sk, sv = po.delete_set(sk, sv, dk)
            assert gone == before - len(sk)
            xk, xv = t.export()
            assert (xk == sk).all() and (xv == sv).all()


def _best(f, between, reps=3):
    times = []
    for _ in range(reps):
        torch.cuda.synchronize()
        a = time.perf_counter()
        f()
        times.append(time.perf_counter() - a)
        between()
    return min(times)


def test_a_long_run_costs_no_walk():
    # Half of a batch is one key.  Where its leaf has new keys too, the epoch
    # costs a look at the run's marks more than where it has none: far less
    # than the sort, and not a step per 32 keys.
    half = 1 << 20
    sk = np.arange(1 << 19, dtype=np.int64) * STEP // 4
    rng = np.random.default_rng(1)
    rest = rng.choice(sk, half)
    hot = np.full(half, sk[1 << 18])
    near = hot[0] + np.array([-2, -1, 1, 2], np.int64)
    plain, mixed = np.concatenate([hot, rest]), np.concatenate([hot, rest[:-4], near])
    absent = np.concatenate([hot + 1, rest[:0]])
    with BPlusTree.bulk_load(cuda(sk), cuda(dg.values_for(sk)), leaf_fill=8) as t:
        p, m, d = cuda(plain), cuda(mixed), cuda(near)
        t.upsert(p, p)
        t_plain = _best(lambda: t.upsert(p, p), lambda: None)
        t.upsert(m, m)
        t.delete(d)
        t_mixed = _best(lambda: t.upsert(m, m), lambda: t.delete(d))
        assert t_mixed < 3 * t_plain, (t_mixed, t_plain)
        a, b = cuda(absent), cuda(np.concatenate([absent, near[-1:]]))
        t.delete(a)
        t_plain = _best(lambda: t.delete(a), lambda: None)
        t.upsert(d, d)
        t_mixed = _best(lambda: t.delete(b), lambda: t.upsert(d, d))
        assert t_mixed < 3 * t_plain, (t_mixed, t_plain)
