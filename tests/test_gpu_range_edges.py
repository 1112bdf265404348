"""GPU parity of the range copy at its chunk edges (128 records, 16-slot
pieces, odd output offsets) and of the locate at the ends of the key space."""
import numpy as np
import pytest

from harmonia_b200 import BPlusTree, datagen as dg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("cfg", [dict(), dict(leaf_fill=5), dict(leaf_cap=64), dict(fanout=128, leaf_cap=64, leaf_fill=33)])
@pytest.mark.parametrize("n", [1, 3, 40, 20_000])
def test_chunk_edges(n, cfg):
    keys = dg.gen_keys(20_000, seed=6)
    sk = np.sort(keys)
    sk, keys = sk - 2**62, keys - 2**62  # negative keys too
    vals = dg.values_for(keys)
    rng = np.random.default_rng(n)
    with BPlusTree.bulk_load(keys, vals, **cfg) as t:
        gone = rng.choice(keys, 4000, replace=False)
        t.delete(gone)  # leaves of many sizes
        ek, ev = po.delete_set(sk, dg.values_for(sk), gone)
        tree = po.PortTree(ek, ev)
        length = rng.choice([0, 1, 15, 16, 17, 127, 128, 129, 500], n).astype(np.int32)
        first = rng.integers(0, len(ek), n)
        start = ek[first] - rng.integers(0, 2, n)
        start[0] = -(2**63)
        start[-1] = ek[-1] + (n % 2)
        got = t.range_search(cuda(start), cuda(length))
        assert all((a.cpu().numpy() == b).all() for a, b in zip(got, tree.range(start, length)))
        end = ek[np.minimum(first + np.maximum(length, 1) - 1, len(ek) - 1)] + rng.integers(-1, 2, n)
        end[-1] = 2**63 - 1
        exp = tree.range_between(start, end)
        for cap in (None, int(exp[0][-1])):
            got = t.range_between(cuda(start), cuda(end), cap=cap)
            assert all((a.cpu().numpy() == b).all() for a, b in zip(got, exp))


def test_scan_in_two_halves():
    """Scans begun and dropped give their scratch back, host and device buffers alike."""
    import ctypes

    from harmonia_b200 import HarmoniaError, native

    keys = dg.gen_keys(5000, seed=3)
    sk = np.sort(keys)
    with BPlusTree.bulk_load(keys, dg.values_for(keys)) as t:
        tree = po.PortTree(sk, dg.values_for(sk))
        start = np.ascontiguousarray(sk[::50])
        end = start + 2**55
        exp = tree.range_between(start, end)
        for s, e in ((start, end), (cuda(start), cuda(end))):
            off = np.zeros(len(start) + 1, np.int64) if s is start else torch.zeros(len(start) + 1, dtype=torch.int64, device="cuda")
            ptr = (lambda a: a.ctypes.data) if s is start else (lambda a: a.data_ptr())
            for _ in range(20):  # more scans than the scratch pool keeps blocks
                scan, total = ctypes.c_void_p(), ctypes.c_size_t()
                native.check(native.lib().hm_range_between_begin(t.handle, ptr(s), ptr(e), len(start), ptr(off),
                                                                 ctypes.byref(total), None, ctypes.byref(scan)))
                assert total.value == exp[0][-1]
                native.check(native.lib().hm_range_finish(scan, None, None))
            with pytest.raises(HarmoniaError) as err:
                t.range_between(s, e, cap=int(exp[0][-1]) - 1)
            assert err.value.code == native.HM_ECAPACITY
            got = t.range_between(s, e)
            assert all((np.asarray(a.cpu() if hasattr(a, "cpu") else a) == b).all() for a, b in zip(got, exp))
        assert native.lib().hm_range_finish(None, None, None) == -1
