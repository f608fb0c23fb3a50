"""The tables that searches derive from a tree (in-order copies, bounding
boxes): kNN and radius calls build them only where they read them, and once
that pays; the answers are the same without."""
import numpy as np
import pytest

import fkdtree_b200 as F
from fkdtree_b200 import _capi
from oracle import nn_ref as NN

pytestmark = pytest.mark.gpu


def _launches(call):
    n0 = _capi.lib().fkd_kernel_launches()
    out = call()
    return _capi.lib().fkd_kernel_launches() - n0, out


def _tree(n, dim=3, seed=2):
    rng = np.random.default_rng(seed)
    x = rng.random((dim, n), dtype=np.float32)
    return rng, x, F.FKDTree(x, rng.permutation(n).astype(np.uint32)).build()


@pytest.mark.parametrize("dim, k", [(1, 12), (2, 7), (3, 2)])
def test_knn_by_threads_builds_no_tables(cuda, dim, k):
    rng, x, t = _tree(50_000, dim)
    ctr = rng.random((dim, 20_000), dtype=np.float32)  # more than the warps take at this k
    first, a = _launches(lambda: t.knn(ctr, k))
    later, b = _launches(lambda: t.knn(ctr, k))
    assert first == later
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1].view(np.uint32), b[1].view(np.uint32))
    t.close()


def test_few_queries_on_a_new_tree_do_without_tables(cuda):
    rng, x, t = _tree(300_000)
    tid = t._ids
    ctr = rng.random((3, 40), dtype=np.float32)
    want = NN.knn(x, tid, ctr, 2)
    counts = []
    for _ in range(12):
        n, got = _launches(lambda: t.knn(ctr, 2))
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
        counts.append(n)
    assert counts[0] == counts[1] == min(counts)  # none yet
    built = [i for i, n in enumerate(counts) if n > min(counts)]
    assert len(built) == 1 and counts[-1] == min(counts)  # built once, kept
    t.build()  # the block is there now: they pay sooner, and the answers stay
    again = [_launches(lambda: t.knn(ctr, 2)) for _ in range(4)]
    assert all(np.array_equal(g[0], want[0]) for _, g in again) and max(n for n, _ in again) > min(counts)
    t.close()


@pytest.mark.parametrize("ordered", [False, True])
def test_balls_with_and_without_tables(cuda, ordered):
    rng, x, t = _tree(300_000, seed=3)
    ctr = rng.random((3, 6_000), dtype=np.float32)
    r = np.full(6_000, 0.012, np.float32)
    first = t.search_radius(ctr, r, ordered=ordered)
    for _ in range(30):
        got = t.search_radius(ctr, r, ordered=ordered)
        assert np.array_equal(got[0], first[0])
        for j in (0, 17, 5_999):  # unordered lists: the same sets
            a, b = (set(o[int(f[j]):int(f[j + 1])].tolist()) for f, o in (got, first))
            assert a == b
        if ordered:
            assert np.array_equal(got[1], first[1])
    assert np.array_equal(t.count_radius(ctr, r), np.diff(first[0]))
    t.close()


@pytest.mark.parametrize("dim, ks, q, n", [(1, (12, 13), 20_000, 30_000), (1, (15, 16), 400_000, 30_000),
                                           (2, (8, 9), 400_000, 30_000), (3, (2, 3), 20_000, 30_000),
                                           (3, (3, 4), 400_000, 30_000), (3, (2, 3), 400_000, 900_000),
                                           (3, (4, 5), 750_000, 30_000), (4, (1, 2), 750_000, 30_000)])
def test_knn_by_threads_and_by_warps(cuda, dim, ks, q, n):
    """Either side of the rule that picks the kernel: the shorter row is the
    beginning of the longer one."""
    rng, x, t = _tree(n, dim, seed=q + n)
    ctr = rng.random((dim, q), dtype=np.float32)
    for _ in range(2):  # (without and with the tables)
        (a, da), (b, db) = (t.knn(ctr, k) for k in ks)
        assert np.array_equal(a, b[:, :ks[0]]) and np.array_equal(da.view(np.uint32), db[:, :ks[0]].view(np.uint32))
    t.close()
