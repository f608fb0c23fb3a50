"""Recorded searches (fkd_walk.cu): a warp walks the tree for one box, 32
subtrees at a time, and the lists are written from the record.  Lists equal the
brute-force scan in heap order (the reference's order) at the tree sizes where
the walk's steps and the last level can go wrong, from a pool too small for the
records, without the in-order copy of the nodes, and through every entry point
that writes lists."""
import numpy as np
import pytest

import fkdtree_b200 as F
from oracle import oracle as O
from tests.test_packets_gpu import _boxes, _points

pytestmark = pytest.mark.gpu


def _case(dim, n, q):
    rng = np.random.default_rng(7 * dim + n)
    c = _points(rng, dim, n)
    ids = rng.permutation(n).astype(np.uint32)
    lo, hi = _boxes(rng, c, q)
    t = F.FKDTree(c, ids).build()
    tab, tid = t.tables()
    _, offs, want, _ = O.search(tab, tid, lo, hi, variant=O.BRUTE)
    return t, lo, hi, offs, want


@pytest.mark.parametrize("dim", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 2, 16, 31, 32, 47, 48, 63, 500, 1023, 1024, 1535, 16_384, 33_333, 65_535])
def test_lists_match_brute_force(cuda, dim, n):
    t, lo, hi, offs, want = _case(dim, n, 300)
    o, got = t.search_boxes(lo, hi, ordered=True)
    assert np.array_equal(o, offs) and np.array_equal(got, want)
    o, got = t.search_boxes(lo, hi, ordered=False)
    assert np.array_equal(o, offs)
    assert np.array_equal(O.digest_of(got, o), O.digest_of(want, offs))
    c, d = t.digest_boxes(lo, hi)
    assert np.array_equal(c, np.diff(offs.astype(np.int64))) and np.array_equal(d, O.digest_of(want, offs))


@pytest.mark.parametrize("knob,value", [("search_pool", 1), ("search_pool", 1024), ("search_pool", 5000),
                                        ("search_bucket", 0), ("search_record", 0), ("search_lanes", 4)])
@pytest.mark.parametrize("dim", [3, 4])
def test_lists_with_other_settings(cuda, dim, knob, value):
    t, lo, hi, offs, want = _case(dim, 20_000, 600)
    t.set_param(knob, value)
    for _ in range(2):
        o, got = t.search_boxes(lo, hi, ordered=True)
        assert np.array_equal(o, offs) and np.array_equal(got, want)
        o, got = t.search_boxes(lo, hi, ordered=False)
        assert np.array_equal(o, offs) and np.array_equal(O.digest_of(got, o), O.digest_of(want, offs))


@pytest.mark.parametrize("pool", [0, 2000])
def test_device_lists(cuda, pool):
    import torch
    t, lo, hi, offs, want = _case(3, 40_000, 5000)  # spatial order of the boxes
    t.set_param("search_pool", pool)
    mins, maxs = torch.from_numpy(lo).to(cuda), torch.from_numpy(hi).to(cuda)
    for ordered in (True, False, True):
        o, got = t.search_boxes(mins, maxs, ordered=ordered)
        assert np.array_equal(o.cpu().numpy(), offs.astype(np.int64))
        g = got.cpu().numpy().view(np.uint32)
        if ordered:
            assert np.array_equal(g, want)
        else:
            assert np.array_equal(O.digest_of(g, offs), O.digest_of(want, offs))


@pytest.mark.parametrize("dim", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 48, 500, 1535, 20_001])
@pytest.mark.parametrize("pool", [0, 1024])
def test_balls_match_brute_force(cuda, dim, n, pool):
    from oracle import nn_ref as NN
    rng = np.random.default_rng(31 * dim + n)
    c = _points(rng, dim, n)
    t = F.FKDTree(c, rng.permutation(n).astype(np.uint32)).build().set_param("search_pool", pool)
    tab, tid = t.tables()
    q = 4100  # above the fewest queries that walk by the bounding boxes
    ctr = np.ascontiguousarray(c[:, rng.integers(0, n, q)])
    rad = rng.choice(np.array([0.0, 1e-3, 0.05, 0.4, 3.0], np.float32), q, p=[0.25, 0.4, 0.33, 0.015, 0.005])
    rad[:6] = [-1.0, np.nan, np.inf, 0.0, 1e30, 1e-30]
    ctr[0, 6:9] = np.nan
    ctr[dim - 1, 9:12] = np.inf
    with np.errstate(invalid="ignore", over="ignore"):
        woff, wids = NN.radius(tab, tid, ctr, rad)
    for _ in range(2):
        off, ids = t.search_radius(ctr, rad)
        assert np.array_equal(off, woff) and np.array_equal(ids, wids)
    assert np.array_equal(t.count_radius(ctr, rad), np.diff(woff.astype(np.int64)))
    off, ids = t.search_radius(ctr, rad, ordered=False)
    assert np.array_equal(off, woff) and np.array_equal(O.digest_of(ids, off), O.digest_of(wids, woff))


@pytest.mark.parametrize("dim,k", [(1, 12), (1, 13), (2, 7), (2, 8), (3, 2), (3, 3), (4, 1), (3, 31), (3, 32), (3, 33),
                                   (2, 64)])
@pytest.mark.parametrize("n", [1, 31, 32, 700, 5000])
@pytest.mark.parametrize("q", [300, 20_000])
def test_neighbours_match_brute_force(cuda, dim, k, n, q):
    """Both kernels (a warp and a thread per query) on either side of the rule between them."""
    from oracle import nn_ref as NN
    rng = np.random.default_rng(dim + 5 * k + n)
    c = _points(rng, dim, n)
    c[:, rng.integers(0, n, n // 10)] = c[:, :1]  # equal distances: the smaller id first
    ids = rng.permutation(n).astype(np.uint32)
    t = F.FKDTree(c, ids).build()
    ctr = np.ascontiguousarray(c[:, rng.integers(0, n, q)])
    ctr[:, q // 2:] += rng.normal(0, 0.05, (dim, q - q // 2)).astype(np.float32)
    ctr[0, 3] = np.nan
    ctr[dim - 1, 4] = np.inf
    got_i, got_d = t.knn(ctr, k)
    pick = np.concatenate([np.arange(10), rng.integers(0, q, 150)])
    with np.errstate(invalid="ignore"):
        want_i, want_d = NN.knn(c, ids, np.ascontiguousarray(ctr[:, pick]), k)
    assert np.array_equal(got_i[pick], want_i)
    assert np.array_equal(got_d[pick].view(np.uint32), want_d.view(np.uint32))


@pytest.mark.parametrize("dim", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 31, 48, 1023, 33_333, 300_000])
def test_few_boxes_share_a_cta(cuda, dim, n):
    """Counts and digests of few boxes: four warps a box, two, and one; boxes that
    hold the whole tree, nothing, a bucket, and a large part of the tree."""
    rng = np.random.default_rng(17 * dim + n)
    c = _points(rng, dim, n)
    ids = rng.permutation(n).astype(np.uint32)
    t = F.FKDTree(c, ids).build()
    tab, tid = t.tables()
    for q in (1, 700, 2_300, 3_900):
        lo, hi = _boxes(rng, c, q)
        w = min(q, 20)
        mid = rng.random((dim, w)).astype(np.float32)
        lo[:, :w], hi[:, :w] = mid - np.float32(0.2), mid + np.float32(0.2)
        _, offs, want, _ = O.search(tab, tid, lo, hi, variant=O.BRUTE if n <= 1023 else O.RECURSIVE)
        k, d = t.digest_boxes(lo, hi)
        assert np.array_equal(k, np.diff(offs.astype(np.int64))), q
        assert np.array_equal(d, O.digest_of(want, offs)), q
        assert np.array_equal(t.count_boxes(lo, hi), k), q
