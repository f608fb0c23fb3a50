"""Leaf buckets of trees whose last level is full, nearly empty or in between:
the walk tests those with points of the last level one by one, the others in
pairs.  Sizes 2^H - 1 + M around both edges of a bucket (16 points of the last
level each) and of a step of 32 buckets, against the oracle."""
import numpy as np
import pytest

import fkdtree_b200 as F
from oracle import nn_ref as NN
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [(H, M) for H in (5, 9, 10) for M in (1, 2, 15, 16, 17, 31, 33, (1 << H) // 2 + 3, (1 << H) - 1, 1 << H) if M <= 1 << H]


@pytest.mark.parametrize("dim", [1, 2, 3, 4])
@pytest.mark.parametrize("H, M", SIZES)
def test_walks_at_bucket_edges(cuda, dim, H, M):
    n = (1 << H) - 1 + M
    rng = np.random.default_rng(100 * H + M + dim)
    x = rng.random((dim, n), dtype=np.float32)
    x[:, rng.integers(0, n, n // 8)] = x[:, rng.integers(0, n, n // 8)]  # repeated points
    ids = rng.permutation(n).astype(np.uint32)
    t = F.FKDTree(x, ids).build()
    tab, tid = t.tables()
    for q in (60, 3_000):  # shared by several warps; a warp each
        lo = rng.random((dim, q), dtype=np.float32) - np.float32(0.2)
        hi = lo + rng.random((dim, q), dtype=np.float32)
        counts, offs, want, _ = O.search(tab, tid, lo, hi, variant=O.LEVEL_ORDER)
        _, digests = O.search_digest(tab, tid, lo, hi)
        assert np.array_equal(t.count_boxes(lo, hi), counts)
        c, d = t.digest_boxes(lo, hi)
        assert np.array_equal(c, counts) and np.array_equal(d, digests)
        o, i = t.search_boxes(lo, hi)
        assert np.array_equal(o, offs) and np.array_equal(i, want)
        o, i = t.search_boxes(lo, hi, ordered=False)
        assert np.array_equal(o, offs) and np.array_equal(O.digest_lists(o, i), digests)
        ctr, r = np.ascontiguousarray(lo + np.float32(0.2)), rng.random(q, dtype=np.float32) * np.float32(0.5)
        o, i = t.search_radius(ctr, r)
        ro, ri = NN.radius(tab, tid, ctr, r)
        assert np.array_equal(o, ro) and np.array_equal(i, ri)
    t.close()


@pytest.mark.parametrize("dim", [1, 2, 3, 4])
@pytest.mark.parametrize("q", [3, 590, 1_190, 2_400, 7_000])
def test_walks_shared_by_warps(cuda, dim, q):
    """Few boxes: eight, four, two warps a box or one; boxes of a few points, of
    a step's worth, of most of the tree."""
    n = 70_001
    rng = np.random.default_rng(q + dim)
    x = rng.random((dim, n), dtype=np.float32)
    ids = rng.permutation(n).astype(np.uint32)
    t = F.FKDTree(x, ids).build()
    tab, tid = t.tables()
    results = np.float32(10.0) ** rng.uniform(0, 4.8, q).astype(np.float32) * np.where(rng.random(q) < 0.05, 1.0, 0.02)
    hw = (0.5 * np.minimum(1.0, results / n) ** (1.0 / dim)).astype(np.float32)
    ctr = x[:, rng.integers(0, n, q)]
    lo, hi = ctr - hw, ctr + hw
    digests = O.search_digest(tab, tid, lo, hi)
    for _ in range(2):
        assert np.array_equal(t.count_boxes(lo, hi), digests[0])
        c, d = t.digest_boxes(lo, hi)
        assert np.array_equal(c, digests[0]) and np.array_equal(d, digests[1])
    if q >= 4_096:  # fewer balls are counted node by node
        near = [len(NN.radius(tab, tid, ctr[:, j:j + 1], hw[j:j + 1])[1]) for j in range(0, q, 100)]
        assert np.array_equal(t.count_radius(ctr, hw)[::100], near)
    t.close()
