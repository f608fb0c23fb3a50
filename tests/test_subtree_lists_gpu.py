"""The presorted-list subtree kernel on coordinates with repeated values, all dimensions."""
import numpy as np
import pytest

import fkdtree_b200 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _tied(rng, n, kind):
    if kind == "layers":  # few values, exact in a few bits: the ranges shift down without loss
        return rng.integers(1, 12, n).astype(np.float32)
    if kind == "runs":  # runs of 31 to 34 equal values in any cell of points
        return np.repeat(rng.random(n // 31 + 1, dtype=np.float32), rng.integers(31, 35, n // 31 + 1))[:n]
    # few values over the whole float range: no common zero bits, 64-bit keys
    pool = np.concatenate([np.float32([-3.4e38, -1.1e-38, -0.0, 0.0, 1.3e-39, 3.3e38]), rng.standard_normal(5).astype(np.float32)])
    return rng.choice(pool, n).astype(np.float32)


@pytest.mark.parametrize("kind", ["layers", "runs", "wide"])
@pytest.mark.parametrize("dim", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 33, 512, 1023, 1024, 1025, 9_001])
def test_repeated_values_are_ordered_by_id(cuda, n, dim, kind):
    """One tied coordinate among continuous ones, then every coordinate tied;
    ids far apart, so that no order of slots or of short ids stands in for them."""
    rng = np.random.default_rng(1000 * dim + n)
    ids = (rng.permutation(n).astype(np.uint64) * 2654435761 % (1 << 32)).astype(np.uint32)
    for tied in ([dim - 1], list(range(dim))):
        c = rng.random((dim, n), dtype=np.float32)
        for w in tied:
            c[w] = rng.permutation(_tied(rng, n, kind)) if kind != "runs" else _tied(rng, n, kind)
        t = F.FKDTree(c, ids).build()
        tab, tid = t.tables()
        t.close()
        want = O.build(c, ids)
        assert np.array_equal(tab.view(np.uint32), want[0].view(np.uint32)), (tied, kind)
        assert np.array_equal(tid, want[1]), (tied, kind)


def test_four_dimensions_in_both_subtree_sizes(cuda):
    rng = np.random.default_rng(5)
    c = rng.random((4, 70_003), dtype=np.float32)
    c[3] = rng.integers(0, 40, c.shape[1]).astype(np.float32)
    ids = rng.permutation(c.shape[1]).astype(np.uint32)
    want = O.build(c, ids)
    for name, v in (("subtree_size", 512), ("subtree_size", 1024), ("subtree", 1)):
        t = F.FKDTree(c, ids).set_param(name, v).build()
        tab, tid = t.tables()
        t.close()
        assert np.array_equal(tab.view(np.uint32), want[0].view(np.uint32)) and np.array_equal(tid, want[1]), (name, v)


@pytest.mark.parametrize("dim", [1, 2, 3, 4])
def test_smallest_trees(cuda, dim):
    """Every shape of the last three levels: all sizes up to 40, values with ties, ids in any order."""
    rng = np.random.default_rng(dim)
    for n in range(1, 41):
        c = rng.integers(0, 6, (dim, n)).astype(np.float32)
        ids = rng.choice(np.iinfo(np.uint32).max, n, replace=False).astype(np.uint32)
        t = F.FKDTree(c, ids).build()
        tab, tid = t.tables()
        t.close()
        want = O.build(c, ids)
        assert np.array_equal(tab.view(np.uint32), want[0].view(np.uint32)) and np.array_equal(tid, want[1]), n
