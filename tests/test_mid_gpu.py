"""The levels one CTA splits in shared memory, against the oracle and the launches per level."""
import numpy as np
import pytest

import fkdtree_b200 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _coords(rng, dim, n, kind):
    if kind == "uniform":
        return rng.random((dim, n), dtype=np.float32)
    if kind == "one_value":  # every pivot is found by the ids
        return np.full((dim, n), 0.25, np.float32)
    if kind == "few":  # more than a candidate list's worth of points hold the pivot's value
        return rng.integers(0, 5, (dim, n)).astype(np.float32)
    c = rng.standard_normal((dim, n)).astype(np.float32)  # both signs, both zeros, infinities, denormals
    c[:, rng.random(n) < 0.2] = -0.0
    c[:, rng.random(n) < 0.2] = 0.0
    c[:, rng.random(n) < 0.05] = np.inf
    c[:, rng.random(n) < 0.05] = -np.inf
    c[:, rng.random(n) < 0.05] = np.float32(1e-42)
    return c


@pytest.mark.parametrize("kind", ["uniform", "one_value", "few", "signs"])
@pytest.mark.parametrize("dim", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [513, 1_025, 2_048, 4_097, 8_191, 8_192, 8_193, 16_384, 40_001])
def test_segments_split_in_shared_memory(cuda, n, dim, kind):
    rng = np.random.default_rng(n + dim)
    c = _coords(rng, dim, n, kind)
    ids = (rng.permutation(n).astype(np.uint64) * 2654435761 % (1 << 32)).astype(np.uint32)
    want = O.build(c, ids)
    for knobs in ({}, {"subtree_size": 512}, {"small_select": 0}):
        t = F.FKDTree(c, ids)
        for k, v in knobs.items():
            t.set_param(k, v)
        tab, tid = t.build().tables()
        t.close()
        assert np.array_equal(tab.view(np.uint32), want[0].view(np.uint32)), knobs
        assert np.array_equal(tid, want[1]), knobs


def test_repeated_points_build(cuda):
    """Points repeated with their ids: any of the copies may be a node; the
    tables then hold every copy once."""
    rng = np.random.default_rng(3)
    n = 8_000
    c = np.repeat(rng.random((3, n // 50), dtype=np.float32), 50, axis=1)
    ids = np.repeat(np.arange(n // 50, dtype=np.uint32), 50)
    t = F.FKDTree(c, ids).build()
    tab, tid = t.tables()
    t.close()
    want = O.build(c, ids)
    assert np.array_equal(tab.view(np.uint32), want[0].view(np.uint32)) and np.array_equal(tid, want[1])


def test_events_of_all_sizes_in_one_batch(cuda):
    """Events whose levels end at every point: none, only in shared memory, and after launches per level."""
    rng = np.random.default_rng(9)
    sizes = [1, 700, 1_030, 3_000, 8_192, 8_193, 17_000, 70_000, 5, 33_000]
    c = [rng.random((3, n), dtype=np.float32) for n in sizes]
    ids = [rng.permutation(n).astype(np.uint32) for n in sizes]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    b = F.Batch([3] * len(sizes), off, np.zeros_like(off))
    b.build(np.concatenate([x.ravel() for x in c]), np.concatenate(ids))
    tab, tid = b.tables()
    for e, n in enumerate(sizes):
        want = O.build(c[e], ids[e])
        lo = int(off[e])
        assert np.array_equal(tab.ravel()[3 * lo:3 * (lo + n)].view(np.uint32), want[0].ravel().view(np.uint32)), e
        assert np.array_equal(tid[lo:lo + n], want[1]), e


@pytest.mark.parametrize("kind", ["uniform", "one_value", "few", "signs"])
@pytest.mark.parametrize("n", [32_769, 65_537, 393_216, 393_217, 400_003])
def test_segments_selected_by_a_cluster(cuda, n, kind):
    """A level of a few long segments, with and without the candidate list, in one launch or by digit passes."""
    rng = np.random.default_rng(n)
    c = _coords(rng, 2, n, kind)
    ids = (rng.permutation(n).astype(np.uint64) * 2654435761 % (1 << 32)).astype(np.uint32)
    want = O.build(c, ids)
    for knobs in ({}, {"small_fix": 0}, {"small_select": 0}):
        t = F.FKDTree(c, ids)
        for k, v in knobs.items():
            t.set_param(k, v)
        tab, tid = t.build().tables()
        t.close()
        assert np.array_equal(tab.view(np.uint32), want[0].view(np.uint32)), knobs
        assert np.array_equal(tid, want[1]), knobs
