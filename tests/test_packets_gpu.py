"""Count and digest searches that walk the tree for 32 boxes at a time
(fkd_packet.cu) and the tables they read (fkd_tables.cu): equal to the oracle
at the sizes where they can go wrong -- trees of one bucket and one point more,
a last level that ends inside a bucket, boxes that hold everything or nothing,
packets whose boxes are far apart -- and to the searches that walk each box
alone."""
import numpy as np
import pytest

import fkdtree_b200 as F
from fkdtree_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

Q = 400_001  # above the smallest number of boxes searched in packets; the last packet is not full


def _points(rng, dim, n):
    c = rng.random((dim, n), dtype=np.float32)
    c[:, rng.random(n) < 0.3] *= np.float32(0.01)  # a dense corner
    c[0, rng.random(n) < 0.05] = np.float32(-0.0)
    c[dim - 1, rng.random(n) < 0.05] = np.float32(0.0)
    c[dim - 1, rng.random(n) < 0.02] = np.inf
    c[0, rng.random(n) < 0.02] = -np.inf
    if dim == 4:
        fin = np.isfinite(c[3])
        c[3, fin] = np.floor(c[3, fin] * 16) / 16
    return c


def _boxes(rng, c, q):
    dim, n = c.shape
    ctr = c[:, rng.integers(0, n, q)]
    hw = rng.choice(np.array([0.0, 1e-3, 0.02, 0.3], np.float32), (1, q), p=[0.3, 0.3, 0.38, 0.02]) * rng.random((dim, q), dtype=np.float32)
    with np.errstate(invalid="ignore"):
        lo, hi = (ctr - hw).astype(np.float32), (ctr + hw).astype(np.float32)
    lo[:, :40], hi[:, 20:60] = -np.inf, np.inf
    lo[:, 60:70], hi[:, 60:70] = hi[:, 60:70] + 1, lo[:, 60:70]  # empty
    lo[0, 70:75] = np.nan
    hi[dim - 1, 75:80] = np.nan
    lo[:, 80:90], hi[:, 80:90] = np.float32(0.0), np.float32(-0.0)
    lo[:, 90:100], hi[:, 90:100] = np.float32(-0.0), np.float32(0.0)
    return lo, hi


@pytest.mark.parametrize("dim", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 2, 15, 31, 32, 47, 63, 64, 95, 1000, 4099, 16_383, 20_011])
def test_packets_match_the_oracle(cuda, dim, n):
    rng = np.random.default_rng(100 * dim + n)
    c = _points(rng, dim, n)
    ids = rng.permutation(n).astype(np.uint32)
    lo, hi = _boxes(rng, c, Q)
    t = F.FKDTree(c, ids).build()
    tab, tid = t.tables()
    want, wdig = O.search_digest(tab, tid, lo, hi)
    cnt, dig = t.digest_boxes(lo, hi)
    assert np.array_equal(t.count_boxes(lo, hi), want)
    assert np.array_equal(cnt, want) and np.array_equal(dig, wdig)
    t.set_param("search_packets", 0)
    c0, d0 = t.digest_boxes(lo, hi)
    assert np.array_equal(c0, want) and np.array_equal(d0, dig)


def test_packets_of_boxes_far_apart(cuda):
    """Few boxes on a large tree: packets give up and their boxes are searched alone."""
    ev = W.clustered_event(n=3_000_000, n_queries=400_000, n_clusters=512, hw_lo=0.0005, hw_hi=0.002, seed=9)
    t = F.FKDTree(ev.coords, ev.ids).build()
    cnt, dig = t.digest_boxes(ev.mins, ev.maxs)
    t.set_param("search_packets", 0)
    c0, d0 = t.digest_boxes(ev.mins, ev.maxs)
    assert np.array_equal(cnt, c0) and np.array_equal(dig, d0)
    assert np.array_equal(t.count_boxes(ev.mins, ev.maxs), c0)


@pytest.mark.parametrize("lanes,big_n,bucket", [(0, 0, 5), (2, 0, 5), (0, 3000, 5), (1, 0, 0)])
def test_batch_packets_uneven_boxes(cuda, lanes, big_n, bucket):
    """Events with no points or boxes, fewer boxes than a packet, and boxes all over the event."""
    rng = np.random.default_rng(77)
    sizes = [40, 0, 1, 31, 32, 5000, 777, 64_000, 33, 2048]
    qn = [100, 3, 33, 0, 1, 31, 5000, 97, 32, 2048]
    dims = [3, 3, 4, 3, 1, 4, 2, 3, 4, 3]
    coords, ids, los, his = [], [], [], []
    for n, q, d in zip(sizes, qn, dims):
        c = _points(rng, d, n) if n else np.zeros((d, 0), np.float32)
        lo, hi = _boxes(rng, c, q) if n and q else (np.zeros((d, q), np.float32), np.ones((d, q), np.float32))
        coords.append(c.reshape(-1))
        ids.append(rng.permutation(n).astype(np.uint32))
        los.append(np.ascontiguousarray(lo).reshape(-1))
        his.append(np.ascontiguousarray(hi).reshape(-1))
    off = lambda x: np.concatenate([[0], np.cumsum(x)]).astype(np.uint64)  # noqa: E731
    b = F.Batch(dims, off(sizes), off(qn))
    b.set_param("search_lanes", lanes)
    b.set_param("search_big_n", big_n)
    b.set_param("search_bucket", bucket)
    b.build(np.concatenate(coords), np.concatenate(ids))
    cnt, dig = b.search_digest(np.concatenate(los), np.concatenate(his))
    at = 0
    for e, (n, q, d) in enumerate(zip(sizes, qn, dims)):
        got_c, got_d = cnt[at:at + q], dig[at:at + q]
        at += q
        if q == 0:
            continue
        if n == 0:
            assert not got_c.any() and not got_d.any()
            continue
        tab, tid = O.build(coords[e].reshape(d, n), ids[e])
        wc, o, found, _ = O.search(tab, tid, los[e].reshape(d, q), his[e].reshape(d, q), variant=O.RECURSIVE)
        assert np.array_equal(got_c, wc) and np.array_equal(got_d, O.digest_of(found, o)), e
