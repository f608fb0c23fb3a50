"""The autotuner leaves the search knobs alone where every box is answered in a
packet of its neighbours: they change nothing there."""
import numpy as np
import pytest

import fkdtree_b200 as F
from fkdtree_b200 import _capi
from fkdtree_b200 import autotune as A


class FakeBatch:
    def __init__(self, packets):
        self.dims = np.array([3] * 8, np.uint32)
        self.pt_off = np.arange(9, dtype=np.uint64) * 20_000
        self.q_off = self.pt_off.copy()
        self.digests_by_packets = packets
        self.params, self.searches = {}, 0

    def set_param(self, name, value):
        self.params[name] = value

    def build(self, coords, ids):
        pass

    def search_digest(self, mins, maxs):
        self.searches += 1


def _tune(b, cache):
    return A.tune_batch(b, None, None, None, None, device="FakeGPU", cache_file=cache, hist_ctas=[148, 296],
                        sync=lambda: None)


def test_no_search_sweep_where_packets_answer(tmp_path):
    cache = str(tmp_path / "tune.json")
    b = FakeBatch(True)
    r = _tune(b, cache)
    assert b.searches == 0 and r["packets"] and not r["cached"]
    assert (r["search_lanes"], r["search_big_n"], r["search_lanes_big"]) == (32, 0, 0)
    assert _tune(FakeBatch(True), cache)["cached"]
    # a batch of the same shape that searches its boxes one by one is swept, and its choice serves both
    b = FakeBatch(False)
    r = _tune(b, cache)
    assert b.searches > 0 and not r["cached"] and not r["packets"]
    assert _tune(FakeBatch(False), cache)["cached"] and _tune(FakeBatch(True), cache)["cached"]


def test_rule_of_packets():
    off = [0, 10_000, 30_000, 50_000]
    assert A.digests_by_packets([3, 3, 4], off, off)
    assert A.digests_by_packets([3, 3, 4], off, [0, 1_250, 3_750, 6_250])
    assert not A.digests_by_packets([3, 3, 4], off, [0, 1_250, 3_749, 6_249])  # too few of the 3-D ones
    assert A.digests_by_packets([3, 3, 4], off, [0, 1_250, 3_750, 3_750])  # none of the 4-D ones


@pytest.mark.gpu
@pytest.mark.parametrize("boxes", [300, 4_000])
def test_rule_is_the_library_s(cuda, boxes):
    rng = np.random.default_rng(1)
    n = 20_000
    x = rng.random((3, n), dtype=np.float32)
    b = F.Batch([3], [0, n], [0, boxes])
    b.build(x.reshape(-1), np.arange(n, dtype=np.uint32))
    lo = np.ascontiguousarray(x[:, :boxes] - np.float32(0.02))
    hi = np.ascontiguousarray(x[:, :boxes] + np.float32(0.02))
    launches, got = [], []
    for packets in (1, 0):
        b.set_param("search_packets", packets)
        n0 = _capi.lib().fkd_kernel_launches()
        got.append(b.search_digest(lo.reshape(-1), hi.reshape(-1)))
        launches.append(_capi.lib().fkd_kernel_launches() - n0)
        if packets:
            by_packets = b.digests_by_packets
    assert not b.digests_by_packets
    assert by_packets == (boxes * A.PACKET_SPARSE >= n) == (launches[0] != launches[1])
    assert all(np.array_equal(p, q) for p, q in zip(*got))
