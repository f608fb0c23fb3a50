"""Calls at the limits: allocations that fail (fkd_debug_fail_alloc), launches
that are refused, slices that do not fit.  A call that cannot do its work says
so, and the handle then answers as if nothing had happened."""
import numpy as np
import pytest

import fkdtree_b200 as F
from fkdtree_b200 import _capi
from fkdtree_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CUDA_ERR, NOMEM, CAPACITY, INTERNAL = 2, 3, 6, 7


@pytest.fixture
def inject():
    L = _capi.lib()
    yield L.fkd_debug_fail_alloc
    L.fkd_debug_fail_alloc(-1)


def _event(n=20_000, q=500, seed=5, half_width=0.03):
    ev = W.uniform_event(n=n, seed=seed, half_width=half_width)
    ev.mins, ev.maxs = np.ascontiguousarray(ev.mins[:, :q]), np.ascontiguousarray(ev.maxs[:, :q])
    return ev


def _lists(t, ev):
    tab, tid = t.tables()
    _, offs, ids, _ = O.search(tab, tid, ev.mins, ev.maxs, variant=O.LEVEL_ORDER)
    return offs, ids


def test_tables_that_found_no_room_are_built_again(cuda, inject):
    """The in-order tables grow when leaf buckets are switched on; when there is
    no room for the larger block, the tables are gone, not marked ready."""
    ev = _event()
    t = F.FKDTree(ev.coords, ev.ids).build()
    offs, ids = _lists(t, ev)
    cap = len(ids)
    t.set_param("search_bucket", 0)
    got = t.search_boxes(ev.mins, ev.maxs, capacity=cap)
    assert np.array_equal(got[0], offs) and np.array_equal(got[1], ids)
    t.set_param("search_bucket", 5)
    inject(0)  # the call's scratch is there: its first allocation is the larger block
    with pytest.raises(F.FKDError) as e:
        t.search_boxes(ev.mins, ev.maxs, capacity=cap)
    assert e.value.status == NOMEM
    inject(-1)
    for bucket in (0, 5):
        t.set_param("search_bucket", bucket)
        got = t.search_boxes(ev.mins, ev.maxs, capacity=cap)
        assert np.array_equal(got[0], offs) and np.array_equal(got[1], ids)
    t.close()
