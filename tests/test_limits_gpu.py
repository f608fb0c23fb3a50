"""Calls at the limits: allocations that fail (fkd_debug_fail_alloc), launches
that are refused, slices that do not fit.  A call that cannot do its work says
so, and the handle then answers as if nothing had happened."""
import threading

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


@pytest.fixture
def refuse():
    L = _capi.lib()
    yield L.fkd_debug_fail_launch
    L.fkd_debug_fail_launch(-1)


def _refuse_all(refuse, call):
    """The call with its first launch refused, its second, ...: an error each
    time, until it has no more of them and succeeds.  Returns their number."""
    for k in range(200):
        refuse(k)
        try:
            call()
        except F.FKDError as e:
            assert e.status == CUDA_ERR, (k, e)
        else:
            refuse(-1)
            return k
    raise AssertionError("the call never ran out of launches")


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


# every launch of a build, refused in turn: selects by digit passes, by one CTA, by a cluster; whole
# segments in shared memory; both subtree kernels
@pytest.mark.parametrize("knobs", [{}, {"small_select": 0}, {"small_fix": 0}, {"subtree": 1}])
@pytest.mark.parametrize("n, dim", [(70_001, 3), (40_000, 4)])
def test_refused_launch_fails_the_build(cuda, refuse, n, dim, knobs):
    ev = W.uniform_event(n=n, dim=dim, seed=8)
    want = O.build(ev.coords, ev.ids)
    t = F.FKDTree(ev.coords, ev.ids)
    for k, v in knobs.items():
        t.set_param(k, v)
    t.build()
    launches = _refuse_all(refuse, t.build)
    assert launches >= 6
    tab, tid = t.tables()
    assert np.array_equal(tab.view(np.uint32), want[0].view(np.uint32)) and np.array_equal(tid, want[1])
    t.close()


def test_refused_launch_fails_the_search(cuda, refuse):
    import torch
    ev = _event(q=5_000)
    t = F.FKDTree(ev.coords, ev.ids).build()
    offs, ids = _lists(t, ev)
    counts = np.diff(offs)
    lo, hi = torch.from_numpy(ev.mins).cuda(), torch.from_numpy(ev.maxs).cuda()
    for search in (lambda: t.search_boxes(ev.mins, ev.maxs, capacity=len(ids)), lambda: t.search_boxes(lo, hi)):
        got = []
        assert _refuse_all(refuse, lambda: got.append(search())) >= 4
        o, i = (np.asarray(x.cpu() if hasattr(x, "cpu") else x) for x in got[-1])
        assert np.array_equal(o.astype(np.uint64), offs) and np.array_equal(i.view(np.uint32), ids)
    for call in (lambda: t.count_boxes(ev.mins, ev.maxs), lambda: t.digest_boxes(ev.mins, ev.maxs)[0]):
        got = []
        assert _refuse_all(refuse, lambda: got.append(call())) >= 3
        assert np.array_equal(got[-1], counts)
    ctr, r = ev.coords[:, :5_000].copy(), np.full(5_000, 0.03, np.float32)
    got = []
    _refuse_all(refuse, lambda: got.append(t.search_radius(ctr, r)))
    o, i = t.search_radius(ctr, r)
    assert np.array_equal(got[-1][0], o) and np.array_equal(got[-1][1], i)
    got = []
    _refuse_all(refuse, lambda: got.append(t.knn(ctr, 8)))
    o, i = t.knn(ctr, 8)
    assert np.array_equal(got[-1][0], o) and np.array_equal(got[-1][1].view(np.uint32), i.view(np.uint32))
    t.close()


def test_refused_launch_fails_the_batch(cuda, refuse):
    import torch
    rng = np.random.default_rng(3)
    sizes = [40_000, 1, 900, 9_000]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    coords = torch.from_numpy(rng.random(3 * int(off[-1]), dtype=np.float32)).cuda()
    ids = torch.arange(int(off[-1]), dtype=torch.int32, device="cuda")
    mins, maxs = coords - 0.02, coords + 0.02
    counts = torch.empty(int(off[-1]), dtype=torch.int32, device="cuda")
    digests = torch.empty(int(off[-1]), dtype=torch.int64, device="cuda")
    b = F.Batch([3] * len(sizes), off, off)
    torch.cuda.synchronize()
    assert _refuse_all(refuse, lambda: b.run(coords, ids, mins, maxs, counts, digests)) >= 12
    torch.cuda.synchronize()
    for e, n in enumerate(sizes):
        s = slice(int(off[e]), int(off[e + 1]))
        x = coords[3 * s.start:3 * s.stop].cpu().numpy().reshape(3, n)
        tab, tid = O.build(x, ids[s].cpu().numpy().view(np.uint32))
        c, d = O.search_digest(tab, tid, x - np.float32(0.02), x + np.float32(0.02))
        assert np.array_equal(counts[s].cpu().numpy().view(np.uint32), c)
        assert np.array_equal(digests[s].cpu().numpy().view(np.uint64), d)


def test_threads_build_different_trees(cuda):
    """Different handles are independent: trees of all sizes that the selects'
    shared memory grows with, built by eight threads at once."""
    sizes = [5_000, 17_000, 36_000, 60_000, 110_000, 200_000, 300_000, 390_000]
    evs = [W.uniform_event(n=n, dim=2 + k % 3, seed=n) for k, n in enumerate(sizes)]
    want = [O.build(ev.coords, ev.ids) for ev in evs]
    trees = [F.FKDTree(ev.coords, ev.ids) for ev in evs]
    gate, errors = threading.Barrier(len(evs)), []

    def work(k):
        try:
            for _ in range(40):
                gate.wait()
                trees[k].build()
                lo, hi = evs[k].coords[:, :64] - np.float32(0.01), evs[k].coords[:, :64] + np.float32(0.01)
                trees[k].set_param("search_record", 0)  # the traversing write pass
                trees[k].set_param("search_lanes", 4)
                offs, _ = trees[k].search_boxes(lo, hi)
                assert np.array_equal(np.diff(offs), trees[k].count_boxes(lo, hi))
        except Exception as e:  # noqa: BLE001 -- reported below
            errors.append((k, repr(e)))
            gate.abort()

    th = [threading.Thread(target=work, args=(k,)) for k in range(len(evs))]
    for x in th:
        x.start()
    for x in th:
        x.join()
    assert not errors, errors
    for t, w in zip(trees, want):
        tab, tid = t.tables()
        assert np.array_equal(tab.view(np.uint32), w[0].view(np.uint32)) and np.array_equal(tid, w[1])
        t.close()


def _write(t, ev, offs, room, ordered, device):
    """fkd_search_write into the slices `offs`: its status."""
    import ctypes as C

    import torch
    L = _capi.lib()
    arrs = [ev.mins, ev.maxs, offs, np.zeros(room, np.uint32)]
    if device:
        arrs = [torch.from_numpy(a.view({np.dtype(np.uint64): np.int64, np.dtype(np.uint32): np.int32}.get(a.dtype, a.dtype)))
                .cuda() for a in arrs]
        torch.cuda.synchronize()
        p = [a.data_ptr() for a in arrs]
    else:
        p = [a.ctypes.data for a in arrs]
    s = L.fkd_search_write(t._h, C.c_void_p(p[0]), C.c_void_p(p[1]), ev.mins.shape[1], C.c_void_p(p[2]), C.c_void_p(p[3]),
                           ordered, int(device))
    return s, (arrs[3].cpu().numpy().view(np.uint32) if device else arrs[3])


@pytest.mark.parametrize("q", [40, 5_000])
@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("ordered", [0, 1])
def test_slice_for_a_box_without_results(cuda, ordered, device, q):
    ev = _event(q=q)
    ev.mins[:, 7] = ev.maxs[:, 7] = 2.0  # holds nothing
    t = F.FKDTree(ev.coords, ev.ids).build()
    offs, ids = _lists(t, ev)
    room = len(ids) + 64
    offs = offs.astype(np.uint64)
    assert offs[7] == offs[8]
    wrong = offs.copy()
    wrong[8:] += 3
    assert _write(t, ev, wrong, room, ordered, device)[0] == INTERNAL
    s, got = _write(t, ev, offs, room, ordered, device)
    assert s == 0
    if ordered:
        assert np.array_equal(got[:len(ids)], ids)
    t.close()


@pytest.mark.parametrize("q", [40, 5_000])
@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("ordered", [0, 1])
def test_slice_too_small(cuda, ordered, device, q):
    """An id that finds no room in its box's slice is a capacity error, whether
    the list is ordered (recorded) or not (traversed); nothing is written past it."""
    ev = _event(q=q)
    t = F.FKDTree(ev.coords, ev.ids).build()
    offs, ids = _lists(t, ev)
    offs = offs.astype(np.uint64)
    short = offs.copy()
    assert offs[10] > offs[9]
    short[10:] -= 1
    s, got = _write(t, ev, short, len(ids) + 64, ordered, device)
    assert s == CAPACITY and not got[len(ids) - 1:].any()
    back = offs.copy()
    back[9] = offs[10] + 2  # box 9's slice ends before it starts
    assert _write(t, ev, back, len(ids) + 64, ordered, device)[0] == CAPACITY
    s, got = _write(t, ev, offs, len(ids) + 64, ordered, device)
    assert s == 0 and (not ordered or np.array_equal(got[:len(ids)], ids))
    t.close()


@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("first, last", [(10, 10), (3, 400)])
def test_slices_out_of_range_are_not_sorted(cuda, first, last, device):
    """Ordered lists written without a record are sorted slice by slice: one that
    ends before it starts, or past the end of the output, is an error."""
    ev = _event(q=500)
    t = F.FKDTree(ev.coords, ev.ids).build().set_param("search_record", 0)
    offs, ids = _lists(t, ev)
    offs = offs.astype(np.uint64)
    wrong = offs.copy()
    wrong[first:last + 1] += np.uint64(1 << 33)
    assert _write(t, ev, wrong, len(ids) + 64, 1, device)[0] in (CAPACITY, INTERNAL)
    s, got = _write(t, ev, offs, len(ids) + 64, 1, device)
    assert s == 0 and np.array_equal(got[:len(ids)], ids)
    t.close()


def _launches(call):
    n0 = _capi.lib().fkd_kernel_launches()
    out = call()
    return _capi.lib().fkd_kernel_launches() - n0, out


def test_small_call_does_not_size_the_pool_of_large_ones(cuda):
    """The record pool holds what the call at hand needs, whatever the slot's
    earlier calls were: no box is left to the traversing pass."""
    ev = W.uniform_event(n=200_000, half_width=0.1, seed=9)
    lo, hi = np.ascontiguousarray(ev.mins[:, :20_000]), np.ascontiguousarray(ev.maxs[:, :20_000])
    a, b = (F.FKDTree(ev.coords, ev.ids).build() for _ in range(2))
    b.search_boxes(lo[:, :10], hi[:, :10])
    cap = int(a.count_boxes(lo, hi).sum(dtype=np.uint64))
    na, ra = _launches(lambda: a.search_boxes(lo, hi, capacity=cap))
    nb, rb = _launches(lambda: b.search_boxes(lo, hi, capacity=cap))
    assert na == nb
    assert np.array_equal(ra[0], rb[0]) and np.array_equal(ra[1], rb[1])
    a.close()
    b.close()


def test_asynchronous_write_learns_its_demand(cuda):
    """An ordered device write of an asynchronous handle cannot wait for its
    demand; the slot's next call has it."""
    import torch
    n, q, hw = 1_000_000, 4_000, 0.5 * (80_000 / 1e6) ** (1 / 3)  # some 1,000 entries a box
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    x = torch.rand((3, n), generator=g, device="cuda")
    c = x[:, :q]
    lo, hi = (c - hw).contiguous(), (c + hw).contiguous()
    t = F.FKDTree(x, flags=_capi.FLAG_ASYNC).build()
    counts = t.count_boxes(lo, hi)
    _capi.check(_capi.lib().fkd_sync(t._h))
    offs = torch.zeros(q + 1, dtype=torch.int64, device="cuda")
    offs[1:] = torch.cumsum(counts.to(torch.int64), 0)
    out = torch.empty(int(offs[-1]), dtype=torch.int32, device="cuda")
    first = torch.zeros_like(out)
    torch.equal(out, first)  # (torch keeps the memory this takes)
    free = []
    for k in range(3):
        _capi.check(_capi.lib().fkd_search_write(t._h, lo.data_ptr(), hi.data_ptr(), q, offs.data_ptr(), out.data_ptr(), 1, 1))
        _capi.check(_capi.lib().fkd_sync(t._h))
        free.append(torch.cuda.mem_get_info()[0])
        if k == 0:
            first.copy_(out)
        assert torch.equal(out, first)
        out.zero_()
    assert free[1] < free[0] and free[2] == free[1]  # one larger pool, then enough
    t.close()


@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("q", [300, 5_000])
def test_searches_when_allocations_fail(cuda, inject, q, device):
    """Every allocation of a search on a fresh handle: reported, or done without;
    never a wrong answer."""
    import torch
    ev = _event(q=q)
    ref = F.FKDTree(ev.coords, ev.ids).build()
    offs, ids = _lists(ref, ev)
    dig = O.search_digest(*ref.tables(), ev.mins, ev.maxs)
    box = [torch.from_numpy(a).cuda() for a in (ev.mins, ev.maxs)] if device else [ev.mins, ev.maxs]
    r = np.full(q, 0.03, np.float32)
    ctr = torch.from_numpy(ev.coords[:, :q].copy()).cuda() if device else ev.coords[:, :q].copy()
    rad, knn = ref.search_radius(ctr, r), ref.knn(ctr, 8)
    num = lambda x: (x.cpu().numpy() if hasattr(x, "cpu") else x)  # noqa: E731
    same = lambda a, b: np.array_equal(num(a).view(np.uint32), num(b).view(np.uint32))  # noqa: E731
    calls = {
        "count": (lambda t: t.count_boxes(*box), lambda c: same(c, dig[0])),
        "digest": (lambda t: t.digest_boxes(*box), lambda g: same(g[0], dig[0]) and np.array_equal(num(g[1]).view(np.uint64), dig[1])),
        "lists": (lambda t: t.search_boxes(*box), lambda g: same(g[1], ids)),
        "balls": (lambda t: t.search_radius(ctr, r), lambda g: same(g[1], rad[1])),
        "knn": (lambda t: t.knn(ctr, 8), lambda g: same(g[0], knn[0]) and same(g[1], knn[1])),
    }
    for name, (call, ok) in calls.items():
        for bucket in (0, 5):
            for k in range(14):  # a new handle each time: its allocations come anew
                t = F.FKDTree(ev.coords, ev.ids).build().set_param("search_bucket", bucket)
                if name in ("balls", "knn"):
                    for _ in range(3):
                        call(t)  # (the tables pay by now)
                    t.build()
                inject(k)
                try:
                    assert ok(call(t)), (name, bucket, k)
                except F.FKDError as e:
                    assert e.status == NOMEM, (name, bucket, k, e)
                inject(-1)
                assert ok(call(t)), (name, bucket, k)
                t.close()


def test_counts_do_without_tables(cuda, inject):
    """Counts and digests without leaf buckets have always worked on the nodes
    alone: with no room for the bounding boxes (and the packets' list) they still do."""
    import torch
    ev = _event(n=60_000, q=60_000)
    t = F.FKDTree(ev.coords, ev.ids).build().set_param("search_bucket", 0)
    lo, hi = (torch.from_numpy(np.tile(a, 7)[:, :400_000].copy()).cuda() for a in (ev.mins, ev.maxs))
    few_lo, few_hi = lo[:, :500].contiguous(), hi[:, :500].contiguous()
    dig = O.search_digest(*t.tables(), ev.mins, ev.maxs)
    num = lambda x, ty: x.cpu().numpy().view(ty)  # noqa: E731
    t.knn(ev.coords[:, :1].copy(), 1)  # a slot is there
    c, d = t.digest_boxes(few_lo, few_hi)
    assert np.array_equal(num(c, np.uint32), dig[0][:500])
    t.build()  # the tables are to be made again, in the room they have: let a larger copy be wanted
    t.set_param("search_bucket", 5)
    inject(0)
    assert np.array_equal(num(t.count_boxes(few_lo, few_hi), np.uint32), dig[0][:500])
    c, d = t.digest_boxes(few_lo, few_hi)
    assert np.array_equal(num(c, np.uint32), dig[0][:500]) and np.array_equal(num(d, np.uint64), dig[1][:500])
    inject(-1)
    for fails in (0, 1, 2):  # the boxes' order is needed, the packets' list of boxes left over is not
        b = F.FKDTree(ev.coords, ev.ids).build()
        b.count_boxes(few_lo, few_hi)
        inject(fails)
        try:
            assert np.array_equal(num(b.count_boxes(lo, hi), np.uint32), np.tile(dig[0], 7)[:400_000])
            assert fails > 0
        except F.FKDError as e:
            assert e.status == NOMEM and fails == 0
        inject(-1)
        assert np.array_equal(num(b.count_boxes(lo, hi), np.uint32), np.tile(dig[0], 7)[:400_000])
        b.close()
    t.close()


def test_batch_when_allocations_fail(cuda, inject):
    import torch
    rng = np.random.default_rng(4)
    sizes = [3_000, 1, 900]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    coords = torch.from_numpy(rng.random(3 * int(off[-1]), dtype=np.float32)).cuda()
    ids = torch.arange(int(off[-1]), dtype=torch.int32, device="cuda")
    mins, maxs = coords - 0.05, coords + 0.05
    want, refused = None, []
    for k in [-1] + list(range(40)):
        inject(k)
        try:
            b = F.Batch([3] * len(sizes), off, off)
        except F.FKDError as e:
            assert e.status == NOMEM
            refused.append(k)
            continue
        inject(-1)
        got = b.build(coords, ids).search_digest(mins, maxs)
        want = want or got
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), k
    inject(-1)
    assert len(refused) >= 15 and 1 <= max(refused) + 1 - len(refused) <= 2  # the bounding boxes, the boxes' order
