"""The calls a program makes through this package's public entry points, as cases that can be timed.

Each case is a dict of plain values; ``kind`` says which call it is:

* ``one``    -- fkd_search of a single host box, as the drop-in's search_in_the_box calls it (the reference
  driver's per-query loop).
* ``build``  -- FKDTree.build of device points, and the tables it leaves (fkd_get_tables) on the device.
* ``host``   -- from_points(...).build().tables() on host FKDPoint records: the whole call, copies included.
* ``boxes``  -- fkd_search of device boxes into buffers the program keeps: offsets and ids, in the
  reference's order (search_boxes' default).
* ``count``  -- count_boxes (search_in_the_box_multiple): result count of every box.
* ``radius`` -- fkd_search_radius of device centres into buffers the program keeps, in search_radius' default
  order.
* ``knn``    -- knn of device centres.
* ``batch``  -- Batch.run: many uneven events built and digest-searched in one call.

Points are ``uniform`` in the unit cube or ``clustered`` (80% in isotropic Gaussian clusters of sigma 0.002
with Dirichlet(1) weights, 20% uniform background: the generator of fkdtree_b200.workloads, drawn on the GPU
here); in 4D the fourth coordinate is one of 16 discrete layers, as in the mixed-dimension event batches.
Ids are a random permutation of 0..n-1.
"""
import ctypes
import math

import numpy as np
import torch

from fkdtree_b200 import Batch, FKDError, FKDTree, lib
from fkdtree_b200._capi import MEM_DEVICE, MEM_HOST

SIGMA = 0.002
CLUSTERED_SHARE = 0.8
LAYERS = 16
LAYER_HW = 0.04  # of a 4D box along the layer coordinate, at least


def listed():
    return [
        # one query at a time from a host loop: the reference driver's TBB loop body, where latency counts
        dict(name="one_box_100k", kind="one", n=100_000, dim=3, data="uniform", results=4.0),
        # the tree of one small event (detector hits of one collision), rebuilt for every event
        dict(name="build_2k", kind="build", n=1_999, dim=3, data="clustered"),
        # the reference's own example size: 100,000 uniform points
        dict(name="build_100k", kind="build", n=100_000, dim=3, data="uniform"),
        # 4D event with a discrete layer coordinate (many ties), odd size
        dict(name="build_4d_1m2", kind="build", n=1_234_567, dim=4, data="clustered"),
        # the large single event of the benchmark
        dict(name="build_16m", kind="build", n=16_777_216, dim=3, data="clustered"),
        # a host program switching from FKDTree_CPU: FKDPoint records in, tables out
        dict(name="host_points_50k", kind="host", n=50_001, dim=3, data="uniform"),
        # every point of the example event queries its neighbourhood (half-width 0.01)
        dict(name="boxes_100k", kind="boxes", n=100_000, q=100_000, dim=3, data="uniform", results=0.8),
        # large boxes (about 4,000 results each) on the large clustered event, ids written out
        dict(name="boxes_16m", kind="boxes", n=16_777_216, q=65_536, dim=3, data="clustered", hw_lo=0.001, hw_hi=0.02),
        # occupancy of a million boxes (search_in_the_box_multiple)
        dict(name="count_16m", kind="count", n=16_777_216, q=1_048_576, dim=3, data="clustered", hw_lo=0.001,
             hw_hi=0.02),
        # fixed-radius neighbours of a part of the points (clustering, isolation sums)
        dict(name="radius_1m", kind="radius", n=1_000_003, q=100_000, dim=3, data="clustered", r=0.004),
        # nearest neighbours of a million points of the large event
        dict(name="knn_16m", kind="knn", n=16_777_216, q=1_048_576, dim=3, data="clustered", k=16),
        # a block of uneven events, a quarter of them 4D, every point a box on its own event
        dict(name="batch_1024", kind="batch", events=1_024, median=20_000, frac_4d=0.25, hw=0.01, lanes=2),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["one", "build", "build", "host", "boxes", "boxes", "count", "radius", "knn", "batch"])
    dim = rng.choice([1, 2, 3, 3, 3] if kind == "radius" else [1, 2, 3, 3, 3, 4])
    data = rng.choice(["uniform", "clustered"])
    if kind == "one":
        return dict(kind=kind, n=_log_int(rng, 1_000, 4_000_000), dim=dim, data=data,
                    results=math.exp(rng.uniform(0.0, math.log(300.0))))
    if kind == "build":
        return dict(kind=kind, n=_log_int(rng, 500, 16_777_216), dim=dim, data=data)
    if kind == "host":
        return dict(kind=kind, n=_log_int(rng, 500, 1_000_000), dim=dim, data=data)
    n = _log_int(rng, 5_000, 16_777_216)
    if kind in ("boxes", "count"):
        q = _log_int(rng, 1_000, 1_048_576)
        c = dict(kind=kind, n=n, q=q, dim=dim, data=data)
        if data == "clustered" and dim >= 3 and n >= 1_000_000:
            c.update(hw_lo=0.001, hw_hi=0.02)
        else:
            c["results"] = min(math.exp(rng.uniform(0.0, math.log(2_000.0))), n / 64.0)
        if kind == "boxes":
            c["q"] = max(1_000, min(c["q"], int(2.5e8 / _expected_results(c))))  # at most 1 GB of ids
        return c
    if kind == "radius":
        n = min(n, 4_000_000)
        q = _log_int(rng, 1_000, 131_072)
        return dict(kind=kind, n=n, q=q, dim=dim, data="uniform",
                    r=_half_width(min(math.exp(rng.uniform(0.0, math.log(500.0))), n / 64.0), n, dim))
    if kind == "knn":
        k = _log_int(rng, 1, 64)
        return dict(kind=kind, n=n, q=_log_int(rng, 1_000, 16_777_216 // max(16, k)), dim=dim, data=data, k=k)
    return dict(kind=kind, events=_log_int(rng, 16, 768), median=_log_int(rng, 5_000, 25_000),
                frac_4d=rng.choice([0.0, 0.25, 0.5]), hw=rng.choice([0.005, 0.01]), lanes=rng.choice([0, 1, 2, 4]))


# ------------------------------------------------------------------ inputs


def _half_width(results, n, dim):
    """Half-width of a box that holds about `results` of n points uniform in the unit cube."""
    return 0.5 * min(1.0, results / n) ** (1.0 / dim)


def _points(gen, n, dim, data):
    """(dim, n) float32 on the GPU."""
    x = torch.rand((dim, n), generator=gen, device="cuda", dtype=torch.float32)
    if data == "clustered":
        k = max(8, min(4096, n // 64))
        m = int(round(n * CLUSTERED_SHARE))
        space = min(dim, 3)
        cuts = torch.sort(torch.rand(k - 1, generator=gen, device="cuda", dtype=torch.float64))[0]  # Dirichlet(1) weights
        which = torch.searchsorted(cuts, torch.rand(m, generator=gen, device="cuda", dtype=torch.float64))
        centre = torch.rand((space, k), generator=gen, device="cuda", dtype=torch.float32)
        put = torch.randperm(n, generator=gen, device="cuda")[:m]
        for c in range(space):
            noise = torch.randn(m, generator=gen, device="cuda", dtype=torch.float32)
            x[c, put] = centre[c, which] + SIGMA * noise
    if dim == 4:
        x[3] = torch.floor(x[3] * LAYERS) / LAYERS
    return x


def _ids(gen, n):
    return torch.randperm(n, generator=gen, device="cuda").to(torch.int32)


def _generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    return gen


def _tree(gen, case):
    x = _points(gen, case["n"], case["dim"], case["data"])
    ids = _ids(gen, case["n"])
    return x, ids, FKDTree(x, ids)


def _boxes(gen, case, x):
    """Boxes centred on random points (dim, q)."""
    q, dim, n = case["q"], case["dim"], case["n"]
    pick = torch.randint(0, n, (q,), generator=gen, device="cuda") if q != n else torch.arange(n, device="cuda")
    centre = x[:, pick]
    if "hw_lo" in case:
        hw = case["hw_lo"] + (case["hw_hi"] - case["hw_lo"]) * torch.rand((dim, q), generator=gen, device="cuda")
    else:
        hw = torch.full((dim, 1), _half_width(case["results"], n, dim), device="cuda")
    if dim == 4:
        hw = hw.expand(dim, q).clone()
        hw[3] = torch.clamp(hw[3], min=LAYER_HW)  # at least the box's own layer
    return (centre - hw).contiguous(), (centre + hw).contiguous()


def _event_sizes(case):
    rng = np.random.default_rng(case["events"] * 1_000_003 + case["median"])
    s = np.exp(np.log(case["median"]) + rng.standard_normal(case["events"]))
    return np.clip(np.rint(s), 1_000, 200_000).astype(np.int64)


def _batch_events(gen, case, seed):
    """Flat coordinates / ids of the events in Batch's layout, and the boxes (one per point)."""
    sizes = _event_sizes(case)
    ne = len(sizes)
    dims = np.where(np.arange(ne) < round(case["frac_4d"] * ne), 4, 3).astype(np.int64)
    pt_off = np.concatenate([[0], np.cumsum(sizes)])
    coff = np.concatenate([[0], np.cumsum(sizes * dims)])
    total = int(pt_off[-1])
    sz = torch.from_numpy(sizes).cuda()
    ev = torch.repeat_interleave(torch.arange(ne, device="cuda"), sz, output_size=total)
    local = torch.arange(total, device="cuda") - torch.from_numpy(pt_off[:-1]).cuda()[ev]
    # 50-500 clusters per event with Dirichlet(1) weights: random cuts of the event's own unit interval
    rng = np.random.default_rng(int(seed) + 1)
    cuts = rng.integers(50, 501, ne) - 1
    owner = torch.repeat_interleave(torch.arange(ne, device="cuda", dtype=torch.float64), torch.from_numpy(cuts).cuda(),
                                    output_size=int(cuts.sum()))
    edges = torch.sort(owner + torch.rand(len(owner), generator=gen, device="cuda", dtype=torch.float64))[0]
    u = ev.to(torch.float64) + torch.rand(total, generator=gen, device="cuda", dtype=torch.float64)
    which = torch.searchsorted(edges, u) + ev
    centre = torch.rand((3, len(owner) + ne), generator=gen, device="cuda", dtype=torch.float32)
    member = torch.rand(total, generator=gen, device="cuda") < CLUSTERED_SHARE
    coords = torch.empty(int(coff[-1]), dtype=torch.float32, device="cuda")
    at = torch.from_numpy(coff[:-1]).cuda()[ev] + local
    for c in range(3):
        near = centre[c, which] + SIGMA * torch.randn(total, generator=gen, device="cuda", dtype=torch.float32)
        coords[at + c * sz[ev]] = torch.where(member, near, torch.rand(total, generator=gen, device="cuda"))
    four = torch.from_numpy(dims).cuda()[ev] == 4
    layer = torch.randint(0, LAYERS, (total,), generator=gen, device="cuda").to(torch.float32) / LAYERS
    coords[(at + 3 * sz[ev])[four]] = layer[four]
    return dims, pt_off, coords, local.to(torch.int32)


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    if kind == "batch":
        dims, pt_off, coords, ids = _batch_events(gen, case, seed)
        hw = case["hw"]
        b = Batch(dims, pt_off, pt_off)
        b.set_param("search_lanes", case["lanes"])  # what the autotuner chooses for events of this size
        total = int(pt_off[-1])
        st = dict(case=case, batch=b, coords=coords, ids=ids, mins=coords - hw, maxs=coords + hw,
                  counts=torch.empty(total, dtype=torch.int32, device="cuda"),
                  digests=torch.empty(total, dtype=torch.int64, device="cuda"))
        torch.cuda.synchronize()  # the batch runs on a stream of its own
        return st
    if kind == "host":
        x = _points(gen, case["n"], case["dim"], case["data"])
        rec = torch.cat([x, _ids(gen, case["n"]).view(torch.float32)[None]]).t().contiguous().cpu().numpy()
        return dict(case=case, tree=FKDTree.from_points(rec, case["dim"]))
    x, ids, tree = _tree(gen, case)
    st = dict(case=case, tree=tree)
    if kind == "build":
        n, dim = case["n"], case["dim"]
        st.update(tab=torch.empty((dim, n), dtype=torch.float32, device="cuda"),
                  tab_ids=torch.empty(n, dtype=torch.int32, device="cuda"))
        return st
    tree.build()
    if kind == "one":
        lo, hi = _boxes(gen, dict(case, q=1), x)
        st.update(mins=lo.cpu().numpy(), maxs=hi.cpu().numpy(), offsets=np.zeros(2, np.uint64),
                  ids=np.zeros(4096, np.uint32))
    elif kind in ("boxes", "count"):
        st["mins"], st["maxs"] = _boxes(gen, case, x)
    else:
        pick = torch.randint(0, case["n"], (case["q"],), generator=gen, device="cuda")
        st["centres"] = x[:, pick].contiguous()
        if kind == "radius":
            st["radii"] = torch.full((case["q"],), case["r"], dtype=torch.float32, device="cuda")
    if kind in ("boxes", "radius"):
        room = int(2.0 * case["q"] * _expected_results(case)) + 64 * case["q"]
        st.update(offsets=torch.zeros(case["q"] + 1, dtype=torch.int64, device="cuda"),
                  ids=torch.zeros(room, dtype=torch.int32, device="cuda"))
    return st


# -------------------------------------------------------------------- calls


def _ok(status):
    if status:
        raise FKDError(status, lib().fkd_last_error().decode())


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        state["batch"].run(state["coords"], state["ids"], state["mins"], state["maxs"], state["counts"],
                           state["digests"])
        return dict(counts=state["counts"], digests=state["digests"])
    tree = state["tree"]
    if kind == "build":
        tree.build()
        _ok(lib().fkd_get_tables(tree._h, state["tab"].data_ptr(), state["tab_ids"].data_ptr(), MEM_DEVICE))
        return dict(tab=state["tab"], ids=state["tab_ids"])
    if kind == "host":
        tab, ids = tree.build().tables()
        return dict(tab=tab, ids=ids)
    if kind == "count":
        return tree.count_boxes(state["mins"], state["maxs"])
    if kind == "knn":
        ids, d2 = tree.knn(state["centres"], case["k"])
        return dict(ids=ids, d2=d2)
    total = ctypes.c_uint64(0)
    offsets, out = state["offsets"], state["ids"]
    if kind == "one":
        _ok(lib().fkd_search(tree._h, state["mins"].ctypes.data, state["maxs"].ctypes.data, 1, offsets.ctypes.data,
                             out.ctypes.data, out.size, ctypes.byref(total), 1, MEM_HOST))
    elif kind == "boxes":
        _ok(lib().fkd_search(tree._h, state["mins"].data_ptr(), state["maxs"].data_ptr(), case["q"],
                             offsets.data_ptr(), out.data_ptr(), out.numel(), ctypes.byref(total), 1, MEM_DEVICE))
    else:
        _ok(lib().fkd_search_radius(tree._h, state["centres"].data_ptr(), state["radii"].data_ptr(), case["q"],
                                    offsets.data_ptr(), out.data_ptr(), out.numel(), ctypes.byref(total), 1,
                                    MEM_DEVICE))
    return dict(total=total.value, offsets=offsets, ids=out)


# --------------------------------------------------------------------- work


def _near(lo, hi):
    """Mean over h in [lo, hi] of P(|a - b| < h), a and b members of one cluster along one dimension."""
    hs = [lo + (hi - lo) * (i + 0.5) / 64 for i in range(64)]
    return sum(math.erf(h / (2.0 * SIGMA)) for h in hs) / 64


def _expected_results(case):
    """Expected results of a box (or ball) centred on a random point."""
    n, dim = case["n"], case["dim"]
    space = min(dim, 3)
    lo, hi = case.get("hw_lo"), case.get("hw_hi")
    if lo is None:
        lo = hi = case["r"] if "r" in case else _half_width(case["results"], n, dim)
    layers = min(1.0, (2 * int(LAYERS * max(lo, LAYER_HW)) + 1) / LAYERS) if dim == 4 else 1.0
    uniform = n * min(1.0, lo + hi) ** space * layers
    near = _near(lo, hi) ** space
    if "r" in case:
        uniform *= (1.0, math.pi / 4.0, math.pi / 6.0)[dim - 1]
        if dim == 3:  # Maxwell distribution of the distance of two members
            x = lo / (SIGMA * math.sqrt(2.0))
            near = math.erf(x / math.sqrt(2.0)) - math.sqrt(2.0 / math.pi) * x * math.exp(-x * x / 2.0)
    if case["data"] != "clustered":
        return max(1.0, uniform)
    k = max(8, min(4096, n // 64))
    own = CLUSTERED_SHARE * n * 2.0 / (k + 1) * near * layers
    return max(1.0, uniform + CLUSTERED_SHARE * own)


def work(case):
    """Bytes every implementation reads and writes once, and the coordinate arithmetic of the kNN answer."""
    kind = case["kind"]
    if kind == "batch":
        # points (with their boxes) in, count and digest of every box out
        sizes = _event_sizes(case)
        ne = len(sizes)
        dims = np.where(np.arange(ne) < round(case["frac_4d"] * ne), 4, 3)
        return dict(bytes=float((sizes * (4 * dims + 4 + 8 * dims + 12)).sum()), flops=0)
    n, dim = case["n"], case["dim"]
    rec = 4 * dim + 4
    if kind in ("build", "host"):
        return dict(bytes=2.0 * n * rec, flops=0)
    if kind == "one":
        return dict(bytes=8.0 * dim + case["results"] * (rec + 4), flops=0)
    q = case["q"]
    if kind == "knn":
        # the tree or the k neighbours of every query, whichever is less; ids and distances out
        return dict(bytes=min(float(n), float(q) * case["k"]) * rec + q * (4.0 * dim + 8.0 * case["k"]),
                    flops=3.0 * dim * q * case["k"])
    res = q * _expected_results(case)
    tree = min(float(n), res) * rec
    if kind == "count":
        return dict(bytes=tree + q * (8.0 * dim + 4), flops=0)
    return dict(bytes=tree + q * (8.0 * dim + 8) + 4.0 * res, flops=0)


# -------------------------------------------------------------------- exact


def _exact_tree(x, ids):
    """The complete tree in heap order by sorting every level: (dim, n) coordinates, ids."""
    dim, n = x.shape
    order = torch.argsort(ids)
    x, ids = x[:, order], ids[order]  # points by id, so that stable sorts break ties by id
    height = n.bit_length() - 1
    last = n - ((1 << height) - 1)
    seg = torch.zeros(n, dtype=torch.int64, device=x.device)  # first in-order position of a point's interval
    heap = torch.empty(n, dtype=torch.int64, device=x.device)
    placed = torch.zeros(n, dtype=torch.bool, device=x.device)
    for d in range(height + 1):
        by = torch.sort(x[d % dim] + 0.0, stable=True)[1]
        by = by[torch.sort(seg[by], stable=True)[1]]  # in-order position -> point
        w = 1 << (height - d)
        t = torch.arange(1 << d, device=x.device)
        start = t * w + torch.clamp(t * w, max=last)
        rank = w // 2 - 1 + torch.clamp(last - t * w, min=0, max=w // 2) if d < height else torch.zeros_like(t)
        if d == height:
            t, start, rank = t[:last], start[:last], rank[:last]
        pos = start + rank
        pivot = by[pos]
        heap[pivot] = (1 << d) - 1 + t
        placed[pivot] = True
        seg[pivot] = pos
        # the points after a pivot inside its interval start a new one
        if d < height:
            begin = torch.zeros(n, dtype=torch.int64, device=x.device)
            begin[pos] = pos
            begin[(pos + 1)[pos + 1 < n]] = (pos + 1)[pos + 1 < n]
            begin[start[rank > 0]] = start[rank > 0]
            first = torch.cummax(begin, 0)[0]
            keep = ~placed[by]
            seg[by[keep]] = first[keep]
    out = torch.empty_like(x)
    out[:, heap] = x
    oid = torch.empty_like(ids)
    oid[heap] = ids
    return out, oid


def exact(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    if kind == "build":
        x = _points(gen, case["n"], case["dim"], case["data"])
        tab, ids = _exact_tree(x, _ids(gen, case["n"]))
        return dict(tab=tab.to(torch.float64), ids=ids)
    if kind == "host":
        x = _points(gen, case["n"], case["dim"], case["data"])
        tab, ids = _exact_tree(x, _ids(gen, case["n"]))
        return dict(tab=tab.to(torch.float64).cpu(), ids=ids.cpu())
    if kind == "knn" and case["n"] * case["q"] <= 4e10:
        x = _points(gen, case["n"], case["dim"], case["data"])
        _ids(gen, case["n"])
        pick = torch.randint(0, case["n"], (case["q"],), generator=gen, device="cuda")
        p = x.to(torch.float64)
        c = p[:, pick]
        rows = []
        step = max(1, int(2.5e8 // case["n"]))
        for j in range(0, case["q"], step):
            d2 = sum((p[a][None, :] - c[a, j:j + step][:, None]) ** 2 for a in range(case["dim"]))
            rows.append(torch.topk(d2, min(case["k"], case["n"]), largest=False)[0])
        return dict(ids=None, d2=torch.cat(rows))
    return None
