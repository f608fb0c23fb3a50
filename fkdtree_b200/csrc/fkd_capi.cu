// fkd_capi.cu -- the C ABI (include/fkdtree_b200.h) over the build and search
// kernels: handle lifetime, device buffers, host staging and error latching.
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "../../include/fkdtree_b200.h"
#include "fkd_internal.h"
#include "fkd_plan.h"
#include "fkd_mlp.h"

using namespace fkd;

namespace fkd {
fkd_status capi_fail(fkd_status s, const std::string& msg);
fkd_status capi_status_from_err(uint32_t e, const char* what);
static unsigned long long g_launches = 0;
void count_launches(uint64_t k) { __atomic_fetch_add(&g_launches, (unsigned long long)k, __ATOMIC_RELAXED); }
uint64_t launches_total() { return __atomic_load_n(&g_launches, __ATOMIC_RELAXED); }

// Allocation failure injection (fkd_debug_fail_alloc): >= 0 counts down the
// device allocations left before one fails; -1 (the default) is off.
// fkd_debug_fail_launch: the same for chained launches.
static int g_fail_alloc = -1, g_fail_launch = -1;
static bool count_down(int& left) {  // true: this one fails
  int v = __atomic_load_n(&left, __ATOMIC_RELAXED);
  while (v >= 0) {
    if (__atomic_compare_exchange_n(&left, &v, v - 1, false, __ATOMIC_RELAXED, __ATOMIC_RELAXED)) return v == 0;
  }
  return false;
}
cudaError_t device_alloc(void** p, size_t bytes) {
  if (count_down(g_fail_alloc)) {
    *p = nullptr;
    return cudaErrorMemoryAllocation;
  }
  const cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaSuccess) (void)cudaGetLastError();  // in the status, not in a later call's
  return e;
}
cudaError_t launch_injected() { return count_down(g_fail_launch) ? cudaErrorLaunchOutOfResources : cudaSuccess; }
}  // namespace fkd

namespace {

thread_local std::string g_last_error;

fkd_status fail(fkd_status s, const std::string& msg) {
  g_last_error = msg;
  return s;
}

#define FKD_CUDA(call)                                                                                    \
  do {                                                                                                    \
    cudaError_t e_ = (call);                                                                              \
    if (e_ != cudaSuccess)                                                                                \
      return fail(e_ == cudaErrorMemoryAllocation ? FKD_ERR_NOMEM : FKD_ERR_CUDA,                         \
                  std::string(#call) + ": " + cudaGetErrorString(e_));                                    \
  } while (0)

struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  cudaError_t ensure(size_t want) {
    if (want <= bytes && p) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
    if (want == 0) return cudaSuccess;
    cudaError_t e = device_alloc(&p, want);
    if (e == cudaSuccess) bytes = want;
    return e;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
  }
  template <class T>
  T* as() const {
    return (T*)p;
  }
};

}  // namespace

// Per-call scratch of the searches.  Every search call leases one slot from
// its handle's pool for its duration, so searches on one built tree may run
// from several host threads at once (the reference's TBB loop over one tree,
// main.cpp:351-359): each has its own staging buffers, error word and -- for
// host-memory calls -- its own stream; the tree tables are only read.
// The words of SearchSlot::err.  Word 0 stays until it is reported; the others
// are cleared at the start of a call, in one go, and the first CTL_HOST come
// back to the host in one copy.
enum : uint32_t {
  CTL_TOTAL = 2,    // results of the call (64 bits)
  CTL_ENTS = 4,     // record entries wanted (64 bits)
  CTL_FLAGS = 6,    // boxes whose record did not fit (64 bits)
  CTL_HOST = 8,
  CTL_LOOSE = 8,    // boxes of packets that gave up (64 bits)
  CTL_QUEUE = 10,   // work counters (QC_COUNT)
  CTL_TICKET = 16,  // two scans' tickets
  CTL_WORDS = 20
};
static_assert(CTL_QUEUE + QC_COUNT <= CTL_TICKET, "work counters");

struct SearchSlot {
  DevBuf qlo, qhi, counts, offsets, partials, out, tmp, digests, qorder;
  DevBuf rec;                    // a recording count pass: what it keeps per box, then the entry pool
  DevBuf one, loose;
  DevBuf err;                    // CTL_WORDS words: the error word, then what a call counts (CTL_*)
  uint32_t* herr = nullptr;      // pinned mirror of err's first CTL_HOST words
  uint32_t* hone = nullptr;      // pinned: the single-box search's count, flag and first ids
  cudaStream_t own = nullptr;    // stream of host-memory calls
  cudaEvent_t done = nullptr;    // the slot's last work (waited on by its next lease)
  uint64_t ent_cap = 0;          // entries of the last call's pool
  uint64_t ent_want = 0;         // the demand of a call that did not fit
  bool demand_due = false;       // an asynchronous call's demand is on its way to herr
  ~SearchSlot() {
    DevBuf* all[] = {&qlo, &qhi, &counts, &offsets, &partials, &out, &tmp, &digests, &qorder,
                     &rec, &err, &one, &loose};
    if (own) cudaStreamSynchronize(own);
    for (DevBuf* b : all) b->release();
    if (herr) cudaFreeHost(herr);
    if (hone) cudaFreeHost(hone);
    if (done) cudaEventDestroy(done);
    if (own) cudaStreamDestroy(own);
  }
};

struct fkd_tree_s {
  int dim = 3;
  uint32_t flags = 0;
  cudaStream_t stream = nullptr;
  int device = 0;
  uint64_t n = 0;
  bool built = false;
  DevBuf nodes, ids, work0, work1, sel, ghist, err, passflags, tmp;
  uint32_t* herr = nullptr;  // pinned mirror of err
  PlanDev plan;              // build plan of the last size built
  uint64_t plan_n = ~0ull;
  uint32_t hist_ctas = 0;    // digit-pass CTAs per level (0: four per SM)
  uint32_t search_lanes = 0; // count / digest lanes per box (0: one warp)
  int subtree = 0;           // subtree kernel: 0 auto, 1 radix select, 2 presorted lists
  int subtree_size = 0;      // presorted subtree size: 0 (1,024), 512 or 1,024 ("subtree_size")
  bool small_select = true;  // one CTA per segment on levels of small segments
  bool box_order = true;     // search boxes in the spatial order of their centres
  fkd_mlp mlp = nullptr;     // learned split (null: plain radix select)
  float mlp_delta = 0.f;
  DevBuf lfeat, lyhat, lrange, lstats, sdig, inord, bnd, tiebuf;
  bool small_fix = true;        // selects stop at SMALL_CAP candidates, the partition orders them ("small_fix")
  bool lin_pass = true;         // a segment's first digit pass bins its value range linearly ("lin_pass")
  uint32_t search_bucket = 5;   // leaf-bucket height of the searches ("search_bucket"; 0: walk every level)
  uint32_t search_bucket_grp = 0;  // ... of the searches with fewer than 32 lanes per box ("search_bucket_lanes")
  bool search_record = true;    // fkd_search records the results in the count pass ("search_record")
  bool search_one = true;       // fkd_search of one host-memory box: one level-order warp ("search_one")
  bool search_packets = true;   // count / digest: neighbouring boxes walk together ("search_packets")
  uint64_t search_pool = 0;     // fixed pool entries ("search_pool"; 0: sized by demand)
  // tables derived from the tree on first use (in-order ids / heap indices /
  // nodes, subtree digests), built once under tree_mu; the events mark them ready
  bool sdig_valid = false;
  bool inorder_valid = false;
  bool ipts_valid = false;
  // ns that kNN and radius calls would have gained from the in-order tables (tables_pay): on this
  // tree, and since the handle was made
  uint64_t nn_rent = 0, nn_rent_all = 0;
  std::mutex tree_mu;
  cudaEvent_t built_ev = nullptr, inorder_ev = nullptr, sdig_ev = nullptr;
  // search slots (SearchSlot): all of them, and the ones not leased
  std::mutex slot_mu;
  std::vector<std::unique_ptr<SearchSlot>> slots;
  std::vector<SearchSlot*> free_slots;
  std::mutex tab_mu;  // fkd_get_tables stages through work0
  // optional per-kernel timing (fkd_set_param "kernel_events"): a ring of
  // KEV_RING event sets, one per build / search call
  static constexpr uint32_t KEV_RING = 64;
  std::vector<cudaEvent_t> kev;  // [slot * 7 + k]: 0 count start, 1 count end, 2 write start, 3 write end,
                                 //                  4 build start, 5 subtree start, 6 build end
  uint64_t kev_builds = 0, kev_searches = 0;

  ~fkd_tree_s() {
    slots.clear();
    DevBuf* all[] = {&nodes, &ids, &work0, &work1, &sel, &ghist, &err, &passflags, &tmp,
                     &lfeat, &lyhat, &lrange, &lstats, &sdig, &inord, &bnd, &tiebuf};
    for (DevBuf* b : all) b->release();
    if (herr) cudaFreeHost(herr);
    for (cudaEvent_t e : kev) cudaEventDestroy(e);
    for (cudaEvent_t e : {built_ev, inorder_ev, sdig_ev})
      if (e) cudaEventDestroy(e);
  }
  cudaEvent_t kev_at(uint64_t call, int k) { return kev[(size_t)(call % KEV_RING) * 7 + k]; }
};

namespace {

fkd_status status_from_err(uint32_t e, const char* what) {
  if (e == 0) return FKD_OK;
  char buf[160];
  if (e & ERRB_NAN) {
    snprintf(buf, sizeof buf, "%s: input coordinates contain NaN", what);
    return fail(FKD_ERR_NAN, buf);
  }
  if (e & ERRB_CAPACITY) {
    snprintf(buf, sizeof buf, "%s: a result or frontier capacity was exceeded", what);
    return fail(FKD_ERR_CAPACITY, buf);
  }
  if (e & ERRB_TIMEOUT) {
    snprintf(buf, sizeof buf, "%s: a bounded device wait gave up", what);
    return fail(FKD_ERR_TIMEOUT, buf);
  }
  snprintf(buf, sizeof buf, "%s: device consistency check failed (0x%x)", what, e);
  return fail(FKD_ERR_INTERNAL, buf);
}

// Reads the handle's (build) error word and clears it.
fkd_status check_err_word(fkd_tree h, const char* what) {
  FKD_CUDA(cudaMemcpyAsync(h->herr, h->err.p, sizeof(uint32_t), cudaMemcpyDeviceToHost, h->stream));
  FKD_CUDA(cudaMemsetAsync(h->err.p, 0, sizeof(uint32_t), h->stream));
  FKD_CUDA(cudaStreamSynchronize(h->stream));
  return status_from_err(*h->herr, what);
}

fkd_status finish(fkd_tree h, const char* what, int mem) {
  if (mem == FKD_MEM_DEVICE && (h->flags & FKD_FLAG_ASYNC)) return FKD_OK;
  return check_err_word(h, what);
}

Table table_of(fkd_tree h) { return Table{h->nodes.as<uint4>(), h->ids.as<uint32_t>()}; }

// Makes the calling thread's current device the handle's for one call.
struct DeviceScope {
  int prev = -1;
  explicit DeviceScope(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess || prev == dev) prev = -1;
    else cudaSetDevice(dev);
  }
  ~DeviceScope() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

// One search call's slot and stream.  Device-memory calls run on the
// handle's stream (stream-ordered with the caller's work); host-memory calls
// are synchronous and run on the slot's own stream, so concurrent ones
// overlap on the GPU.  Every lease first waits for the slot's previous work
// and for the last build; release records the slot's completion event and
// returns it to the pool.
struct Lease {
  fkd_tree h = nullptr;
  SearchSlot* s = nullptr;
  cudaStream_t st = nullptr;
  ~Lease() {
    if (!s) return;
    cudaEventRecord(s->done, st);
    std::lock_guard<std::mutex> g(h->slot_mu);
    h->free_slots.push_back(s);
  }
};

fkd_status lease_slot(fkd_tree h, int mem, Lease* L) {
  SearchSlot* s = nullptr;
  {
    std::lock_guard<std::mutex> g(h->slot_mu);
    if (!h->free_slots.empty()) {
      s = h->free_slots.back();
      h->free_slots.pop_back();
    }
  }
  if (!s) {
    std::unique_ptr<SearchSlot> ns(new (std::nothrow) SearchSlot());
    if (!ns) return fail(FKD_ERR_NOMEM, "host allocation failed");
    FKD_CUDA(cudaStreamCreateWithFlags(&ns->own, cudaStreamNonBlocking));
    FKD_CUDA(cudaEventCreateWithFlags(&ns->done, cudaEventDisableTiming));
    FKD_CUDA(ns->err.ensure(sizeof(uint32_t) * CTL_WORDS));
    FKD_CUDA(cudaMallocHost((void**)&ns->herr, sizeof(uint32_t) * CTL_HOST));
    FKD_CUDA(cudaMemsetAsync(ns->err.p, 0, sizeof(uint32_t) * CTL_WORDS, ns->own));
    FKD_CUDA(cudaEventRecord(ns->done, ns->own));
    s = ns.get();
    std::lock_guard<std::mutex> g(h->slot_mu);
    h->slots.push_back(std::move(ns));
  }
  L->h = h;
  L->s = s;
  L->st = mem == FKD_MEM_DEVICE ? h->stream : s->own;
  FKD_CUDA(cudaStreamWaitEvent(L->st, s->done, 0));
  if (L->st != h->stream) FKD_CUDA(cudaStreamWaitEvent(L->st, h->built_ev, 0));
  return FKD_OK;
}

// The error word of a slot whose control words have come back (an error latched
// by an earlier asynchronous call that used the slot is reported here too).
fkd_status report_slot_err(const Lease& L, const char* what) {
  const uint32_t e = *L.s->herr;
  if (e != 0) {
    FKD_CUDA(cudaMemsetAsync(L.s->err.p, 0, sizeof(uint32_t), L.st));
    FKD_CUDA(cudaStreamSynchronize(L.st));
  }
  return status_from_err(e, what);
}

// Brings the control words to the host and waits for them.
fkd_status fetch_ctl(const Lease& L) {
  FKD_CUDA(cudaMemcpyAsync(L.s->herr, L.s->err.p, sizeof(uint32_t) * CTL_HOST, cudaMemcpyDeviceToHost, L.st));
  FKD_CUDA(cudaStreamSynchronize(L.st));
  return FKD_OK;
}

// Clears what a call counts.
fkd_status clear_ctl(const Lease& L) {
  FKD_CUDA(cudaMemsetAsync(L.s->err.as<uint32_t>() + 1, 0, sizeof(uint32_t) * (CTL_WORDS - 1), L.st));
  return FKD_OK;
}

fkd_status check_slot_err(const Lease& L, const char* what) {
  const fkd_status s = fetch_ctl(L);
  return s != FKD_OK ? s : report_slot_err(L, what);
}

fkd_status finish_search(fkd_tree h, const Lease& L, const char* what, int mem) {
  if (mem == FKD_MEM_DEVICE && (h->flags & FKD_FLAG_ASYNC)) return FKD_OK;
  return check_slot_err(L, what);
}

__global__ void k_tables_out(uint32_t n, int dim, const uint4* __restrict__ nodes, float* __restrict__ tab) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint4 v = nodes[i];
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  for (int c = 0; c < dim; ++c) tab[(uint64_t)c * n + i] = __uint_as_float(w[c]);
}

// Stages host boxes (or aliases device boxes).
fkd_status stage_boxes(fkd_tree h, const Lease& L, const float* mins, const float* maxs, uint64_t q, int mem,
                       Boxes* b) {
  b->q = q;
  b->stride = q;
  if (mem == FKD_MEM_DEVICE) {
    b->lo = mins;
    b->hi = maxs;
    return FKD_OK;
  }
  SearchSlot* s = L.s;
  const size_t bytes = (size_t)h->dim * q * sizeof(float);
  FKD_CUDA(s->qlo.ensure(bytes ? bytes : 4));
  FKD_CUDA(s->qhi.ensure(bytes ? bytes : 4));
  if (bytes) {
    FKD_CUDA(cudaMemcpyAsync(s->qlo.p, mins, bytes, cudaMemcpyHostToDevice, L.st));
    FKD_CUDA(cudaMemcpyAsync(s->qhi.p, maxs, bytes, cudaMemcpyHostToDevice, L.st));
  }
  b->lo = s->qlo.as<float>();
  b->hi = s->qhi.as<float>();
  return FKD_OK;
}

// The tables derived from a tree for the searches, in one allocation (a first
// search on a new handle pays for every cudaMalloc): bounding boxes, the
// in-order copy of the nodes when wanted, ids in in-order position.
size_t inorder_bytes(uint64_t n, bool ipts) {
  return bb_nodes(n, 1) * 2 * sizeof(float4) + (ipts ? n * sizeof(uint4) : 0) + n * sizeof(uint32_t);
}
Table inorder_tables(fkd_tree h, bool ipts) {
  Table t = table_of(h);
  t.bb = h->inord.as<float4>();
  uint4* p = (uint4*)(t.bb + bb_nodes(h->n, 1) * 2);
  t.ipts = ipts ? p : nullptr;
  t.dids = (uint32_t*)(ipts ? p + h->n : p);
  return t;
}

SearchCtx search_ctx(fkd_tree h, const Lease& L, const Boxes& b) {
  SearchCtx sc;
  memset(&sc, 0, sizeof sc);
  sc.g = make_geom((uint32_t)h->n);
  sc.tab = table_of(h);
  if (h->inorder_valid) {
    Table t = inorder_tables(h, h->ipts_valid);
    sc.tab.bb = t.bb;
    sc.tab.dids = t.dids;
    sc.tab.ipts = t.ipts;
  }
  if ((h->search_bucket || h->search_bucket_grp) && sc.tab.ipts) {
    sc.bucket = h->search_bucket;
    sc.bucket_grp = h->search_bucket_grp;
  }
  sc.boxes = b;
  sc.qcounter = L.s->err.as<uint32_t>() + CTL_QUEUE;
  sc.qready = 1;
  sc.err = L.s->err.as<uint32_t>();
  sc.stream = L.st;
  sc.capacity = ~0ull;
  sc.lanes = h->search_lanes;
  return sc;
}

fkd_status check_search_args(fkd_tree h, const float* mins, const float* maxs, uint64_t q, int mem) {
  if (!h) return fail(FKD_ERR_ARG, "null handle");
  if (!h->built) return fail(FKD_ERR_STATE, "search before build");
  if (mem != FKD_MEM_HOST && mem != FKD_MEM_DEVICE) return fail(FKD_ERR_ARG, "mem must be FKD_MEM_HOST or FKD_MEM_DEVICE");
  if (q > 0xffffffffull) return fail(FKD_ERR_ARG, "at most 2^32-1 boxes per call");
  if (q && (!mins || !maxs)) return fail(FKD_ERR_ARG, "null box bounds");
  return FKD_OK;
}

// Boxes below this count are searched in the caller's order: a spatial order
// only pays when many boxes share the tree's cache lines.
constexpr uint64_t BOX_ORDER_MIN = 4096;

// Spatial processing order of the boxes (fkd_search.cu: launch_box_order).
// start (optional): where their walks may begin.
fkd_status box_order(fkd_tree h, const Lease& L, const Boxes& b, const uint32_t** order,
                     const uint32_t** start = nullptr) {
  *order = nullptr;
  if (start) *start = nullptr;
  if (!h->box_order || b.q < BOX_ORDER_MIN) return FKD_OK;
  FKD_CUDA(L.s->qorder.ensure(box_order_words(b.q) * sizeof(uint32_t)));
  uint32_t* o = nullptr;
  uint32_t* st = nullptr;
  FKD_CUDA(launch_box_order(make_geom((uint32_t)h->n), table_of(h), b, h->dim, L.s->qorder.as<uint32_t>(), &o, L.st,
                            start ? &st : nullptr, L.s->err.as<uint32_t>() + CTL_TICKET));
  if (start) *start = st;
  *order = o;
  return FKD_OK;
}

// Packets (fkd_packet.cu) need the boxes' spatial order, enough of them to
// fill the GPU with warps of 32 boxes, and neighbours near enough to share
// subtrees: up to eight points per box in 1-D and 2-D, fewer where the walk beats
// them sooner -- in 3-D and 4-D, the more so the more of the leaf buckets are
// without points of the last level, which a walk tests in pairs and a packet, one
// point per lane, does not (f: the share that reaches into it).  Counts on one B200,
// packets against a warp per box (us):
//   boxes / points      262,144 / 1M  400,000 / 0.3M  524,288 / 1M   1M / 1M      1M / 4M      1M / 8M        1M / 2^24
//   10 results          296 / 253     308 / 352       406 / 441      568 / 776    801 / 827    1,011 / 855    1,581 / 975
//   500 results         842 / 822     900 / 1,177     1,181 / 1,559  1,791 / 2,869  2,331 / 3,145  3,006 / 3,164  4,992 / 3,613
//   mixed, clustered    372 / 353     301 / 344       502 / 618      762 / 1,110  1,754 / 2,096  3,057 / 3,082  7,639 / 5,304
//   3-D, f = 0, 100 results   400,000 / 2^19  557 / 647   400,000 / 2^20  739 / 673   600,000 / 2^22  1,314 / 1,015
//        f = 0.5              600,000 / 1.6M  874 / 967   400,000 / 1.6M  708 / 678
//   4-D, f = 0                1M / 2^20  2,733 / 2,733    600,000 / 2^20  1,984 / 1,674   1M / 2^22  4,243 / 3,003
//        f = 0.9              600,000 / 1M  1,521 / 1,662    600,000 / 4M  2,293 / 1,785
constexpr uint64_t PACKET_MIN = 393216;
bool in_packets(fkd_tree h, uint64_t q) {
  const Geom g = make_geom((uint32_t)h->n);
  // points per box, in eighths
  const uint64_t sparse = h->dim <= 2 ? 64u : h->dim == 3 ? 16u + (48ull * g.M >> g.H) : 8u + (32ull * g.M >> g.H);
  return h->search_packets && q >= PACKET_MIN && q * sparse >= 8u * h->n;
}

// Count / digest search of sc: in packets where that pays, else each box
// alone; node by node when there was no room for the bounding boxes.
fkd_status search_shared(fkd_tree h, const Lease& L, SearchCtx& sc, int mode) {
  if (!sc.tab.bb) {
    if (sc.lanes == 0 || sc.lanes == 32) sc.lanes = 16;
  } else if (sc.order && in_packets(h, sc.boxes.q) &&
             L.s->loose.ensure(sc.boxes.q * sizeof(uint32_t)) == cudaSuccess) {
    sc.loose = L.s->loose.as<uint32_t>();
    sc.loose_ctr = (unsigned long long*)(L.s->err.as<uint32_t>() + CTL_LOOSE);
    FKD_CUDA(launch_packets(sc, h->dim, mode));
    return FKD_OK;
  }
  FKD_CUDA(launch_search(sc, h->dim, mode));
  return FKD_OK;
}

// count pass into dcounts (device); rec (optional): the entry pool fields of a
// recording count pass
fkd_status count_pass(fkd_tree h, const Lease& L, const Boxes& b, uint32_t* dcounts, const uint32_t* order,
                      const uint32_t* start, const SearchCtx* rec = nullptr) {
  SearchCtx sc = search_ctx(h, L, b);
  sc.counts = dcounts;
  sc.order = order;
  sc.start = start;
  if (rec) {
    sc.ents = rec->ents;
    sc.ent_ctr = rec->ent_ctr;
    sc.ent_cap = rec->ent_cap;
    sc.erec = rec->erec;
    sc.ehist = rec->ehist;
    sc.flags = rec->flags;
    sc.flag_ctr = rec->flag_ctr;
    FKD_CUDA(launch_walk(sc, h->dim, SEARCH_COUNT));
    return FKD_OK;
  }
  return search_shared(h, L, sc, SEARCH_COUNT);
}

// In-order ids and the subtrees' bounding boxes of the
// current tree -- and, with leaf buckets on, the in-order copy of the nodes --
// built once per tree by the
// first search that needs them; every caller's stream then waits for them.
fkd_status ensure_inorder(fkd_tree h, cudaStream_t st) {
  if (h->n == 0) return FKD_OK;
  {
    std::lock_guard<std::mutex> g(h->tree_mu);
    const bool want_ipts = h->search_bucket != 0 || h->search_bucket_grp != 0;
    if (!h->inorder_valid || (want_ipts && !h->ipts_valid)) {
      // a larger block takes the place of the tables (the copy of the nodes is wanted now): until it is
      // filled there are none, whatever fails on the way
      h->inorder_valid = h->ipts_valid = false;
      FKD_CUDA(h->inord.ensure(inorder_bytes(h->n, want_ipts)));
      const Table t = inorder_tables(h, want_ipts);
      FKD_CUDA(launch_tables(h->plan.evs, 1, (uint32_t)h->n, t, h->dim, st));
      FKD_CUDA(cudaEventRecord(h->inorder_ev, st));
      h->inorder_valid = true;
      h->ipts_valid = want_ipts;
    }
  }
  FKD_CUDA(cudaStreamWaitEvent(st, h->inorder_ev, 0));
  return FKD_OK;
}

// Radius searches walk by the bounding boxes from this many queries on: a walk
// node by node (k_radius) has 32 nodes of a query in flight, which serves few
// queries faster, on one B200 (us, k_radius against the walk, unordered lists):
// 1,000 queries of 5 results 86 / 91, 3,000 of 130 112 / 126, 100,000 of 5 585 /
// 453, of 130 753 / 578; ordered, where the record saves the sort: 1,000
// 90 / 113, 3,000 151 / 144, 100,000 of 130 1918 / 525.
constexpr uint64_t RADIUS_WALK_MIN = BOX_ORDER_MIN, RADIUS_RECORD_MIN = 2048;

// kNN and radius searches can also do without the in-order tables (a thread per
// query, a walk node by node), and a tree that is asked once should: the tables
// cost 10 us and 12 ns per 1,000 points, and a handle that has none yet some
// 350 us to allocate them (below 2 MB only when they do not fit a block of that size
// that is there: the less, the rarer).  They are built once the calls could have gained that much from them
// (`gain` ns by this one), the calls on this tree for the first and all on the
// handle for the second: the calls before are as fast as without tables, and all of
// them together at most twice as slow as with the better choice.  First call on a
// new handle / on a rebuilt tree / later ones, us, without tables and with them at once:
//   64 neighbours of 1,000 queries, 10^6 points    1,906 / 1,719 / 1,699    530 / 82 / 62
//   1 neighbour of 1,000 queries, 10^6 points        233 / 119 / 105        493 / 57 / 34
//   1 neighbour of 1,000 queries, 2^24 points        263 / 164 / 118        770 / 247 / 35
//   16,384 balls of 5 points, ordered, 10^6          358 / 258 / 253        1,335 / 155 / 132
bool tables_pay(fkd_tree h, uint64_t gain) {
  std::lock_guard<std::mutex> g(h->tree_mu);
  const bool want_ipts = h->search_bucket != 0 || h->search_bucket_grp != 0;
  if (h->inorder_valid && (!want_ipts || h->ipts_valid)) return true;
  const size_t need = inorder_bytes(h->n, want_ipts);
  const uint64_t cost = h->inord.bytes >= need ? 0u : need >= (2u << 20) ? 350000u : 350000ull * need >> 22;
  h->nn_rent += gain;
  h->nn_rent_all += gain;
  return h->nn_rent >= 10000u + h->n * 12u / 1000u && h->nn_rent_all >= cost;
}

// What a call gains, in ns (the table's figures and others of the same measurement: a lone query of k
// neighbours 12 + 4.5 k us, some thousand 50 + 16 k, more of them by the query; balls by the query, more
// where the record also saves the sort).
uint64_t knn_gain(uint32_t k, uint64_t q) {
  return q < 32u ? 12000u + 4500ull * k : 40000u + 16000ull * k + (q > 16384u ? (q - 16384u) * k * 3u / 10u : 0u);
}
uint64_t radius_gain(uint64_t q, int ordered) { return ordered ? 15000u + 6u * q : 20000u + q * 14u / 10u; }

// The tables for a search that can also do without: *on is false when there is
// no room for them.
fkd_status walk_tables(fkd_tree h, cudaStream_t st, bool* on) {
  const fkd_status s = ensure_inorder(h, st);
  *on = s == FKD_OK && h->n != 0;
  if (s == FKD_ERR_NOMEM) {
    (void)cudaGetLastError();
    return FKD_OK;
  }
  return s;
}

// Subtree digests of the current tree (digest search), built once per tree.
fkd_status ensure_sdig(fkd_tree h, cudaStream_t st) {
  if (h->n == 0) return FKD_OK;
  {
    std::lock_guard<std::mutex> g(h->tree_mu);
    if (!h->sdig_valid) {
      FKD_CUDA(h->sdig.ensure(h->n * sizeof(unsigned long long)));
      Table t = table_of(h);
      t.sdig = h->sdig.as<unsigned long long>();
      FKD_CUDA(launch_tables(h->plan.evs, 1, (uint32_t)h->n, t, h->dim, st));
      FKD_CUDA(cudaEventRecord(h->sdig_ev, st));
      h->sdig_valid = true;
    }
  }
  FKD_CUDA(cudaStreamWaitEvent(st, h->sdig_ev, 0));
  return FKD_OK;
}

}  // namespace

namespace fkd {
fkd_status capi_fail(fkd_status s, const std::string& msg) { return fail(s, msg); }
fkd_status capi_status_from_err(uint32_t e, const char* what) { return status_from_err(e, what); }
}  // namespace fkd

extern "C" {

const char* fkd_version(void) { return "fkdtree_b200 0.1 (sm_100a)"; }

uint64_t fkd_kernel_launches(void) { return launches_total(); }

const char* fkd_last_error(void) { return g_last_error.c_str(); }

void fkd_debug_fail_alloc(int32_t after) { __atomic_store_n(&fkd::g_fail_alloc, after < 0 ? -1 : after, __ATOMIC_RELAXED); }

void fkd_debug_fail_launch(int32_t after) { __atomic_store_n(&fkd::g_fail_launch, after < 0 ? -1 : after, __ATOMIC_RELAXED); }

fkd_status fkd_create(int dim, uint32_t flags, void* stream, fkd_tree* out) {
  if (!out) return fail(FKD_ERR_ARG, "null output handle pointer");
  *out = nullptr;
  if (dim < 1 || dim > 4) return fail(FKD_ERR_ARG, "dim must be 1..4");
  fkd_tree h = new (std::nothrow) fkd_tree_s();
  if (!h) return fail(FKD_ERR_NOMEM, "host allocation failed");
  h->dim = dim;
  h->flags = flags;
  h->stream = (cudaStream_t)stream;
  cudaError_t e = cudaGetDevice(&h->device);
  if (e == cudaSuccess) e = h->err.ensure(sizeof(uint32_t) * 4);
  if (e == cudaSuccess) e = h->passflags.ensure(sizeof(uint32_t) * 64);
  if (e == cudaSuccess) e = h->lstats.ensure(4 * sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMemsetAsync(h->lstats.p, 0, 4 * sizeof(unsigned long long), h->stream);
  if (e == cudaSuccess) e = cudaMallocHost((void**)&h->herr, sizeof(uint32_t) * 16);
  for (cudaEvent_t* ev : {&h->built_ev, &h->inorder_ev, &h->sdig_ev})
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaMemsetAsync(h->err.p, 0, sizeof(uint32_t), h->stream);
  if (e == cudaSuccess) e = cudaEventRecord(h->built_ev, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  if (e != cudaSuccess) {
    delete h;
    return fail(e == cudaErrorMemoryAllocation ? FKD_ERR_NOMEM : FKD_ERR_CUDA,
                std::string("fkd_create: ") + cudaGetErrorString(e));
  }
  *out = h;
  g_last_error.clear();
  return FKD_OK;
}

fkd_status fkd_destroy(fkd_tree h) {
  if (!h) return FKD_OK;
  DeviceScope ds(h->device);
  cudaStreamSynchronize(h->stream);
  delete h;
  return FKD_OK;
}

fkd_status fkd_set_stream(fkd_tree h, void* stream) {
  if (!h) return fail(FKD_ERR_ARG, "null handle");
  h->stream = (cudaStream_t)stream;
  return FKD_OK;
}

}  // extern "C"

namespace {

// Points in the reference's FKDPoint<float, dim> layout (FKDPoint.h:102-103:
// dim coordinates then the id, (dim + 1) words per point) to the SoA records
// of the build (coordinate c of point i at soa[c*n + i], ids at soa[dim*n + i]).
__global__ void k_points_to_soa(const uint32_t* __restrict__ pts, uint64_t n, int dim, uint32_t* __restrict__ soa) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t* p = pts + i * (uint64_t)(dim + 1);
  for (int w = 0; w <= dim; ++w) soa[(uint64_t)w * n + i] = __ldg(p + w);
}

// fkd_build (coords + ids SoA) and fkd_build_points (AoS points) share this.
fkd_status build_impl(fkd_tree h, const float* coords, const uint32_t* ids, const void* points, uint64_t n,
                             int mem) {
  if (!h) return fail(FKD_ERR_ARG, "null handle");
  if (mem != FKD_MEM_HOST && mem != FKD_MEM_DEVICE) return fail(FKD_ERR_ARG, "mem must be FKD_MEM_HOST or FKD_MEM_DEVICE");
  if (n >= (1ull << 31)) return fail(FKD_ERR_ARG, "at most 2^31-1 points per tree");
  if (n && !points && (!coords || !ids)) return fail(FKD_ERR_ARG, "null coords or ids");
  DeviceScope ds(h->device);
  h->built = false;
  {
    std::lock_guard<std::mutex> g(h->tree_mu);
    h->sdig_valid = false;
    h->inorder_valid = false;
    h->ipts_valid = false;
    h->nn_rent = 0;
  }
  h->n = n;
  if (n == 0) {
    h->built = true;
    FKD_CUDA(cudaEventRecord(h->built_ev, h->stream));
    return FKD_OK;
  }
  const int dim = h->dim;
  if (h->plan_n != n) {
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device);
    PlanHost ph;
    const uint32_t n32 = (uint32_t)n, base0 = 0u;
    plan_build(&n32, &base0, 1, dim, h->hist_ctas ? h->hist_ctas : 4u * (uint32_t)sms, ph, h->subtree_size);
    // a failed upload leaves no plan: the next build must plan again
    h->plan_n = ~0ull;
    FKD_CUDA(h->plan.upload(ph, h->stream));
    h->plan_n = n;
  }
  const size_t rec_bytes = (size_t)(dim + 1) * n * sizeof(uint32_t);
  FKD_CUDA(h->nodes.ensure(n * sizeof(uint4)));
  FKD_CUDA(h->ids.ensure(n * sizeof(uint32_t)));
  FKD_CUDA(h->work1.ensure(rec_bytes));
  if (!h->plan.levels.empty()) {
    FKD_CUDA(h->work0.ensure(rec_bytes));
    FKD_CUDA(h->sel.ensure(2 * sizeof(SegSel) * (size_t)h->plan.maxseg));
    FKD_CUDA(h->bnd.ensure(2 * sizeof(uint2) * (size_t)h->plan.maxseg));
    if (h->small_fix) FKD_CUDA(h->tiebuf.ensure((size_t)h->plan.maxseg * SMALL_CAP * (dim + 1) * sizeof(uint32_t)));
    const size_t gw = (size_t)h->plan.maxseg * HIST_BINS;
    FKD_CUDA(h->ghist.ensure(gw * sizeof(uint32_t)));
  }
  FKD_CUDA(cudaMemsetAsync(h->err.p, 0, sizeof(uint32_t), h->stream));
  BuildCtx bc;
  if (points) {
    uint32_t* w1 = h->work1.as<uint32_t>();
    const uint32_t* src = (const uint32_t*)points;
    if (mem == FKD_MEM_HOST) {
      FKD_CUDA(h->tmp.ensure(rec_bytes));
      FKD_CUDA(cudaMemcpyAsync(h->tmp.p, points, rec_bytes, cudaMemcpyHostToDevice, h->stream));
      src = h->tmp.as<uint32_t>();
    }
    k_points_to_soa<<<(unsigned)((n + 255) / 256), 256, 0, h->stream>>>(src, n, dim, w1);
    count_launches(1);
    FKD_CUDA(cudaGetLastError());
    bc.input = CSoA{w1, w1 + (size_t)dim * n, n};
  } else if (mem == FKD_MEM_HOST) {
    uint32_t* w1 = h->work1.as<uint32_t>();
    FKD_CUDA(cudaMemcpyAsync(w1, coords, (size_t)dim * n * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    FKD_CUDA(cudaMemcpyAsync(w1 + (size_t)dim * n, ids, n * sizeof(uint32_t), cudaMemcpyHostToDevice, h->stream));
    bc.input = CSoA{w1, w1 + (size_t)dim * n, n};
  } else {
    bc.input = CSoA{(const uint32_t*)coords, ids, n};
  }
  uint32_t* w0 = h->work0.as<uint32_t>();
  uint32_t* w1 = h->work1.as<uint32_t>();
  bc.work[0] = SoA{w0, w0 ? w0 + (size_t)dim * n : nullptr, n};
  bc.work[1] = SoA{w1, w1 + (size_t)dim * n, n};
  bc.evs = h->plan.evs;
  bc.nlevels = (uint32_t)h->plan.levels.size();
  bc.levels = h->plan.levels.data();
  bc.subs = h->plan.subs;
  bc.nsub = h->plan.nsub;
  bc.mids = h->plan.mids;
  bc.nmid = h->plan.nmid;
  bc.sel = h->sel.as<SegSel>();
  bc.ghist = h->ghist.as<uint32_t>();
  bc.tab = table_of(h);
  bc.err = h->err.as<uint32_t>();
  bc.pending = h->passflags.as<uint32_t>();
  bc.bnd = h->plan.levels.empty() ? nullptr : h->bnd.as<uint2>();
  bc.tiebuf = (h->small_fix && !h->plan.levels.empty()) ? h->tiebuf.as<uint32_t>() : nullptr;
  bc.lin = h->lin_pass;
  bc.bnd_stride = h->plan.maxseg;
  // a 4-D tree of a few points has no use for four sorted lists of 1,024 slots (1 point 28 us with the
  // radix select, 36 with the lists; 100 equal ones 40 and 53; 512 random ones 61 and 49)
  bc.subtree = h->subtree == 0 && dim == 4 && n <= 128u ? 1 : h->subtree;
  bc.subn = h->subtree_size;
  bc.small_select = h->small_select;
  bc.stream = h->stream;
  memset(&bc.learn, 0, sizeof bc.learn);
  bc.learn.stats = h->lstats.as<unsigned long long>();  // [3] counts the digit passes of every build
  if (h->mlp && !h->plan.levels.empty()) {
    const size_t ms = h->plan.maxseg;
    FKD_CUDA(h->lfeat.ensure(ms * FKD_MLP_FEATURES * sizeof(float)));
    FKD_CUDA(h->lyhat.ensure(ms * sizeof(float)));
    FKD_CUDA(h->lrange.ensure(ms * sizeof(float2)));
    FKD_CUDA(h->lstats.ensure(4 * sizeof(unsigned long long)));
    bc.learn.params = mlp_params(h->mlp);
    bc.learn.delta = h->mlp_delta;
    bc.learn.feat = h->lfeat.as<float>();
    bc.learn.yhat = h->lyhat.as<float>();
    bc.learn.range = h->lrange.as<float2>();
    bc.learn.stats = h->lstats.as<unsigned long long>();
  }
  const bool kt = !h->kev.empty();
  if (kt) {
    FKD_CUDA(cudaEventRecord(h->kev_at(h->kev_builds, 4), h->stream));
    bc.ev_sub = h->kev_at(h->kev_builds, 5);
  }
  FKD_CUDA(launch_build(bc, dim));
  if (kt) {
    FKD_CUDA(cudaEventRecord(h->kev_at(h->kev_builds, 6), h->stream));
    ++h->kev_builds;
  }
  FKD_CUDA(cudaEventRecord(h->built_ev, h->stream));
  h->built = true;
  fkd_status s = finish(h, points ? "fkd_build_points" : "fkd_build", mem);
  if (s != FKD_OK) h->built = false;
  return s;
}

}  // namespace

extern "C" {

fkd_status fkd_build(fkd_tree h, const float* coords, const uint32_t* ids, uint64_t n, int mem) {
  return build_impl(h, coords, ids, nullptr, n, mem);
}

fkd_status fkd_build_points(fkd_tree h, const void* points, uint64_t n, int mem) {
  if (n && !points) return fail(FKD_ERR_ARG, "null points");
  return build_impl(h, nullptr, nullptr, points, n, mem);
}

fkd_status fkd_size(fkd_tree h, uint64_t* n) {
  if (!h || !n) return fail(FKD_ERR_ARG, "null argument");
  *n = h->built ? h->n : 0;
  return FKD_OK;
}

fkd_status fkd_get_tables(fkd_tree h, float* tab, uint32_t* tab_ids, int mem) {
  if (!h) return fail(FKD_ERR_ARG, "null handle");
  if (!h->built) return fail(FKD_ERR_STATE, "tables requested before build");
  if (mem != FKD_MEM_HOST && mem != FKD_MEM_DEVICE) return fail(FKD_ERR_ARG, "mem must be FKD_MEM_HOST or FKD_MEM_DEVICE");
  const uint64_t n = h->n;
  if (n == 0) return FKD_OK;
  DeviceScope ds(h->device);
  std::lock_guard<std::mutex> g(h->tab_mu);
  if (tab) {
    float* dst = tab;
    if (mem == FKD_MEM_HOST) {
      FKD_CUDA(h->work0.ensure((size_t)(h->dim + 1) * n * sizeof(uint32_t)));
      dst = h->work0.as<float>();
    }
    k_tables_out<<<(unsigned)((n + 255) / 256), 256, 0, h->stream>>>((uint32_t)n, h->dim, h->nodes.as<uint4>(), dst);
    count_launches(1);
    FKD_CUDA(cudaGetLastError());
    if (mem == FKD_MEM_HOST)
      FKD_CUDA(cudaMemcpyAsync(tab, dst, (size_t)h->dim * n * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
  }
  if (tab_ids)
    FKD_CUDA(cudaMemcpyAsync(tab_ids, h->ids.p, n * sizeof(uint32_t),
                             mem == FKD_MEM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice, h->stream));
  if (mem == FKD_MEM_HOST || !(h->flags & FKD_FLAG_ASYNC)) FKD_CUDA(cudaStreamSynchronize(h->stream));
  return FKD_OK;
}

fkd_status fkd_search_count(fkd_tree h, const float* mins, const float* maxs, uint64_t q, uint32_t* counts, int mem) {
  fkd_status s = check_search_args(h, mins, maxs, q, mem);
  if (s != FKD_OK) return s;
  if (q && !counts) return fail(FKD_ERR_ARG, "null counts");
  if (q == 0) return FKD_OK;
  DeviceScope ds(h->device);
  Lease L;
  if ((s = lease_slot(h, mem, &L)) != FKD_OK) return s;
  if ((s = clear_ctl(L)) != FKD_OK) return s;
  Boxes b;
  if ((s = stage_boxes(h, L, mins, maxs, q, mem, &b)) != FKD_OK) return s;
  uint32_t* dc = counts;
  if (mem == FKD_MEM_HOST) {
    FKD_CUDA(L.s->counts.ensure(q * sizeof(uint32_t)));
    dc = L.s->counts.as<uint32_t>();
  }
  bool walk = false;
  if ((s = walk_tables(h, L.st, &walk)) != FKD_OK) return s;
  const uint32_t* order = nullptr;
  const uint32_t* start = nullptr;
  if ((s = box_order(h, L, b, &order, &start)) != FKD_OK) return s;
  if ((s = count_pass(h, L, b, dc, order, start)) != FKD_OK) return s;
  if (mem == FKD_MEM_HOST)
    FKD_CUDA(cudaMemcpyAsync(counts, dc, q * sizeof(uint32_t), cudaMemcpyDeviceToHost, L.st));
  return finish_search(h, L, "fkd_search_count", mem);
}

}  // extern "C"

namespace {

// Offsets (and their total, on the host) of the slot's counts; waits for the
// stream, and brings the other control words along.
fkd_status scan_total(const Lease& L, uint64_t q, uint64_t* doff, uint64_t* total) {
  SearchSlot* sl = L.s;
  uint32_t* ctl = sl->err.as<uint32_t>();
  FKD_CUDA(launch_scan_counts(sl->counts.as<uint32_t>(), q, doff, sl->partials.as<unsigned long long>(), L.st,
                              ctl + CTL_TICKET + 1, (uint64_t*)(ctl + CTL_TOTAL)));
  const fkd_status s = fetch_ctl(L);
  memcpy(total, sl->herr + CTL_TOTAL, sizeof(uint64_t));
  return s;
}

// Takes note of the demand a recording pass met (its control words have come back): when it did not
// fit, the next call's pool holds it with room to spare.  Returns the boxes left over.
uint64_t record_demand(fkd_tree h, SearchSlot* sl) {
  uint64_t dem[2];
  memcpy(dem, sl->herr + CTL_ENTS, sizeof dem);
  if (!h->search_pool && dem[0] > sl->ent_cap)
    sl->ent_want = std::max<uint64_t>(sl->ent_want, dem[0] + dem[0] / 4 + (1u << 20));
  return dem[1];
}

// The entry pool of a recording count pass (fkd_walk.cu): `guess` entries per box,
// or what an earlier call that did not fit asked for; *on is false when recording
// is off or there is no room for it (the boxes are then traversed twice).  One
// allocation with what is kept per box, for the sake of a handle's first call: each
// takes some 350 us (100,000 small boxes, first call on a handle 1,773 us with four).
fkd_status record_setup(fkd_tree h, const Lease& L, uint64_t q, int ordered, SearchCtx* rec, bool* on,
                        uint64_t guess = 256) {
  SearchSlot* sl = L.s;
  memset(rec, 0, sizeof *rec);
  *on = q > 0 && h->search_record && (h->search_lanes == 0 || h->search_lanes == 32);
  if (!*on) return FKD_OK;
  if (sl->demand_due && cudaEventQuery(sl->done) == cudaSuccess) record_demand(h, sl);
  (void)cudaGetLastError();  // (not ready: the demand is lost, nothing else)
  sl->demand_due = false;
  uint64_t want = std::max<uint64_t>(sl->ent_want, guess * q + (3u << 19));
  if (h->search_pool) want = h->search_pool;
  if (want > 0xfffffff0ull) want = 0xfffffff0ull;  // entries are numbered in 32 bits
  const uint64_t hist = ordered ? q * 32 * sizeof(uint32_t) : 0, fixed = hist + q * sizeof(uint2) + (q + (q & 1)) * sizeof(uint32_t);
  if (sl->rec.ensure(fixed + want * sizeof(uint2)) != cudaSuccess) {
    (void)cudaGetLastError();
    sl->rec.release();
    sl->ent_want = 0;
    *on = false;
    return FKD_OK;
  }
  uint32_t* ctl = sl->err.as<uint32_t>();
  char* at = sl->rec.as<char>();
  rec->ehist = ordered ? (uint32_t*)at : nullptr;
  rec->erec = (uint2*)(at + hist);
  rec->flags = (uint32_t*)(rec->erec + q);
  rec->ents = (uint2*)(at + fixed);
  rec->ent_ctr = (unsigned long long*)(ctl + CTL_ENTS);
  rec->ent_cap = std::min<uint64_t>((sl->rec.bytes - fixed) / sizeof(uint2), h->search_pool ? h->search_pool : 0xfffffff0ull);
  sl->ent_cap = rec->ent_cap;
  rec->flag_ctr = (unsigned long long*)(ctl + CTL_FLAGS);
  return FKD_OK;
}

// Room for what a call cannot do without: the record, which it can, gives way.
cudaError_t ensure_or_drop(const Lease& L, DevBuf& b, size_t bytes, bool* rec_on) {
  cudaError_t e = b.ensure(bytes);
  if (e != cudaErrorMemoryAllocation || !*rec_on) return e;
  *rec_on = false;
  if ((e = cudaStreamSynchronize(L.st)) != cudaSuccess) return e;
  L.s->rec.release();
  return b.ensure(bytes);
}

// rec: the entry pool the count pass filled (null: traverse every box); with
// it, k_emit writes the recorded boxes and the traversal only visits those
// whose entries did not fit (`left`, when the caller knows there are any).
fkd_status write_pass(fkd_tree h, const Lease& L, const Boxes& b, const uint64_t* doffsets, uint32_t* dout,
                      uint64_t total, int ordered, const uint32_t* order, const SearchCtx* rec = nullptr,
                      bool left = true) {
  fkd_status s0 = ensure_inorder(h, L.st);
  if (s0 != FKD_OK) return s0;
  SearchCtx sc = search_ctx(h, L, b);
  sc.order = order;
  sc.offsets = doffsets;
  sc.out = dout;
  sc.capacity = total;
  sc.heap_out = ordered ? 1 : 0;
  if (rec) {
    SearchCtx x = sc;
    x.ents = rec->ents;
    x.ent_cap = rec->ent_cap;
    x.erec = rec->erec;
    x.ehist = rec->ehist;
    FKD_CUDA(launch_emit(x, ordered));
    if (!left) return FKD_OK;
    sc.order = rec->flags;
    sc.qdev = rec->flag_ctr;
  }
  FKD_CUDA(launch_search(sc, h->dim, SEARCH_WRITE));
  if (ordered) {
    FKD_CUDA(L.s->tmp.ensure(total ? total * sizeof(uint32_t) : 4));
    FKD_CUDA(launch_order_results(sc.g, sc.tab, doffsets, b.q, dout, total, L.s->tmp.as<uint32_t>(), sc.err, L.st,
                                  rec ? sc.order : nullptr, sc.qdev));
  }
  return FKD_OK;
}

}  // namespace

extern "C" {

fkd_status fkd_search_write(fkd_tree h, const float* mins, const float* maxs, uint64_t q, const uint64_t* offsets,
                            uint32_t* ids_out, int ordered, int mem) {
  fkd_status s = check_search_args(h, mins, maxs, q, mem);
  if (s != FKD_OK) return s;
  if (!offsets) return fail(FKD_ERR_ARG, "null offsets");
  if (q == 0) return FKD_OK;
  DeviceScope ds(h->device);
  Lease L;
  if ((s = lease_slot(h, mem, &L)) != FKD_OK) return s;
  if ((s = clear_ctl(L)) != FKD_OK) return s;
  SearchSlot* sl = L.s;
  Boxes b;
  if ((s = stage_boxes(h, L, mins, maxs, q, mem, &b)) != FKD_OK) return s;
  const uint64_t* doff = offsets;
  uint32_t* dout = ids_out;
  uint64_t total = 0;
  if (mem == FKD_MEM_HOST) {
    total = offsets[q];
    if (total && !ids_out) return fail(FKD_ERR_ARG, "null ids_out");
    FKD_CUDA(sl->offsets.ensure((q + 1) * sizeof(uint64_t)));
    FKD_CUDA(cudaMemcpyAsync(sl->offsets.p, offsets, (q + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice, L.st));
    doff = sl->offsets.as<uint64_t>();
    FKD_CUDA(sl->out.ensure(total ? total * sizeof(uint32_t) : 4));
    dout = sl->out.as<uint32_t>();
  } else {
    FKD_CUDA(cudaMemcpyAsync(sl->herr + CTL_TOTAL, offsets + q, sizeof(uint64_t), cudaMemcpyDeviceToHost, L.st));
    FKD_CUDA(cudaStreamSynchronize(L.st));
    memcpy(&total, sl->herr + CTL_TOTAL, sizeof(uint64_t));
    if (total && !ids_out) return fail(FKD_ERR_ARG, "null ids_out");
  }
  const uint32_t* order = nullptr;
  const uint32_t* start = nullptr;
  if ((s = box_order(h, L, b, &order, &start)) != FKD_OK) return s;
  // ordered lists: record and emit, as fkd_search does (one traversal, no sort)
  SearchCtx rec;
  bool rec_on = false;
  if (ordered) {
    if ((s = ensure_inorder(h, L.st)) != FKD_OK) return s;
    FKD_CUDA(sl->tmp.ensure(total ? total * sizeof(uint32_t) : 4));  // (write_pass's: before what can be done without)
    if ((s = record_setup(h, L, q, ordered, &rec, &rec_on)) != FKD_OK) return s;
    rec_on = rec_on && sl->counts.ensure(q * sizeof(uint32_t)) == cudaSuccess;
    if (rec_on) {
      if ((s = count_pass(h, L, b, sl->counts.as<uint32_t>(), order, start, &rec)) != FKD_OK) return s;
    }
  }
  if ((s = write_pass(h, L, b, doff, dout, total, ordered, order, rec_on ? &rec : nullptr)) != FKD_OK) return s;
  if (mem == FKD_MEM_HOST && total)
    FKD_CUDA(cudaMemcpyAsync(ids_out, dout, total * sizeof(uint32_t), cudaMemcpyDeviceToHost, L.st));
  const bool async = mem == FKD_MEM_DEVICE && (h->flags & FKD_FLAG_ASYNC);
  if (rec_on && async) {  // read at the slot's next lease
    FKD_CUDA(cudaMemcpyAsync(sl->herr + CTL_ENTS, sl->err.as<uint32_t>() + CTL_ENTS, 2 * sizeof(uint64_t),
                             cudaMemcpyDeviceToHost, L.st));
    sl->demand_due = true;
  }
  s = finish_search(h, L, "fkd_search_write", mem);
  if (rec_on && !async) record_demand(h, sl);
  return s;
}

}  // extern "C"

namespace {

// fkd_search of one host-memory box (the drop-in's search_in_the_box): one
// launch of k_one, one copy back of its count and first ids, one wait -- in
// place of staging, count pass, scan, write pass and their two waits.  Its
// list is the level-order one (ascending heap index), which serves ordered
// and unordered calls alike.  Sets *general (returning FKD_OK, outputs
// untouched) when the general path must answer instead: a NaN bound (whose
// meaning the general path defines), a frontier too wide for the warp, or
// more results than its buffer holds.
constexpr uint32_t ONE_CAP = 1u << 16;   // ids k_one writes
constexpr uint32_t ONE_FIRST = 1024;     // ids copied back with the count
fkd_status search_one(fkd_tree h, const float* mins, const float* maxs, uint64_t* offsets_out, uint32_t* ids_out,
                      uint64_t capacity, uint64_t* total, bool* general) {
  *general = false;
  OneBox bx;
  for (int c = 0; c < 4; ++c) bx.lo[c] = bx.hi[c] = 0.f;
  for (int c = 0; c < h->dim; ++c) {
    if (mins[c] != mins[c] || maxs[c] != maxs[c]) {
      *general = true;
      return FKD_OK;
    }
    bx.lo[c] = mins[c];
    bx.hi[c] = maxs[c];
  }
  DeviceScope ds(h->device);
  Lease L;
  fkd_status s = lease_slot(h, FKD_MEM_HOST, &L);
  if (s != FKD_OK) return s;
  SearchSlot* sl = L.s;
  FKD_CUDA(sl->one.ensure((4 + ONE_CAP) * sizeof(uint32_t)));
  if (!sl->hone) FKD_CUDA(cudaMallocHost((void**)&sl->hone, (4 + ONE_FIRST) * sizeof(uint32_t)));
  const uint32_t cap = (uint32_t)std::min<uint64_t>(capacity, ONE_CAP);
  const uint32_t first = std::min(cap, ONE_FIRST);
  FKD_CUDA(launch_one(table_of(h), (uint32_t)h->n, h->dim, bx, sl->one.as<uint32_t>(), cap, L.st));
  FKD_CUDA(cudaMemcpyAsync(sl->hone, sl->one.p, (4 + first) * sizeof(uint32_t), cudaMemcpyDeviceToHost, L.st));
  FKD_CUDA(cudaStreamSynchronize(L.st));
  const uint64_t tot = sl->hone[0];
  if (sl->hone[1] || (tot > cap && tot <= capacity)) {
    *general = true;
    return FKD_OK;
  }
  offsets_out[0] = 0;
  offsets_out[1] = tot;
  *total = tot;
  if (tot > capacity) {
    char buf[128];
    snprintf(buf, sizeof buf, "fkd_search: %llu results exceed the capacity of %llu ids", (unsigned long long)tot,
             (unsigned long long)capacity);
    return fail(FKD_ERR_CAPACITY, buf);
  }
  if (tot && !ids_out) return fail(FKD_ERR_ARG, "null ids_out");
  memcpy(ids_out, sl->hone + 4, std::min<uint64_t>(tot, first) * sizeof(uint32_t));
  if (tot > first) {
    FKD_CUDA(cudaMemcpyAsync(ids_out + first, sl->one.as<uint32_t>() + 4 + first, (tot - first) * sizeof(uint32_t),
                             cudaMemcpyDeviceToHost, L.st));
    FKD_CUDA(cudaStreamSynchronize(L.st));
  }
  return FKD_OK;
}

}  // namespace

extern "C" {

fkd_status fkd_search(fkd_tree h, const float* mins, const float* maxs, uint64_t q, uint64_t* offsets_out,
                      uint32_t* ids_out, uint64_t capacity, uint64_t* total, int ordered, int mem) {
  fkd_status s = check_search_args(h, mins, maxs, q, mem);
  if (s != FKD_OK) return s;
  if (!offsets_out || !total) return fail(FKD_ERR_ARG, "null offsets_out or total");
  if (q == 1 && mem == FKD_MEM_HOST && h->search_one && h->n <= 0xffffffffull) {
    bool general = false;
    s = search_one(h, mins, maxs, offsets_out, ids_out, capacity, total, &general);
    if (s != FKD_OK || !general) return s;
  }
  DeviceScope ds(h->device);
  Lease L;
  if ((s = lease_slot(h, mem, &L)) != FKD_OK) return s;
  if ((s = clear_ctl(L)) != FKD_OK) return s;
  SearchSlot* sl = L.s;
  const cudaStream_t st = L.st;
  Boxes b;
  if ((s = stage_boxes(h, L, mins, maxs, q, mem, &b)) != FKD_OK) return s;
  FKD_CUDA(sl->counts.ensure(q ? q * sizeof(uint32_t) : 4));
  FKD_CUDA(sl->partials.ensure(scan_partials_words(q) * sizeof(unsigned long long)));
  uint64_t* doff = offsets_out;
  if (mem == FKD_MEM_HOST) {
    FKD_CUDA(sl->offsets.ensure((q + 1) * sizeof(uint64_t)));
    doff = sl->offsets.as<uint64_t>();
  }
  const uint32_t* order = nullptr;
  const uint32_t* start = nullptr;
  if (q && (s = box_order(h, L, b, &order, &start)) != FKD_OK) return s;
  if ((s = ensure_inorder(h, st)) != FKD_OK) return s;
  // per-kernel events only for calls on the handle's stream (a benchmark's
  // single-threaded loop); the ring is not shared between threads
  const bool kt = !h->kev.empty() && st == h->stream;
  if (kt) FKD_CUDA(cudaEventRecord(h->kev_at(h->kev_searches, 0), st));
  // The count pass records every box's result (fkd_walk.cu); boxes whose record
  // does not fit the pool are traversed again by the write pass.
  SearchCtx rec;
  bool rec_on = false;
  if ((s = record_setup(h, L, q, ordered, &rec, &rec_on)) != FKD_OK) return s;
  if (q && (s = count_pass(h, L, b, sl->counts.as<uint32_t>(), order, start, rec_on ? &rec : nullptr)) != FKD_OK) return s;
  if (kt) FKD_CUDA(cudaEventRecord(h->kev_at(h->kev_searches, 1), st));
  uint64_t tot = 0;
  if ((s = scan_total(L, q, doff, &tot)) != FKD_OK) return s;
  bool left = false;
  if (rec_on) left = record_demand(h, sl) != 0;
  *total = tot;
  if ((s = report_slot_err(L, "fkd_search (count)")) != FKD_OK) return s;
  if (mem == FKD_MEM_HOST)
    FKD_CUDA(cudaMemcpyAsync(offsets_out, doff, (q + 1) * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
  if (tot > capacity) {
    FKD_CUDA(cudaStreamSynchronize(st));
    char buf[128];
    snprintf(buf, sizeof buf, "fkd_search: %llu results exceed the capacity of %llu ids", (unsigned long long)tot,
             (unsigned long long)capacity);
    return fail(FKD_ERR_CAPACITY, buf);
  }
  if (tot && !ids_out) return fail(FKD_ERR_ARG, "null ids_out");
  if (tot == 0) {
    if (kt) {
      FKD_CUDA(cudaEventRecord(h->kev_at(h->kev_searches, 2), st));
      FKD_CUDA(cudaEventRecord(h->kev_at(h->kev_searches, 3), st));
      ++h->kev_searches;
    }
    FKD_CUDA(cudaStreamSynchronize(st));
    return FKD_OK;
  }
  uint32_t* dout = ids_out;
  if (mem == FKD_MEM_HOST) {
    FKD_CUDA(ensure_or_drop(L, sl->out, tot * sizeof(uint32_t), &rec_on));
    dout = sl->out.as<uint32_t>();
  }
  if (ordered && (!rec_on || left)) FKD_CUDA(ensure_or_drop(L, sl->tmp, tot * sizeof(uint32_t), &rec_on));
  if (kt) FKD_CUDA(cudaEventRecord(h->kev_at(h->kev_searches, 2), st));
  if ((s = write_pass(h, L, b, doff, dout, tot, ordered, order, rec_on ? &rec : nullptr, left)) != FKD_OK) return s;
  if (kt) {
    FKD_CUDA(cudaEventRecord(h->kev_at(h->kev_searches, 3), st));
    ++h->kev_searches;
  }
  if (mem == FKD_MEM_HOST)
    FKD_CUDA(cudaMemcpyAsync(ids_out, dout, tot * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  return finish_search(h, L, "fkd_search", mem);
}

fkd_status fkd_search_digest(fkd_tree h, const float* mins, const float* maxs, uint64_t q, uint32_t* counts,
                             uint64_t* digests, int mem) {
  fkd_status s = check_search_args(h, mins, maxs, q, mem);
  if (s != FKD_OK) return s;
  if (q && (!counts || !digests)) return fail(FKD_ERR_ARG, "null counts or digests");
  if (q == 0) return FKD_OK;
  DeviceScope ds(h->device);
  Lease L;
  if ((s = lease_slot(h, mem, &L)) != FKD_OK) return s;
  if ((s = clear_ctl(L)) != FKD_OK) return s;
  Boxes b;
  if ((s = stage_boxes(h, L, mins, maxs, q, mem, &b)) != FKD_OK) return s;
  uint32_t* dc = counts;
  uint64_t* dd = digests;
  if (mem == FKD_MEM_HOST) {
    FKD_CUDA(L.s->counts.ensure(q * sizeof(uint32_t)));
    FKD_CUDA(L.s->digests.ensure(q * sizeof(uint64_t)));
    dc = L.s->counts.as<uint32_t>();
    dd = L.s->digests.as<uint64_t>();
  }
  if ((s = ensure_sdig(h, L.st)) != FKD_OK) return s;
  bool walk = false;
  if ((s = walk_tables(h, L.st, &walk)) != FKD_OK) return s;
  const uint32_t* order = nullptr;
  const uint32_t* start = nullptr;
  if ((s = box_order(h, L, b, &order, &start)) != FKD_OK) return s;
  SearchCtx sc = search_ctx(h, L, b);
  sc.start = start;
  sc.tab.sdig = h->sdig.as<unsigned long long>();
  sc.order = order;
  sc.counts = dc;
  sc.digests = (unsigned long long*)dd;
  if ((s = search_shared(h, L, sc, SEARCH_DIGEST)) != FKD_OK) return s;
  if (mem == FKD_MEM_HOST) {
    FKD_CUDA(cudaMemcpyAsync(counts, dc, q * sizeof(uint32_t), cudaMemcpyDeviceToHost, L.st));
    FKD_CUDA(cudaMemcpyAsync(digests, dd, q * sizeof(uint64_t), cudaMemcpyDeviceToHost, L.st));
  }
  return finish_search(h, L, "fkd_search_digest", mem);
}

}  // extern "C"

namespace {

fkd_status check_nn_args(fkd_tree h, const float* centers, uint64_t q, int mem) {
  if (!h) return fail(FKD_ERR_ARG, "null handle");
  if (!h->built) return fail(FKD_ERR_STATE, "search before build");
  if (mem != FKD_MEM_HOST && mem != FKD_MEM_DEVICE) return fail(FKD_ERR_ARG, "mem must be FKD_MEM_HOST or FKD_MEM_DEVICE");
  if (q > 0xffffffffull) return fail(FKD_ERR_ARG, "at most 2^32-1 queries per call");
  if (q && !centers) return fail(FKD_ERR_ARG, "null centers");
  return FKD_OK;
}

// Stages host centres (dim*q SoA) and radii (q, optional) or aliases device ones.
fkd_status stage_centres(fkd_tree h, const Lease& L, const float* centers, const float* radii, uint64_t q, int mem,
                         const float** dctr, const float** drad) {
  if (mem == FKD_MEM_DEVICE) {
    *dctr = centers;
    if (drad) *drad = radii;
    return FKD_OK;
  }
  SearchSlot* s = L.s;
  const size_t cb = (size_t)h->dim * q * sizeof(float);
  FKD_CUDA(s->qlo.ensure(cb ? cb : 4));
  if (cb) FKD_CUDA(cudaMemcpyAsync(s->qlo.p, centers, cb, cudaMemcpyHostToDevice, L.st));
  *dctr = s->qlo.as<float>();
  if (drad) {
    FKD_CUDA(s->qhi.ensure(q ? q * sizeof(float) : 4));
    if (q) FKD_CUDA(cudaMemcpyAsync(s->qhi.p, radii, q * sizeof(float), cudaMemcpyHostToDevice, L.st));
    *drad = s->qhi.as<float>();
  }
  return FKD_OK;
}

// Spatial order of the query centres (the box order of zero-size boxes).
fkd_status centre_order(fkd_tree h, const Lease& L, const float* dctr, uint64_t q, const uint32_t** order) {
  Boxes b;
  b.lo = dctr;
  b.hi = dctr;
  b.stride = q;
  b.q = q;
  return box_order(h, L, b, order);
}

}  // namespace

extern "C" {

fkd_status fkd_search_radius_count(fkd_tree h, const float* centers, const float* radii, uint64_t q,
                                   uint32_t* counts, int mem) {
  fkd_status s = check_nn_args(h, centers, q, mem);
  if (s != FKD_OK) return s;
  if (q && (!radii || !counts)) return fail(FKD_ERR_ARG, "null radii or counts");
  if (q == 0) return FKD_OK;
  DeviceScope ds(h->device);
  Lease L;
  if ((s = lease_slot(h, mem, &L)) != FKD_OK) return s;
  if ((s = clear_ctl(L)) != FKD_OK) return s;
  const float *dctr = nullptr, *drad = nullptr;
  if ((s = stage_centres(h, L, centers, radii, q, mem, &dctr, &drad)) != FKD_OK) return s;
  uint32_t* dc = counts;
  if (mem == FKD_MEM_HOST) {
    FKD_CUDA(L.s->counts.ensure(q * sizeof(uint32_t)));
    dc = L.s->counts.as<uint32_t>();
  }
  const uint32_t* order = nullptr;
  if ((s = centre_order(h, L, dctr, q, &order)) != FKD_OK) return s;
  bool walk = false;
  if (q >= RADIUS_WALK_MIN && tables_pay(h, radius_gain(q, 0)) && (s = walk_tables(h, L.st, &walk)) != FKD_OK) return s;
  if (walk) {
    SearchCtx sc = search_ctx(h, L, Boxes{dctr, drad, q, q});
    sc.order = order;
    sc.counts = dc;
    FKD_CUDA(launch_walk_balls(sc, h->dim));
  } else {
    FKD_CUDA(launch_radius(make_geom((uint32_t)h->n), table_of(h), dctr, drad, q, order, dc, nullptr, nullptr, 0,
                           L.s->err.as<uint32_t>(), h->dim, L.st));
  }
  if (mem == FKD_MEM_HOST)
    FKD_CUDA(cudaMemcpyAsync(counts, dc, q * sizeof(uint32_t), cudaMemcpyDeviceToHost, L.st));
  return finish_search(h, L, "fkd_search_radius_count", mem);
}

fkd_status fkd_search_radius(fkd_tree h, const float* centers, const float* radii, uint64_t q, uint64_t* offsets_out,
                             uint32_t* ids_out, uint64_t capacity, uint64_t* total, int ordered, int mem) {
  fkd_status s = check_nn_args(h, centers, q, mem);
  if (s != FKD_OK) return s;
  if (!offsets_out || !total) return fail(FKD_ERR_ARG, "null offsets_out or total");
  if (q && !radii) return fail(FKD_ERR_ARG, "null radii");
  DeviceScope ds(h->device);
  Lease L;
  if ((s = lease_slot(h, mem, &L)) != FKD_OK) return s;
  if ((s = clear_ctl(L)) != FKD_OK) return s;
  SearchSlot* sl = L.s;
  const cudaStream_t st = L.st;
  const float *dctr = nullptr, *drad = nullptr;
  if ((s = stage_centres(h, L, centers, radii, q, mem, &dctr, &drad)) != FKD_OK) return s;
  FKD_CUDA(sl->counts.ensure(q ? q * sizeof(uint32_t) : 4));
  FKD_CUDA(sl->partials.ensure(scan_partials_words(q) * sizeof(unsigned long long)));
  uint64_t* doff = offsets_out;
  if (mem == FKD_MEM_HOST) {
    FKD_CUDA(sl->offsets.ensure((q + 1) * sizeof(uint64_t)));
    doff = sl->offsets.as<uint64_t>();
  }
  const uint32_t* order = nullptr;
  if (q && (s = centre_order(h, L, dctr, q, &order)) != FKD_OK) return s;
  const Geom g = make_geom((uint32_t)h->n);
  const Table tab = table_of(h);
  uint32_t* err = sl->err.as<uint32_t>();
  // by the subtrees' bounding boxes; an ordered search records its lists as the box search does
  bool walk = false, rec_on = false;
  SearchCtx rec;
  if (q >= (ordered ? RADIUS_RECORD_MIN : RADIUS_WALK_MIN) && tables_pay(h, radius_gain(q, ordered)) &&
      (s = walk_tables(h, st, &walk)) != FKD_OK)
    return s;
  if (walk) {
    if (ordered && (s = record_setup(h, L, q, 1, &rec, &rec_on, 128)) != FKD_OK) return s;
    SearchCtx sc = search_ctx(h, L, Boxes{dctr, drad, q, q});
    sc.order = order;
    sc.counts = sl->counts.as<uint32_t>();
    if (rec_on) {
      sc.ents = rec.ents;
      sc.ent_ctr = rec.ent_ctr;
      sc.ent_cap = rec.ent_cap;
      sc.erec = rec.erec;
      sc.ehist = rec.ehist;
      sc.flags = rec.flags;
      sc.flag_ctr = rec.flag_ctr;
    }
    FKD_CUDA(launch_walk_balls(sc, h->dim));
  } else {
    FKD_CUDA(launch_radius(g, tab, dctr, drad, q, order, sl->counts.as<uint32_t>(), nullptr, nullptr, 0, err, h->dim,
                           st));
  }
  uint64_t tot = 0;
  if ((s = scan_total(L, q, doff, &tot)) != FKD_OK) return s;
  const bool left = rec_on && record_demand(h, sl) != 0;
  *total = tot;
  if ((s = report_slot_err(L, "fkd_search_radius (count)")) != FKD_OK) return s;
  if (mem == FKD_MEM_HOST)
    FKD_CUDA(cudaMemcpyAsync(offsets_out, doff, (q + 1) * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
  if (tot > capacity) {
    FKD_CUDA(cudaStreamSynchronize(st));
    char buf[128];
    snprintf(buf, sizeof buf, "fkd_search_radius: %llu results exceed the capacity of %llu ids",
             (unsigned long long)tot, (unsigned long long)capacity);
    return fail(FKD_ERR_CAPACITY, buf);
  }
  if (tot && !ids_out) return fail(FKD_ERR_ARG, "null ids_out");
  if (tot == 0) {
    FKD_CUDA(cudaStreamSynchronize(st));
    return FKD_OK;
  }
  uint32_t* dout = ids_out;
  if (mem == FKD_MEM_HOST) {
    FKD_CUDA(ensure_or_drop(L, sl->out, tot * sizeof(uint32_t), &rec_on));
    dout = sl->out.as<uint32_t>();
  }
  if (ordered && (!rec_on || left)) FKD_CUDA(ensure_or_drop(L, sl->tmp, tot * sizeof(uint32_t), &rec_on));
  if (rec_on) {
    SearchCtx x = search_ctx(h, L, Boxes{dctr, drad, q, q});
    x.order = order;
    x.offsets = doff;
    x.out = dout;
    x.capacity = tot;
    x.ents = rec.ents;
    x.ent_cap = rec.ent_cap;
    x.erec = rec.erec;
    x.ehist = rec.ehist;
    FKD_CUDA(launch_emit(x, 1));
  }
  // without a record (or for the queries it has no room for), ordered: the write pass emits heap
  // indices that k_order sorts and maps to ids
  if (!rec_on || left) {
    const uint32_t* list = rec_on ? rec.flags : order;
    const unsigned long long* nlist = rec_on ? rec.flag_ctr : nullptr;
    FKD_CUDA(launch_radius(g, tab, dctr, drad, q, list, nullptr, doff, dout, ordered ? 1 : 0, err, h->dim, st, nlist));
    if (ordered)
      FKD_CUDA(launch_order_results(g, tab, doff, q, dout, tot, sl->tmp.as<uint32_t>(), err, st,
                                    rec_on ? list : nullptr, nlist));
  }
  if (mem == FKD_MEM_HOST)
    FKD_CUDA(cudaMemcpyAsync(ids_out, dout, tot * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  return finish_search(h, L, "fkd_search_radius", mem);
}

uint32_t fkd_knn_max_k(void) { return KNN_MAX; }

fkd_status fkd_search_knn(fkd_tree h, const float* centers, uint64_t q, uint32_t k, uint32_t* ids_out,
                          float* dist2_out, int mem) {
  fkd_status s = check_nn_args(h, centers, q, mem);
  if (s != FKD_OK) return s;
  if (k < 1 || k > KNN_MAX) return fail(FKD_ERR_ARG, "k must be 1..fkd_knn_max_k()");
  if (q && !ids_out) return fail(FKD_ERR_ARG, "null ids_out");
  if (q == 0) return FKD_OK;
  DeviceScope ds(h->device);
  Lease L;
  if ((s = lease_slot(h, mem, &L)) != FKD_OK) return s;
  if ((s = clear_ctl(L)) != FKD_OK) return s;
  SearchSlot* sl = L.s;
  const float* dctr = nullptr;
  if ((s = stage_centres(h, L, centers, nullptr, q, mem, &dctr, nullptr)) != FKD_OK) return s;
  const uint64_t cells = q * (uint64_t)k;
  uint32_t* di = ids_out;
  float* dd = dist2_out;
  if (mem == FKD_MEM_HOST) {
    FKD_CUDA(sl->out.ensure(cells * sizeof(uint32_t)));
    di = sl->out.as<uint32_t>();
    if (dist2_out) {
      FKD_CUDA(sl->tmp.ensure(cells * sizeof(float)));
      dd = sl->tmp.as<float>();
    }
  }
  const uint32_t* order = nullptr;
  if ((s = centre_order(h, L, dctr, q, &order)) != FKD_OK) return s;
  bool walk = false;  // else a thread per query, which reads no tables
  if (knn_by_warps(h->dim, k, q, h->n) && tables_pay(h, knn_gain(k, q)) && (s = walk_tables(h, L.st, &walk)) != FKD_OK)
    return s;
  const Table tab = walk ? search_ctx(h, L, Boxes{dctr, dctr, q, q}).tab : table_of(h);
  FKD_CUDA(launch_knn(make_geom((uint32_t)h->n), tab, dctr, q, order, k, di, dd, sl->err.as<uint32_t>(), h->dim,
                      L.st));
  if (mem == FKD_MEM_HOST) {
    FKD_CUDA(cudaMemcpyAsync(ids_out, di, cells * sizeof(uint32_t), cudaMemcpyDeviceToHost, L.st));
    if (dist2_out) FKD_CUDA(cudaMemcpyAsync(dist2_out, dd, cells * sizeof(float), cudaMemcpyDeviceToHost, L.st));
  }
  return finish_search(h, L, "fkd_search_knn", mem);
}

fkd_status fkd_set_param(fkd_tree h, const char* name, int64_t value) {
  if (!h || !name) return fail(FKD_ERR_ARG, "null argument");
  if (strcmp(name, "hist_ctas") == 0) {
    if (value < 0 || value > (1 << 20)) return fail(FKD_ERR_ARG, "hist_ctas out of range");
    h->hist_ctas = (uint32_t)value;
    h->plan_n = ~0ull;  // re-plan at the next build
    return FKD_OK;
  }
  if (strcmp(name, "search_lanes") == 0) {
    if (value != 0 && value != 1 && value != 2 && value != 4 && value != 8 && value != 16 && value != 32)
      return fail(FKD_ERR_ARG, "search_lanes must be 0, 1, 2, 4, 8, 16 or 32");
    h->search_lanes = (uint32_t)value;
    return FKD_OK;
  }
  if (strcmp(name, "box_order") == 0) {
    if (value != 0 && value != 1) return fail(FKD_ERR_ARG, "box_order must be 0 or 1");
    h->box_order = value != 0;
    return FKD_OK;
  }
  if (strcmp(name, "small_select") == 0) {
    if (value != 0 && value != 1) return fail(FKD_ERR_ARG, "small_select must be 0 or 1");
    h->small_select = value != 0;
    return FKD_OK;
  }
  if (strcmp(name, "subtree") == 0) {
    if (value < 0 || value > 2) return fail(FKD_ERR_ARG, "subtree must be 0, 1 or 2");
    h->subtree = (int)value;
    return FKD_OK;
  }
  if (strcmp(name, "subtree_size") == 0) {
    if (value != 0 && value != 512 && value != 1024) return fail(FKD_ERR_ARG, "subtree_size must be 0, 512 or 1024");
    h->subtree_size = (int)value;
    h->plan_n = ~0ull;  // re-plan at the next build
    return FKD_OK;
  }
  if (strcmp(name, "small_fix") == 0) {
    if (value != 0 && value != 1) return fail(FKD_ERR_ARG, "small_fix must be 0 or 1");
    h->small_fix = value != 0;
    return FKD_OK;
  }
  if (strcmp(name, "lin_pass") == 0) {
    if (value != 0 && value != 1) return fail(FKD_ERR_ARG, "lin_pass must be 0 or 1");
    h->lin_pass = value != 0;
    return FKD_OK;
  }
  if (strcmp(name, "search_bucket") == 0) {
    if (value < 0 || value > (int64_t)BUCKET_MAX) return fail(FKD_ERR_ARG, "search_bucket must be 0..6");
    h->search_bucket = (uint32_t)value;
    return FKD_OK;
  }
  if (strcmp(name, "bucket_runs") == 0) {
    if (value != 0 && value != 1) return fail(FKD_ERR_ARG, "bucket_runs must be 0 or 1");
    return FKD_OK;  // the recorded lists always hold runs
  }
  if (strcmp(name, "search_bucket_lanes") == 0) {
    if (value < 0 || value > 3) return fail(FKD_ERR_ARG, "search_bucket_lanes must be 0..3");
    h->search_bucket_grp = (uint32_t)value;
    return FKD_OK;
  }
  if (strcmp(name, "search_record") == 0) {
    if (value != 0 && value != 1) return fail(FKD_ERR_ARG, "search_record must be 0 or 1");
    h->search_record = value != 0;
    return FKD_OK;
  }
  if (strcmp(name, "search_packets") == 0) {
    if (value != 0 && value != 1) return fail(FKD_ERR_ARG, "search_packets must be 0 or 1");
    h->search_packets = value != 0;
    return FKD_OK;
  }
  if (strcmp(name, "search_one") == 0) {
    if (value != 0 && value != 1) return fail(FKD_ERR_ARG, "search_one must be 0 or 1");
    h->search_one = value != 0;
    return FKD_OK;
  }
  if (strcmp(name, "search_pool") == 0) {
    if (value < 0 || value > 0xffffffffll) return fail(FKD_ERR_ARG, "search_pool out of range");
    h->search_pool = (uint64_t)value;
    return FKD_OK;
  }
  if (strcmp(name, "kernel_events") == 0) {
    if (value != 0 && value != 1) return fail(FKD_ERR_ARG, "kernel_events must be 0 or 1");
    FKD_CUDA(cudaStreamSynchronize(h->stream));
    for (cudaEvent_t e : h->kev) cudaEventDestroy(e);
    h->kev.clear();
    h->kev_builds = h->kev_searches = 0;
    if (value) {
      FKD_CUDA(cudaSetDevice(h->device));
      h->kev.resize((size_t)fkd_tree_s::KEV_RING * 7, nullptr);
      for (cudaEvent_t& e : h->kev) {
        cudaError_t ce = cudaEventCreate(&e);
        if (ce != cudaSuccess) {
          e = nullptr;
          for (cudaEvent_t x : h->kev)
            if (x) cudaEventDestroy(x);
          h->kev.clear();
          return fail(FKD_ERR_CUDA, std::string("kernel_events: ") + cudaGetErrorString(ce));
        }
      }
    }
    return FKD_OK;
  }
  return fail(FKD_ERR_ARG, std::string("unknown parameter ") + name);
}

fkd_status fkd_kernel_times(fkd_tree h, uint32_t back, float* ms) {
  if (!h || !ms) return fail(FKD_ERR_ARG, "null argument");
  if (h->kev.empty()) return fail(FKD_ERR_STATE, "kernel_events is off");
  float v[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  if (back < fkd_tree_s::KEV_RING && back < h->kev_searches) {
    const uint64_t c = h->kev_searches - 1 - back;
    FKD_CUDA(cudaEventSynchronize(h->kev_at(c, 3)));
    FKD_CUDA(cudaEventElapsedTime(&v[0], h->kev_at(c, 0), h->kev_at(c, 1)));
    FKD_CUDA(cudaEventElapsedTime(&v[1], h->kev_at(c, 2), h->kev_at(c, 3)));
  }
  if (back < fkd_tree_s::KEV_RING && back < h->kev_builds) {
    const uint64_t c = h->kev_builds - 1 - back;
    FKD_CUDA(cudaEventSynchronize(h->kev_at(c, 6)));
    FKD_CUDA(cudaEventElapsedTime(&v[2], h->kev_at(c, 4), h->kev_at(c, 6)));
    FKD_CUDA(cudaEventElapsedTime(&v[3], h->kev_at(c, 4), h->kev_at(c, 5)));
    FKD_CUDA(cudaEventElapsedTime(&v[4], h->kev_at(c, 5), h->kev_at(c, 6)));
  }
  memcpy(ms, v, sizeof v);
  return FKD_OK;
}

fkd_status fkd_set_mlp(fkd_tree h, fkd_mlp m, float delta) {
  if (!h) return fail(FKD_ERR_ARG, "null handle");
  if (m && !(delta > 0.f)) return fail(FKD_ERR_ARG, "delta must be positive");
  h->mlp = m;
  h->mlp_delta = delta;
  if (m) {
    FKD_CUDA(h->lstats.ensure(4 * sizeof(unsigned long long)));
    FKD_CUDA(cudaMemsetAsync(h->lstats.p, 0, 4 * sizeof(unsigned long long), h->stream));
  }
  return FKD_OK;
}

fkd_status fkd_learn_stats(fkd_tree h, uint64_t* stats, int reset) {
  if (!h || !stats) return fail(FKD_ERR_ARG, "null argument");
  stats[0] = stats[1] = stats[2] = stats[3] = 0;
  if (!h->lstats.p) return FKD_OK;
  FKD_CUDA(cudaMemcpyAsync(stats, h->lstats.p, 4 * sizeof(uint64_t), cudaMemcpyDeviceToHost, h->stream));
  if (reset) FKD_CUDA(cudaMemsetAsync(h->lstats.p, 0, 4 * sizeof(unsigned long long), h->stream));
  FKD_CUDA(cudaStreamSynchronize(h->stream));
  return FKD_OK;
}

fkd_status fkd_sync(fkd_tree h) {
  if (!h) return fail(FKD_ERR_ARG, "null handle");
  DeviceScope ds(h->device);
  fkd_status s = check_err_word(h, "fkd_sync");
  if (s != FKD_OK) return s;
  // asynchronous searches latch into the error word of the slot they leased
  std::vector<SearchSlot*> all;
  {
    std::lock_guard<std::mutex> g(h->slot_mu);
    for (auto& p : h->slots) all.push_back(p.get());
  }
  for (SearchSlot* sl : all) {
    FKD_CUDA(cudaStreamWaitEvent(h->stream, sl->done, 0));
    FKD_CUDA(cudaMemcpyAsync(h->herr + 1, sl->err.p, sizeof(uint32_t), cudaMemcpyDeviceToHost, h->stream));
    FKD_CUDA(cudaMemsetAsync(sl->err.p, 0, sizeof(uint32_t), h->stream));
    FKD_CUDA(cudaStreamSynchronize(h->stream));
    if ((s = status_from_err(h->herr[1], "fkd_sync")) != FKD_OK) return s;
  }
  return FKD_OK;
}

}  // extern "C"
