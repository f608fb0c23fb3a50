// fkd_internal.h -- declarations shared by the library's translation units.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fkd_common.cuh"

namespace fkd {

// Process-wide count of kernel launches issued by this library (telemetry for
// benchmarks: how many of the library's own kernels ran in a timed region).
void count_launches(uint64_t k);
uint64_t launches_total();
// cudaMalloc with the allocation-failure injection of fkd_debug_fail_alloc
cudaError_t device_alloc(void** p, size_t bytes);
// what fkd_debug_fail_launch has in store for the next chained launch (cudaSuccess: nothing)
cudaError_t launch_injected();

// Chained launches.  A kernel launched by chain_launch may start while the
// kernel before it in the stream is still finishing: it calls chain_wait()
// first, in every CTA and before any return, which waits until that kernel is
// complete and its writes are visible, and lets the next launch start the same
// way.  What is saved is the launch latency between short kernels of one chain
// (the build of 100,000 points is some fifty of them).
//
// A refused launch is in the status chain_launch returns and nowhere else: the
// runtime's last error is cleared, so that no later call reports it.  Whoever
// launches a kernel that later ones build on has to stop there (FKD_CHAIN):
// they would work on what an earlier call left in their inputs.
#ifdef __CUDACC__
#define FKD_CHAIN(...)                                  \
  do {                                                  \
    const cudaError_t fkd_e_ = chain_launch(__VA_ARGS__); \
    if (fkd_e_ != cudaSuccess) return fkd_e_;           \
  } while (0)

__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... P, class... A>
[[nodiscard]] inline cudaError_t chain_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                A&&... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  count_launches(1);
  cudaError_t e = launch_injected();
  if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  if (e != cudaSuccess) (void)cudaGetLastError();
  return e;
}
#endif

// Lets a kernel's launches have up to `most` bytes of dynamic shared memory.
// The limit is the function's, shared by all threads of the process: `most` is
// the kernel's own maximum, never a call's size, which another thread's smaller
// call could put in its place before this one launches.
template <class K>
inline cudaError_t allow_smem(K kernel, size_t most) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}

// Per-segment state of the global-level select (one per node of the level
// being split).  The digit passes (k_hist) narrow an interval [klo, khi] of
// 64-bit order keys (mono(coordinate) << 32 | id) that holds the pivot: the
// candidates are the segment's points whose key lies in it, krem the pivot's
// rank among them and cnt their number.  While the interval spans several
// coordinate values its id part is the full range and a pass bins the value
// (linearly in the float value for the first pass of a segment whose value
// range is known, `lin`; else the key bits); once the value is fixed a pass
// bins the id.  The select is done when one candidate is left, when the
// interval is one key (repeated keys), or when at most SMALL_CAP candidates
// are left (`small`): the partition then parks them and k_level_end orders
// them by key.  k_select_small and the learned bracket also keep the prefix
// form (prefix / bits) of the levels they serve.
struct SegSel {
  unsigned long long prefix;  // k_select_small: the known top `bits` bits of the pivot key
  uint32_t bits;              // 0..64
  uint32_t krem;              // rank of the pivot among the candidates
  uint32_t cnt;               // number of candidates
  uint32_t done;              // the pivot is determined (or `small`)
  uint32_t tiles_done;        // CTAs of the current pass that finished
  uint32_t curL, curR, curE;  // partition cursors
  uint32_t verify;            // 1: [klo, khi] is a predicted block, the next pass verifies it
  uint32_t below;             // verify pass: points whose key lies below the block
  uint32_t kfull;             // the pivot rank within the segment (fallback restart)
  uint32_t bits0;             // the common prefix every key of the segment shares
  unsigned long long prefix0;
  uint32_t small;             // done with cnt <= SMALL_CAP candidates: the partition parks them
  uint32_t lin;               // the next pass bins the value linearly: bin = floor((v - vmin) * scale)
  unsigned long long klo, khi;    // the candidate key interval
  unsigned long long klo0, khi0;  // the segment's own interval (fallback restart)
  float vmin, scale;              // linear binning of the next pass
  float vmin0, scale0;            // ... of the segment's own range (restart)
  uint32_t lin0;
  uint32_t cmin, cmax;            // the pass's smallest / largest candidate value key (id once the
                                  // value is fixed): the next interval is clipped to them
};
// Candidates a select may leave for the partition to order itself (one warp
// sorts them); more are narrowed by further digit passes.
constexpr uint32_t SMALL_CAP = 32;

constexpr int FKD_MLP_FEATURES = 40;  // node summary width (== FKD_MLP_IN of the C ABI)

// Learned-split state of a build (all null / zero for the plain build).
struct LearnCtx {
  const float* params;  // MLP parameters (null: plain radix select)
  float delta;          // bracket half-width, in units of the sample range
  float* feat;          // >= maxseg * 40 features
  float* yhat;          // >= maxseg predictions
  float2* range;        // >= maxseg sample ranges (min, max) along the split dimension
  unsigned long long* stats;  // [0] brackets tried, [1] verified, [2] fell back
  // recording mode (training data): targets of every global segment
  float* rec_x;         // features of recorded segments (rows of 40)
  float* rec_t;         // their targets
  unsigned long long* rec_n;  // running count
  uint64_t rec_cap;
};

// One event (one independent tree) of a build: its geometry, the position of
// its first point in the concatenated working arrays / node tables, the number
// of levels the global kernels split (d0), and where its boxes are.
struct EvDesc {
  Geom g;
  uint32_t base;     // first point / node of the event
  uint32_t d0;       // global levels of this event
  uint32_t dm;       // ... of which the launches per level split the first dm, the last d0 - dm are left
                     // to the kernel that takes a whole segment (k_mid), when the build uses it
  uint32_t nq;       // boxes of the event
  uint64_t qbase;    // index of the event's first box in the launch's box space
  uint64_t qcbase;   // offset of the event's box coordinates (SoA slice: [c*nq + j])
  uint64_t qout;     // index of the event's first box in the caller's output arrays
};

// Device-side plan of a (batched) build: per global level the list of
// (event, segment) pairs and the CTA -> (segment, tile) maps of the digit and
// partition kernels; the list of (event, subtree) roots of the subtree kernel.
struct LevelPlan {
  const uint2* segs;    // (event, index-in-level)
  uint32_t nseg;
  const uint2* htiles;  // digit-pass CTA -> (segment, tile)
  uint32_t nhtile;
  uint32_t hts;         // digit-pass tile length
  const uint2* ptiles;  // partition CTA -> (segment, tile)
  uint32_t nptile;
  const uint32_t* child;  // per segment: its left child's index in the next level (~0u: not a global segment)
  uint32_t maxlen;        // longest segment of the level
  // the part (a prefix of each list) that a build with k_mid splits by launches per level
  uint32_t nseg_m, nhtile_m, nptile_m;
};

struct BuildCtx {
  const EvDesc* evs;
  uint32_t nlevels;
  const LevelPlan* levels;  // host array of nlevels
  const uint2* subs;        // (event, subtree index at the event's d0)
  uint32_t nsub;
  const uint2* mids = nullptr;  // (event, segment index at the event's dm)
  uint32_t nmid = 0;
  CSoA input;     // the points to build from (device, SoA with stride = total points)
  SoA work[2];    // ping-pong working records
  SegSel* sel;    // 2 x bnd_stride: the select states of a level and the next
  uint32_t* ghist;
  uint32_t* pending;  // one word per digit pass (+1): does that pass have work
  uint32_t* tiebuf = nullptr;  // >= max segments * SMALL_CAP * (dim + 1) words: the candidates a select
                               // leaves to the partition (null: every select narrows to one key)
  uint2* bnd = nullptr;    // 2 x bnd_stride: per-segment (min, max) of the split coordinate's
                           // order bits, written by the previous level's partition (null: unused)
  uint32_t bnd_stride = 0; // >= max segments of a level
  Table tab;
  uint32_t* err;
  cudaStream_t stream;
  LearnCtx learn;
  cudaEvent_t ev_sub = nullptr;  // optional: recorded right before the subtree kernel
  int subtree = 0;               // shared-memory subtree kernel: 0 auto, 1 radix select, 2 presorted lists
  bool small_select = true;      // levels of small segments: one CTA per segment selects or splits (k_mid)
  bool lin = true;               // a segment's first digit pass bins its value range linearly
  int subn = 0;                  // presorted subtree size the plan was made for (0: 1,024)
};

// Number of levels split by the global kernels (the first level whose
// intervals all fit the shared-memory subtree kernel).
// subn: the presorted-list kernel's subtree size (512 or 1,024; 0 = 1,024).
uint32_t build_global_levels(uint32_t n, int dim, int subn = 0);
int sub_capacity(int dim);
int sorted_sub_capacity(int subn = 0);  // largest subtree of the presorted-list kernel
uint32_t mid_capacity();  // largest segment k_mid takes
constexpr uint32_t HIST_BINS = 2048;  // global digit histogram per segment
#ifndef FKD_PART_PIPT
#define FKD_PART_PIPT 4
#endif
constexpr uint32_t PART_TILE = 256 * FKD_PART_PIPT;  // records per partition CTA
constexpr uint32_t HIST_STEP = 2048;  // digit-pass tile granularity
cudaError_t launch_build(BuildCtx& bc, int dim);
// fkd_mid.cu: the levels from an event's dm to its d0, one CTA per segment
cudaError_t launch_mid(const EvDesc* evs, const uint2* mids, uint32_t nmid, CSoA in, SoA b0, SoA b1, Table tab,
                       uint32_t* err, int dim, cudaStream_t stream);
// fkd_subtree_sort.cu: the subtree kernel by presorted lists
cudaError_t launch_subtree_sorted(const EvDesc* evs, const uint2* subs, uint32_t nsub, CSoA in, CSoA b0, CSoA b1,
                                  Table tab, uint32_t* err, int dim, int subn, cudaStream_t stream);
// The shared-memory subtree kernel alone, for events whose d0 is 0 (reads
// every event from `src`).
cudaError_t launch_subtree_direct(const EvDesc* evs, const uint2* subs, uint32_t nsub, CSoA src, Table tab,
                                  uint32_t* err, int dim, cudaStream_t stream);
// fkd_features.cu: node summaries, bracket initialisation, target recording
cudaError_t launch_features(uint32_t d, const EvDesc* evs, const uint2* segs, uint32_t nseg, CSoA src, int dim,
                            float* feat, float2* range, cudaStream_t stream);
cudaError_t launch_bracket(uint32_t d, const EvDesc* evs, const uint2* segs, uint32_t nseg, const float* yhat,
                           const float2* range, float delta, SegSel* sel, unsigned long long* stats,
                           cudaStream_t stream);
cudaError_t launch_record(uint32_t d, const EvDesc* evs, const uint2* segs, uint32_t nseg, int dim, Table tab,
                          const float* feat, const float2* range, float* rec_x, float* rec_t,
                          unsigned long long* rec_n, uint64_t rec_cap, cudaStream_t stream);

// ------------------------------------------------------------------ search

struct Boxes {
  const float* lo;  // lo[c*stride + j]
  const float* hi;
  uint64_t stride;
  uint64_t q;
};

enum SearchMode { SEARCH_COUNT = 0, SEARCH_WRITE = 1, SEARCH_DIGEST = 2 };

// The kernels that take boxes from a work counter, for SearchCtx::qready.
enum { QC_WALK = 0, QC_PACKET = 1, QC_LEFT = 2, QC_EMIT = 3, QC_WRITE = 4, QC_LANES = 5, QC_COUNT = 6 };

struct SearchCtx {
  Geom g;
  Table tab;
  Boxes boxes;
  const EvDesc* evs;       // batched search: per-event geometry / bases (null: one event, g + tab)
  uint32_t nev;
  const uint32_t* order;   // optional processing order of the boxes (null: 0..q-1)
  const uint32_t* start;   // optional, with order: per box, a node whose subtree holds all of its results
  uint32_t* counts;        // SEARCH_COUNT / SEARCH_DIGEST
  const uint64_t* offsets; // SEARCH_WRITE
  uint32_t* out;           // SEARCH_WRITE (heap indices when `heap_out`)
  uint64_t capacity;       // ids the output can hold
  unsigned long long* digests;  // SEARCH_DIGEST
  uint32_t* qcounter;      // work counter: zeroed by the launcher, or
  int qready;              // 1: qcounter[QC_*] are zero, one for each kernel of the call
  uint32_t* err;
  int heap_out;            // write heap indices instead of ids
  uint32_t lanes;          // count / digest: lanes per box (1, 2, 4, 8, 16; 0 or 32: one warp per box)
  const uint32_t* evsel;   // batched search over a subset of the events (null: all boxes in order)
  const uint64_t* evsel_q; // exclusive prefix of the subset's box counts (nsel + 1 entries)
  uint32_t nsel;
  // recording count pass (fkd_walk.cu; null ents: no record): every box's result as a list of
  // entries in in-order position, which k_emit writes out
  uint2* ents;
  unsigned long long* ent_ctr;   // entries reserved (zeroed by the caller; counts past ent_cap)
  uint64_t ent_cap;
  uint2* erec;                   // per box: its first entry, its entries
  uint32_t* ehist;               // ordered lists: 32 words per box, where each depth's results start
  uint32_t* flags;               // boxes whose entries did not fit (the write pass traverses them)
  unsigned long long* flag_ctr;  // (zeroed by the caller)
  // leaf buckets (needs tab.ipts): visited subtrees of height <= bucket are
  // scanned in in-order layout instead of walked (0: walk every level)
  uint32_t bucket;
  uint32_t bucket_grp;           // the same for the searches with fewer than 32 lanes per box (one lane
                                 // scans a bucket of at most 2^(h+1)-1 points)
  // packets (fkd_packet.cu): the boxes of packets that gave up, and their number
  uint32_t* loose;
  unsigned long long* loose_ctr;
  const unsigned long long* qdev;  // the number of boxes when only the device knows it (null: boxes.q)
  cudaStream_t stream;
};

cudaError_t launch_search(const SearchCtx& sc, int dim, int mode);
// One box searched by one warp, level by level (no count pass): out[0] the
// result count, out[1] a frontier overflow flag, out[4 ..] the first cap ids
// in ascending heap order.
struct OneBox {
  float lo[4], hi[4];
};
cudaError_t launch_one(const Table& tab, uint32_t n, int dim, const OneBox& bx, uint32_t* out, uint32_t cap,
                       cudaStream_t stream);
// fkd_walk.cu: count / digest search of one box per warp by the subtrees'
// bounding boxes (needs tab.bb, tab.ipts; 4-D: tab.dids); with sc.ents a count
// also records the results.
cudaError_t launch_walk(const SearchCtx& sc, int dim, int mode);
// The same for balls (radius search): sc.boxes.lo = centres, sc.boxes.hi =
// radii; a count, or (sc.ents, sc.ehist) a recorded ordered list.
cudaError_t launch_walk_balls(const SearchCtx& sc, int dim);
// Writes the recorded results to sc.out (needs tab.dids), in the reference's
// order or in in-order position.
cudaError_t launch_emit(const SearchCtx& sc, int ordered);
// fkd_tables.cu: fills those of tab.dids / ipts / bb / sdig that are
// set, for every event (max_n: the largest event's points).  The write passes
// need dids, SEARCH_DIGEST sdig, the leaf-bucket scans ipts, the
// packets bb and ipts.
cudaError_t launch_tables(const EvDesc* evs, uint32_t nev, uint32_t max_n, const Table& tab, int dim,
                          cudaStream_t stream);
// Largest leaf-bucket height the searches accept (subtrees of up to 2^(h+1)-1 points).
constexpr uint32_t BUCKET_MAX = 6;
// Sorts every box's result slice by heap index and maps it to ids; with
// `list` only the boxes list[0 .. *nlist).
cudaError_t launch_order_results(const Geom& g, const Table& tab, const uint64_t* offsets, uint64_t q, uint32_t* out,
                                 uint64_t capacity, uint32_t* tmp, uint32_t* err, cudaStream_t stream, const uint32_t* list = nullptr,
                                 const unsigned long long* nlist = nullptr);
// Processing order of the boxes (see fkd_search.cu); scratch holds
// box_order_words(q) words; *order_out points into it.
size_t box_order_words(uint64_t q);
// start_out (optional, for boxes): per box, the first node the box straddles
// -- the walk from the root would visit one child of each of its ancestors, and
// none of their points is inside.
cudaError_t launch_box_order(const Geom& g, const Table& tab, const Boxes& b, int dim, uint32_t* scratch,
                             uint32_t** order_out, cudaStream_t stream, uint32_t** start_out = nullptr,
                             uint32_t* ticket = nullptr);
// fkd_nn.cu: radius search (a warp per query) and k-nearest-neighbour search
// (a warp per query where the derived tables are there and knn_by_warps, else a
// thread per query); ctr is the SoA centre array of stride q.  launch_radius counts into
// `counts` when `out` is null, else writes heap indices (heap_out) or ids at
// `offsets`; with nq only the queries order[0 .. *nq).
constexpr uint32_t KNN_MAX = 64;
cudaError_t launch_radius(const Geom& g, const Table& tab, const float* ctr, const float* rad, uint64_t q,
                          const uint32_t* order, uint32_t* counts, const uint64_t* offsets, uint32_t* out,
                          int heap_out, uint32_t* err, int dim, cudaStream_t stream,
                          const unsigned long long* nq = nullptr);
bool knn_by_warps(int dim, uint32_t k, uint64_t q, uint64_t n);
cudaError_t launch_knn(const Geom& g, const Table& tab, const float* ctr, uint64_t q, const uint32_t* order,
                       uint32_t k, uint32_t* ids, float* d2, uint32_t* err, int dim, cudaStream_t stream);
// fkd_packet.cu: count / digest search of 32 neighbouring boxes per warp.
// Needs sc.order (boxes of one event contiguous), tab.bb (4-D: tab.dids) and
// sc.loose (sc.boxes.q entries, which may overlay nothing sc.order uses): the
// boxes of packets that give up are searched by launch_walk.
cudaError_t launch_packets(SearchCtx& sc, int dim, int mode);
// Spatial order of a batch's boxes, event by event; scratch holds
// event_order_words words, *order_out points into it.  Its first b.q words are
// free again afterwards.
size_t event_order_words(uint64_t npts, uint32_t nev, uint64_t q);
cudaError_t launch_event_order(const EvDesc* evs, uint32_t nev, uint64_t npts, const Table& tab, const Boxes& b, int dim,
                               uint32_t* scratch, uint32_t** order_out, cudaStream_t stream);
// Exclusive prefix sum of q uint32 counts into q+1 uint64 offsets.
// ticket (optional): a zero word, used up by the call, that saves a launch;
// total (optional) receives offsets[q] too.
cudaError_t launch_scan_counts(const uint32_t* counts, uint64_t q, uint64_t* offsets, unsigned long long* partials,
                               cudaStream_t stream, uint32_t* ticket = nullptr, uint64_t* total = nullptr);
// The work counter of a kernel of sc's call (QC_*), zero.
cudaError_t work_counter(SearchCtx& sc, int which);
size_t scan_partials_words(uint64_t q);

}  // namespace fkd
