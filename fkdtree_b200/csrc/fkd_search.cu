// fkd_search.cu -- box search on the flat tree (sm_100a).
//
// Semantics: FKDTree_CPU::search_in_the_box (FKDTree_cpu.h:123-169) and its
// BFS / branchless / recursive variants (:72-121, :25-70, :171-207) all return
// the ids of exactly the points inside the closed box (intersects /
// is_in_the_box, FKDTree_cpu.h:302-321): a child is skipped only when the
// node's split value proves the whole subtree lies outside.  The GPU visits
// the same children by the same tests -- left unless v < lo[c], right when
// v < lo[c] or lo[c] <= v <= hi[c] -- so its result set is the reference's.
//
// Shape: one warp per box, boxes handed out by an atomic counter to a
// persistent grid.  The frontier is a per-warp stack in shared memory (the
// FQueue replacement): the warp pops up to 32 nodes, each lane tests one node
// with a single 16-byte load, and the children are pushed back in lane order.
// Popping the top 32 of a depth-sorted stack keeps it depth-sorted and leaves
// at most min(64, 2^d) entries at depth d (stack_cap); the bound is still
// checked and reported (FKD_ERR_CAPACITY) rather than trusted.
//
// Every node also carries a 2*dim-bit mask saying which sides of its cell
// (the closed slab its ancestors' split values bound it by) already lie
// inside the box.  A child whose mask is full is inside entirely: its
// subtree is counted in closed form and, when ids are wanted, copied as one
// contiguous run of the in-order id table (fkd_tables.cu): the subtree of node
// (d, t) holds exactly the in-order positions [start(d,t), start(d,t) + len(d,t)),
// the interval the build gave it.
//
// Two passes ("count then write"): a count pass fills counts, a prefix sum
// turns them into offsets, and the ids go to every box's slice.  Usually the
// count pass records the boxes' results and k_emit writes them out
// (fkd_walk.cu); k_search_write below, the traversing write pass, serves
// fkd_search_write of unordered lists and the boxes a full entry pool missed.
// Counts and digests come from packets of boxes (fkd_packet.cu), a warp per
// box (fkd_walk.cu) or 1-16 lanes per box (k_search_grp), several boxes per
// warp.
#include <math.h>

#include "fkd_walk.cuh"

namespace fkd {

constexpr int QT = 128;  // threads per CTA
constexpr int QW = QT / 32;
constexpr int JOBS = 256;      // contained-subtree jobs buffered per warp
constexpr int JFLUSH = JOBS - 64;  // one step adds at most 64
#ifndef FKD_EU
#define FKD_EU 4
#endif
constexpr int EU = FKD_EU;         // emission windows with loads in flight (measured: 4 beats 2 by 5%)
constexpr int BQ = 128;          // leaf buckets queued per warp (one step adds at most 64)

__device__ __forceinline__ uint32_t lanemask_lt_s() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

__device__ __forceinline__ float sel4(uint32_t c, float a, float b, float d, float e) {
  return c == 0 ? a : (c == 1 ? b : (c == 2 ? d : e));
}

// The geometry of the deepest trees (2^31 - 1 points).
inline Geom deepest() { return make_geom(0x7fffffffu); }

// Popping the top 32 of a depth-sorted stack leaves at most 64 entries per
// depth, and depth d has only 2^d nodes: sum over d of min(64, 2^d), plus one.
// With leaf buckets of height b (and the in-order nodes to scan them) no node
// deeper than H - b - 1 is ever pushed.
__host__ __device__ inline uint32_t stack_cap(const Geom& g, uint32_t bucket = 0u) {
  const uint32_t dmax = bucket ? (g.H > bucket ? g.H - bucket - 1u : 0u) : g.H;
  uint32_t c = 1u;
  for (uint32_t d = 0; d <= dmax; ++d) c += d < 6u ? (1u << d) : 64u;
  return c;
}

// Copies the concatenation of nj runs of in-order positions -- run k starts at
// position st[k] and lands at out[base + pre[k]], pre being the exclusive
// prefix of the run lengths and total their sum -- with one warp: their ids
// (dids), or their heap indices.
// Each lane step writes 32 consecutive output slots; a lane finds its run
// from the bitmask of the runs that start inside the window (EU windows with
// loads in flight).  st / pre live in shared memory; slots at or past
// `limit` are not written and set `failed`.
__device__ __forceinline__ void copy_runs(const uint32_t* st, const uint32_t* pre, uint32_t nj, uint32_t total,
                                          const Geom& g, const uint32_t* __restrict__ dids, bool heap,
                                          uint32_t* __restrict__ out,
                                          uint64_t base, uint64_t limit, bool& failed) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t jb = 0u;  // the run holding output slot o0 (warp-uniform)
  for (uint32_t o0 = 0; o0 < total; o0 += 32u * EU) {
    uint32_t src[EU];
    bool ok[EU];
#pragma unroll
    for (int u = 0; u < EU; ++u) {
      const uint32_t w0 = o0 + 32u * u;
      const uint32_t k = jb + lane;
      const bool kv = k < nj;
      const uint32_t pk = kv ? pre[k] : total;
      const uint32_t sk = kv ? st[k] : 0u;
      // runs after jb start after w0 (every run holds at least one id)
      const uint32_t B = __reduce_or_sync(0xffffffffu, (lane > 0u && kv && pk < w0 + 32u) ? (1u << (pk - w0)) : 0u);
      const uint32_t jl = __popc(B & (0xffffffffu >> (31u - lane)));
      const uint32_t mp = __shfl_sync(0xffffffffu, pk, jl);
      const uint32_t ms = __shfl_sync(0xffffffffu, sk, jl);
      ok[u] = w0 + lane < total;
      src[u] = ms + (w0 + lane - mp);
      // the run holding w0 + 32: the one holding w0 + 31, or the next if it starts there
      uint32_t nb = jb + __popc(B);
      if (nb + 1u < nj && pre[nb + 1u] == w0 + 32u) ++nb;
      jb = nb;
    }
    uint32_t v[EU];
#pragma unroll
    for (int u = 0; u < EU; ++u) {
      uint32_t d, t;
      v[u] = ok[u] ? (heap ? inorder_node(g, src[u], &d, &t) : __ldg(dids + src[u])) : 0u;
    }
#pragma unroll
    for (int u = 0; u < EU; ++u) {
      if (ok[u]) {
        const uint64_t pos = base + o0 + 32u * u + lane;
        if (pos < limit)
          out[pos] = v[u];
        else
          failed = true;
      }
    }
  }
}

// The traversing write pass: a warp per box, for boxes no recording count
// pass served (fkd_search_write of unordered lists, a full entry pool).
template <int DIM>
__global__ void __launch_bounds__(QT, 8) k_search_write(SearchCtx sc, uint32_t cap) {
  chain_wait();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t jst[QW][JOBS];   // in-order start of each buffered subtree
  __shared__ uint32_t jlen[QW][JOBS];  // its size
  __shared__ uint32_t jpre[QW][JOBS];  // exclusive prefix of the sizes
  __shared__ uint32_t bq_st[QW][BQ];   // leaf buckets: in-order start of each queued subtree
  __shared__ uint32_t bq_len[QW][BQ];  // its size (the scan overwrites it with the exclusive prefix)
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t* stk_node = (uint32_t*)smem_raw + (size_t)warp * cap;
  uint8_t* stk_mask = (uint8_t*)((uint32_t*)smem_raw + (size_t)QW * cap) + (size_t)warp * cap;
  constexpr uint32_t FULL = (1u << (2 * DIM)) - 1u;
  const uint32_t lt = lanemask_lt_s();
  const uint64_t nq = sc.qdev ? *sc.qdev : sc.boxes.q;
  const Geom g = sc.g;
  const Table tab = sc.tab;
  const uint32_t n = g.n;
  // children at depth >= bdep are leaf buckets: subtrees of height <= sc.bucket, scanned in in-order layout
  const uint32_t bdep = (tab.ipts && sc.bucket) ? (g.H > sc.bucket ? g.H - sc.bucket : 0u) : 0xffffffffu;

  for (;;) {
    uint32_t qi = 0;
    if (lane == 0) qi = atomicAdd(sc.qcounter, 1u);
    qi = __shfl_sync(0xffffffffu, qi, 0);
    if ((uint64_t)qi >= nq) break;
    const uint32_t qj = sc.order ? sc.order[qi] : qi;
    float lo[4] = {0.f, 0.f, 0.f, 0.f}, hi[4] = {0.f, 0.f, 0.f, 0.f};
    uint32_t mask0 = 0u;
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      lo[c] = sc.boxes.lo[(uint64_t)c * sc.boxes.stride + qj];
      hi[c] = sc.boxes.hi[(uint64_t)c * sc.boxes.stride + qj];
      if (lo[c] == -INFINITY) mask0 |= 1u << (2 * c);
      if (hi[c] == INFINITY) mask0 |= 2u << (2 * c);
    }
    uint64_t cursor = sc.offsets[qj];
    const uint64_t cend = sc.offsets[qj + 1u];
    bool failed = false;
    uint32_t njobs = 0;  // warp-uniform

    // Emits one id per lane with v set, packed at the cursor.
    auto emit_ballot = [&](bool v, uint32_t node, uint32_t id) {
      const uint32_t bv = __ballot_sync(0xffffffffu, v);
      if (v) {
        const uint64_t pos = cursor + __popc(bv & lt);
        if (pos < cend && pos < sc.capacity)
          sc.out[pos] = sc.heap_out ? node : id;
        else
          failed = true;
      }
      cursor += __popc(bv);
    };

    // Emits the whole subtrees buffered in the job list: job k is the run
    // [jst[k], jst[k] + jlen[k]) of in-order positions, where every subtree is
    // one contiguous range; the runs are concatenated at the cursor.
    auto run_jobs = [&](uint32_t nj) {
      uint32_t carry = 0u;
      for (uint32_t e0 = 0; e0 < nj; e0 += 32u) {
        const uint32_t e = e0 + lane;
        const uint32_t len = e < nj ? jlen[warp][e] : 0u;
        uint32_t incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= (uint32_t)o) incl += y;
        }
        if (e < nj) jpre[warp][e] = carry + incl - len;
        carry += __shfl_sync(0xffffffffu, incl, 31);
      }
      __syncwarp();
      const uint64_t limit = cend < sc.capacity ? cend : sc.capacity;
      copy_runs(jst[warp], jpre[warp], nj, carry, g, tab.dids, sc.heap_out != 0, sc.out, cursor, limit, failed);
      cursor += carry;
      __syncwarp();
    };

    // Scans the queued leaf buckets: bucket k is the in-order range
    // [bq_st[k], bq_st[k] + bq_len[k]) of a subtree the walk would enter;
    // the ranges are concatenated and every lane tests one point per step
    // (16-byte loads of consecutive in-order nodes) -- the same points the
    // walk would have found, since the walk only skips subtrees that lie
    // outside the box.
    uint32_t nb = 0;  // queued buckets (warp-uniform)
    auto scan_buckets = [&](uint32_t nbk) {
      uint32_t carry = 0u;
      for (uint32_t e0 = 0; e0 < nbk; e0 += 32u) {
        const uint32_t e = e0 + lane;
        const uint32_t len = e < nbk ? bq_len[warp][e] : 0u;
        uint32_t incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= (uint32_t)o) incl += y;
        }
        if (e < nbk) bq_len[warp][e] = carry + incl - len;
        carry += __shfl_sync(0xffffffffu, incl, 31);
      }
      __syncwarp();
      const uint32_t total = carry;
      uint32_t jb = 0u;  // the bucket holding slot w0 (warp-uniform)
      for (uint32_t w0 = 0; w0 < total; w0 += 32u) {
        const uint32_t k = jb + lane;
        const bool kv = k < nbk;
        const uint32_t pk = kv ? bq_len[warp][k] : total;
        const uint32_t sk = kv ? bq_st[warp][k] : 0u;
        // buckets after jb start after w0 (every bucket holds at least one point)
        const uint32_t B = __reduce_or_sync(0xffffffffu, (lane > 0u && kv && pk < w0 + 32u) ? (1u << (pk - w0)) : 0u);
        const uint32_t jl = __popc(B & (0xffffffffu >> (31u - lane)));
        const uint32_t mp = __shfl_sync(0xffffffffu, pk, jl);
        const uint32_t ms = __shfl_sync(0xffffffffu, sk, jl);
        uint32_t nbn = jb + __popc(B);
        if (nbn + 1u < nbk && bq_len[warp][nbn + 1u] == w0 + 32u) ++nbn;
        const bool ok = w0 + lane < total;
        const uint32_t pos = ms + (w0 + lane - mp);
        jb = nbn;
        bool hit = ok;
        uint32_t idv = 0u, node = 0u;
        if (ok) {
          const uint4 pt = __ldg(tab.ipts + pos);
          if (DIM > 0) hit &= (__uint_as_float(pt.x) <= hi[0] && __uint_as_float(pt.x) >= lo[0]);
          if (DIM > 1) hit &= (__uint_as_float(pt.y) <= hi[1] && __uint_as_float(pt.y) >= lo[1]);
          if (DIM > 2) hit &= (__uint_as_float(pt.z) <= hi[2] && __uint_as_float(pt.z) >= lo[2]);
          if (DIM > 3) hit &= (__uint_as_float(pt.w) <= hi[3] && __uint_as_float(pt.w) >= lo[3]);
          idv = pt.w;
        }
        if (hit) {
          uint32_t d, t;
          if (sc.heap_out)
            node = inorder_node(g, pos, &d, &t);
          else if (DIM > 3)
            idv = __ldg(tab.dids + pos);
        }
        emit_ballot(hit, node, idv);
      }
      __syncwarp();
    };

    int top = 0;
    if (n > 0) {
      if (mask0 == FULL) {
        if (lane == 0) {
          jst[warp][0] = 0u;
          jlen[warp][0] = n;
        }
        njobs = 1;
        __syncwarp();
      } else {
        // descend, all lanes alike, while the box lies on one side of the
        // node's split: such a node is outside the box and the walk would
        // visit only that one child; the walk starts at the first node the
        // box straddles (its cell's mask is still mask0)
        uint32_t r = 0u, dep = 0u;
        bool empty = false;
        while (dep + 1u < bdep) {
          const uint32_t c = dep % (uint32_t)DIM;
          const uint4 nd = __ldg(tab.nodes + r);
          const float v = sel4(c, __uint_as_float(nd.x), __uint_as_float(nd.y), __uint_as_float(nd.z),
                               __uint_as_float(nd.w));
          const float loc = sel4(c, lo[0], lo[1], lo[2], lo[3]);
          const float hic = sel4(c, hi[0], hi[1], hi[2], hi[3]);
          uint32_t nx;
          if (v < loc)
            nx = 2u * r + 2u;  // the walk visits the right child only
          else if (v > hic)
            nx = 2u * r + 1u;  // the left child only
          else
            break;
          if (nx >= n) {  // that child does not exist: nothing is inside
            empty = true;
            break;
          }
          r = nx;
          ++dep;
        }
        if (!empty) {
          if (lane == 0) {
            stk_node[0] = r;
            stk_mask[0] = (uint8_t)(mask0 | (DIM == 3 ? ((dep % 3u) << 6) : 0u));
          }
          top = 1;
        }
      }
    }
    __syncwarp();

    while (top > 0) {
      const int gcount = top < 32 ? top : 32;
      const int base = top - gcount;
      const bool have = (int)lane < gcount;
      uint32_t i = 0u, mask = 0u;
      if (have) {
        i = stk_node[base + lane];
        mask = stk_mask[base + lane];
      }
      __syncwarp();
      top = base;
      bool emit = false, pushL = false, pushR = false, contL = false, contR = false;
      bool bucketL = false, bucketR = false;
      uint32_t maskL = 0u, maskR = 0u, idv = 0u, cnext = 0u;
      if (have) {
        // 3D: the node's split dimension rides in the top bits of its mask byte
        uint32_t c;
        if (DIM == 3) {
          c = mask >> 6;
          mask &= 0x3fu;
        } else {
          c = floor_log2_u32(i + 1u) % DIM;
        }
        cnext = c + 1u == (uint32_t)DIM ? 0u : c + 1u;
        const uint4 nd = __ldg(tab.nodes + i);
        const float x0 = __uint_as_float(nd.x), x1 = __uint_as_float(nd.y), x2 = __uint_as_float(nd.z),
                    x3 = __uint_as_float(nd.w);
        const float v = sel4(c, x0, x1, x2, x3);
        const float loc = sel4(c, lo[0], lo[1], lo[2], lo[3]);
        const float hic = sel4(c, hi[0], hi[1], hi[2], hi[3]);
        const bool inter = v <= hic && v >= loc;
        const bool lower = v < loc;
        if (inter) {
          bool in = true;
          if (DIM > 0) in &= (x0 <= hi[0] && x0 >= lo[0]);
          if (DIM > 1) in &= (x1 <= hi[1] && x1 >= lo[1]);
          if (DIM > 2) in &= (x2 <= hi[2] && x2 >= lo[2]);
          if (DIM > 3) in &= (x3 <= hi[3] && x3 >= lo[3]);
          emit = in;
        }
        if (emit) idv = DIM <= 3 ? nd.w : __ldg(tab.ids + i);
        const uint32_t l = 2u * i + 1u;
        const bool visitL = !lower && l < n;
        const bool visitR = (lower || inter) && l + 1u < n;
        maskL = mask | (v <= hic ? (2u << (2 * c)) : 0u);
        maskR = mask | (v >= loc ? (1u << (2 * c)) : 0u);
        contL = visitL && maskL == FULL;
        contR = visitR && maskR == FULL;
        pushL = visitL && !contL;
        pushR = visitR && !contR;
        if (pushL || pushR) {
          // children at the bucket depth are scanned, not walked
          const uint32_t dep = 31u - (uint32_t)__clz(i + 1u);
          if (dep + 1u >= bdep) {
            bucketL = pushL;
            bucketR = pushR;
            pushL = pushR = false;
          }
        }
      }
      emit_ballot(emit, i, idv);
      // buffer the contained subtrees; emit them in bulk when the buffer fills
      const uint32_t bl = __ballot_sync(0xffffffffu, contL), br = __ballot_sync(0xffffffffu, contR);
      const uint32_t jp = njobs + __popc(bl & lt) + __popc(br & lt);
      if (contL || contR) {
        // the children of node (dep, t) are (dep + 1, 2t) and (dep + 1, 2t + 1)
        const uint32_t dc = floor_log2_u32(i + 1u) + 1u;
        const uint32_t tl = 2u * (i + 1u - (1u << (dc - 1u)));
        if (contL) {
          jst[warp][jp] = seg_start(g, dc, tl);
          jlen[warp][jp] = seg_len(g, dc, tl);
        }
        if (contR) {
          const uint32_t q2 = jp + (contL ? 1u : 0u);
          jst[warp][q2] = seg_start(g, dc, tl + 1u);
          jlen[warp][q2] = seg_len(g, dc, tl + 1u);
        }
      }
      njobs += __popc(bl) + __popc(br);
      if (njobs > (uint32_t)JFLUSH) {
        __syncwarp();
        run_jobs(njobs);
        njobs = 0;
      }
      // push the children in lane order (keeps the stack depth-sorted)
      const uint32_t bpl = __ballot_sync(0xffffffffu, pushL), bpr = __ballot_sync(0xffffffffu, pushR);
      const uint32_t tot = __popc(bpl) + __popc(bpr);
      if ((uint32_t)top + tot > cap) {
        failed = true;
        break;
      }
      uint32_t p = (uint32_t)top + __popc(bpl & lt) + __popc(bpr & lt);
      const uint32_t ctag = DIM == 3 ? cnext << 6 : 0u;
      if (pushL) {
        stk_node[p] = 2u * i + 1u;
        stk_mask[p] = (uint8_t)(maskL | ctag);
        ++p;
      }
      if (pushR) {
        stk_node[p] = 2u * i + 2u;
        stk_mask[p] = (uint8_t)(maskR | ctag);
      }
      top += (int)tot;
      // queue the leaf buckets
      const uint32_t bbl = __ballot_sync(0xffffffffu, bucketL), bbr = __ballot_sync(0xffffffffu, bucketR);
      if (bbl | bbr) {
        uint32_t q = nb + __popc(bbl & lt) + __popc(bbr & lt);
        if (bucketL || bucketR) {
          const uint32_t dc = floor_log2_u32(i + 1u) + 1u;
          const uint32_t tl = 2u * (i + 1u - (1u << (dc - 1u)));
          if (bucketL) {
            bq_st[warp][q] = seg_start(g, dc, tl);
            bq_len[warp][q] = seg_len(g, dc, tl);
            ++q;
          }
          if (bucketR) {
            bq_st[warp][q] = seg_start(g, dc, tl + 1u);
            bq_len[warp][q] = seg_len(g, dc, tl + 1u);
          }
        }
        nb += __popc(bbl) + __popc(bbr);
        if (nb > (uint32_t)(BQ - 64)) {
          __syncwarp();
          scan_buckets(nb);
          nb = 0;
        }
      }
      __syncwarp();
    }
    if (nb) {
      __syncwarp();
      scan_buckets(nb);
      nb = 0;
    }
    if (njobs) {
      __syncwarp();
      run_jobs(njobs);
    }
    if (lane == 0 && cursor != cend) atomicOr(sc.err, ERRB_INTERNAL);
    if (__any_sync(0xffffffffu, failed) && lane == 0) atomicOr(sc.err, ERRB_CAPACITY);
    __syncwarp();
  }
}

// Count / digest with G < 32 lanes per box (G = 1: a thread per box): a warp
// holds 32/G boxes, each group with its own depth-sorted stack (popping the
// top G keeps at most 2G entries per depth, so 2G*(H+1) + 1 bound it), and a
// group that finishes takes the next box at once.  Small boxes near the root
// keep only a few nodes in flight; packing several per warp fills the lanes
// those steps leave idle.  Same node tests as k_search_write; contained subtrees are
// counted in closed form, or by their digest.
__host__ __device__ inline uint32_t stack_cap_lanes(const Geom& g, uint32_t G) { return 2u * G * (g.H + 1u) + 1u; }

template <int DIM, int MODE, int G, bool BKT>
__global__ void __launch_bounds__(QT) k_search_grp(SearchCtx sc, uint32_t cap) {
  chain_wait();
  static_assert(G == 1 || G == 2 || G == 4 || G == 8 || G == 16, "group width");
  constexpr int NG = QT / G;
  constexpr uint32_t GM = (1u << G) - 1u;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t grp = threadIdx.x / G, gl = threadIdx.x % G;
  const uint32_t gsh = lane & ~(uint32_t)(G - 1);
  const uint32_t gmask = GM << gsh;
  const uint32_t glt = (1u << gl) - 1u;
  uint32_t* stk_node = (uint32_t*)smem_raw + (size_t)grp * cap;
  uint8_t* stk_mask = (uint8_t*)((uint32_t*)smem_raw + (size_t)NG * cap) + (size_t)grp * cap;
  constexpr uint32_t FULL = (1u << (2 * DIM)) - 1u;

  uint32_t cur_ev = 0;
  bool active = false, exhausted = false, failed = false;
  int top = 0;
  uint64_t oj = 0;
  Geom g = sc.g;
  Table tab = sc.tab;
  float lo[4] = {0.f, 0.f, 0.f, 0.f}, hi[4] = {0.f, 0.f, 0.f, 0.f};
  unsigned long long acc = 0ull, acc2 = 0ull;
  // children at depth >= bdep are leaf buckets: pushed with BUCKET_BIT set and,
  // when popped, their points scanned by the lane that popped them
  uint32_t bdep = 0xffffffffu;
  constexpr uint32_t BUCKET_BIT = 0x80000000u;  // node indices stay below 2^31

  // the group's result for its current box (group-uniform call)
  auto finish = [&]() {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      acc += __shfl_xor_sync(gmask, acc, o);
      if (MODE == SEARCH_DIGEST) acc2 += __shfl_xor_sync(gmask, acc2, o);
    }
    const bool anyfail = __any_sync(gmask, failed);
    if (gl == 0) {
      if (MODE == SEARCH_COUNT) {
        sc.counts[oj] = (uint32_t)acc;
        if (acc > 0xffffffffull) atomicOr(sc.err, ERRB_CAPACITY);
      } else {
        sc.digests[oj] = acc;
        sc.counts[oj] = (uint32_t)acc2;
      }
      if (anyfail) atomicOr(sc.err, ERRB_CAPACITY);
    }
    active = false;
    failed = false;
  };

  for (;;) {
    // groups without a box take boxes until one needs a traversal
    while (!active && !exhausted) {
      uint32_t qi = 0;
      if (gl == 0) qi = atomicAdd(sc.qcounter, 1u);
      qi = __shfl_sync(gmask, qi, 0, G);
      if ((uint64_t)qi >= sc.boxes.q) {
        exhausted = true;
        break;
      }
      uint32_t qj = sc.order ? sc.order[qi] : qi;
      if (sc.evsel) qj = select_box(sc, qi, cur_ev);
      oj = qj;
      g = sc.g;
      tab = sc.tab;
      const float* blo = sc.boxes.lo;
      const float* bhi = sc.boxes.hi;
      uint64_t bstride = sc.boxes.stride, bj = qj;
      if (sc.evs) {
        while (cur_ev + 1u < sc.nev && (uint64_t)qj >= sc.evs[cur_ev + 1u].qbase) ++cur_ev;
        const EvDesc& ev = sc.evs[cur_ev];
        g = ev.g;
        tab.nodes = sc.tab.nodes + ev.base;
        tab.ids = sc.tab.ids + ev.base;
        tab.sdig = sc.tab.sdig ? sc.tab.sdig + ev.base : nullptr;
        tab.ipts = sc.tab.ipts ? sc.tab.ipts + ev.base : nullptr;
        tab.dids = sc.tab.dids ? sc.tab.dids + ev.base : nullptr;
        blo = sc.boxes.lo + ev.qcbase;
        bhi = sc.boxes.hi + ev.qcbase;
        bstride = ev.nq;
        bj = qj - ev.qbase;
        oj = ev.qout + bj;
      }
      uint32_t mask0 = 0u;
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        lo[c] = blo[(uint64_t)c * bstride + bj];
        hi[c] = bhi[(uint64_t)c * bstride + bj];
        if (lo[c] == -INFINITY) mask0 |= 1u << (2 * c);
        if (hi[c] == INFINITY) mask0 |= 2u << (2 * c);
      }
      acc = 0ull;
      acc2 = 0ull;
      if (BKT) bdep = (tab.ipts && sc.bucket_grp) ? (g.H > sc.bucket_grp ? g.H - sc.bucket_grp : 0u) : 0xffffffffu;
      if (g.n == 0) {
        finish();
      } else if (mask0 == FULL) {
        if (gl == 0) {
          if (MODE == SEARCH_COUNT) {
            acc = g.n;
          } else {
            acc = tab.sdig[0];
            acc2 = g.n;
          }
        }
        finish();
      } else {
        // (no descent here: a group taking a box would hold up the other
        // groups of its warp for a chain of dependent loads)
        if (gl == 0) {
          stk_node[0] = 0u;
          stk_mask[0] = (uint8_t)mask0;
        }
        top = 1;
        active = true;
      }
    }
    if (!__any_sync(0xffffffffu, active)) break;
    __syncwarp();

    const int gcount = top < G ? top : G;
    const int base = top - gcount;
    const bool have = (int)gl < gcount;
    uint32_t i = 0u, mask = 0u;
    if (have) {
      i = stk_node[base + gl];
      mask = stk_mask[base + gl];
    }
    __syncwarp();
    top = base;
    bool pushL = false, pushR = false, bucket = false;
    uint32_t maskL = 0u, maskR = 0u;
    if (BKT && have && (i & BUCKET_BIT)) {
      // a leaf bucket: its subtree is the in-order range [S, S + len)
      bucket = true;
      const uint32_t nb = i & ~BUCKET_BIT;
      const uint32_t dep = floor_log2_u32(nb + 1u);
      const uint32_t t = nb + 1u - (1u << dep);
      const uint32_t S = seg_start(g, dep, t), len = seg_len(g, dep, t);
      for (uint32_t k = 0; k < len; ++k) {
        const uint4 pt = __ldg(tab.ipts + S + k);
        bool in = true;
        if (DIM > 0) in &= (__uint_as_float(pt.x) <= hi[0] && __uint_as_float(pt.x) >= lo[0]);
        if (DIM > 1) in &= (__uint_as_float(pt.y) <= hi[1] && __uint_as_float(pt.y) >= lo[1]);
        if (DIM > 2) in &= (__uint_as_float(pt.z) <= hi[2] && __uint_as_float(pt.z) >= lo[2]);
        if (DIM > 3) in &= (__uint_as_float(pt.w) <= hi[3] && __uint_as_float(pt.w) >= lo[3]);
        if (in) {
          if (MODE == SEARCH_COUNT) {
            acc += 1u;
          } else {
            acc2 += 1u;
            acc += mix64(DIM <= 3 ? pt.w : __ldg(tab.dids + S + k));
          }
        }
      }
    }
    if (have && !bucket) {
      const uint32_t dep = floor_log2_u32(i + 1u);
      const uint32_t c = dep % DIM;
      const uint4 nd = __ldg(tab.nodes + i);
      const float x0 = __uint_as_float(nd.x), x1 = __uint_as_float(nd.y), x2 = __uint_as_float(nd.z),
                  x3 = __uint_as_float(nd.w);
      const float v = sel4(c, x0, x1, x2, x3);
      const float loc = sel4(c, lo[0], lo[1], lo[2], lo[3]);
      const float hic = sel4(c, hi[0], hi[1], hi[2], hi[3]);
      const bool inter = v <= hic && v >= loc;
      const bool lower = v < loc;
      bool emit = false;
      if (inter) {
        bool in = true;
        if (DIM > 0) in &= (x0 <= hi[0] && x0 >= lo[0]);
        if (DIM > 1) in &= (x1 <= hi[1] && x1 >= lo[1]);
        if (DIM > 2) in &= (x2 <= hi[2] && x2 >= lo[2]);
        if (DIM > 3) in &= (x3 <= hi[3] && x3 >= lo[3]);
        emit = in;
      }
      const uint32_t l = 2u * i + 1u;
      const bool visitL = !lower && l < g.n;
      const bool visitR = (lower || inter) && l + 1u < g.n;
      maskL = mask | (v <= hic ? (2u << (2 * c)) : 0u);
      maskR = mask | (v >= loc ? (1u << (2 * c)) : 0u);
      const bool contL = visitL && maskL == FULL;
      const bool contR = visitR && maskR == FULL;
      pushL = visitL && !contL;
      pushR = visitR && !contR;
      const uint32_t cnt = (emit ? 1u : 0u) + (contL ? subtree_size(g, l) : 0u) + (contR ? subtree_size(g, l + 1u) : 0u);
      if (MODE == SEARCH_COUNT) {
        acc += cnt;
      } else {
        acc2 += cnt;
        if (emit) acc += mix64(DIM <= 3 ? nd.w : __ldg(tab.ids + i));
        if (contL) acc += tab.sdig[l];
        if (contR) acc += tab.sdig[l + 1u];
      }
    }
    const uint32_t bpl = (__ballot_sync(0xffffffffu, pushL) >> gsh) & GM;
    const uint32_t bpr = (__ballot_sync(0xffffffffu, pushR) >> gsh) & GM;
    const uint32_t tot = __popc(bpl) + __popc(bpr);
    if ((uint32_t)top + tot > cap) {
      failed = true;  // group-uniform: abandon the box, report capacity
      top = 0;
    } else {
      uint32_t p = (uint32_t)top + __popc(bpl & glt) + __popc(bpr & glt);
      // children at the bucket depth go on the stack as buckets
      const uint32_t btag = (BKT && (pushL || pushR) && floor_log2_u32(i + 1u) + 1u >= bdep) ? BUCKET_BIT : 0u;
      if (pushL) {
        stk_node[p] = (2u * i + 1u) | btag;
        stk_mask[p] = (uint8_t)maskL;
        ++p;
      }
      if (pushR) {
        stk_node[p] = (2u * i + 2u) | btag;
        stk_mask[p] = (uint8_t)maskR;
      }
      top += (int)tot;
    }
    __syncwarp();
    if (active && top == 0) finish();
  }
}

template <int DIM, int MODE, int G, bool BKT>
static cudaError_t run_search_grp_b(SearchCtx& sc) {
  const uint32_t cap = stack_cap_lanes(sc.g, G);
  const size_t smem = (size_t)(QT / G) * cap * 5u;
  cudaError_t e = allow_smem(k_search_grp<DIM, MODE, G, BKT>, (size_t)(QT / G) * stack_cap_lanes(deepest(), G) * 5u);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_search_grp<DIM, MODE, G, BKT>, QT, smem);
  if (e != cudaSuccess) return e;
  if (per < 1) per = 1;
  uint64_t blocks = (uint64_t)sms * per;
  const uint64_t need = (sc.boxes.q + (QT / G) - 1) / (QT / G);
  if (blocks > need) blocks = need ? need : 1;
  e = work_counter(sc, QC_LANES);
  if (e != cudaSuccess) return e;
  FKD_CHAIN(k_search_grp<DIM, MODE, G, BKT>, dim3((unsigned)blocks), dim3(QT), smem, sc.stream, sc, cap);
  return cudaGetLastError();
}

// The leaf-bucket variant only when buckets are asked for: the plain kernel
// stays free of the bucket branch.
template <int DIM, int MODE, int G>
static cudaError_t run_search_grp(SearchCtx& sc) {
  if (sc.tab.ipts && sc.bucket_grp) return run_search_grp_b<DIM, MODE, G, true>(sc);
  return run_search_grp_b<DIM, MODE, G, false>(sc);
}

cudaError_t work_counter(SearchCtx& sc, int which) {
  if (!sc.qready) return cudaMemsetAsync(sc.qcounter, 0, sizeof(uint32_t), sc.stream);
  sc.qcounter += which;  // (sc is the launch's own copy)
  return cudaSuccess;
}

template <int DIM>
static cudaError_t run_search_write(SearchCtx& sc) {
  const uint32_t cap = stack_cap(sc.g, sc.tab.ipts ? sc.bucket : 0u);
  const size_t smem = (size_t)QW * cap * 5u;
  cudaError_t e = allow_smem(k_search_write<DIM>, (size_t)QW * stack_cap(deepest()) * 5u);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_search_write<DIM>, QT, smem);
  if (e != cudaSuccess) return e;
  if (per < 1) per = 1;
  uint64_t blocks = (uint64_t)sms * per;
  const uint64_t need = (sc.boxes.q + QW - 1) / QW;
  if (blocks > need) blocks = need ? need : 1;
  e = work_counter(sc, QC_WRITE);
  if (e != cudaSuccess) return e;
  FKD_CHAIN(k_search_write<DIM>, dim3((unsigned)blocks), dim3(QT), smem, sc.stream, sc, cap);
  return cudaGetLastError();
}

template <int DIM, int MODE>
static cudaError_t run_search_lanes(SearchCtx& sc) {
  switch (sc.lanes) {
    case 1: return run_search_grp<DIM, MODE, 1>(sc);
    case 2: return run_search_grp<DIM, MODE, 2>(sc);
    case 4: return run_search_grp<DIM, MODE, 4>(sc);
    case 8: return run_search_grp<DIM, MODE, 8>(sc);
    case 16: return run_search_grp<DIM, MODE, 16>(sc);
    default: return launch_walk(sc, DIM, MODE);
  }
}

template <int DIM>
static cudaError_t run_search_mode(SearchCtx& sc, int mode) {
  switch (mode) {
    case SEARCH_COUNT: return run_search_lanes<DIM, SEARCH_COUNT>(sc);
    case SEARCH_WRITE: return run_search_write<DIM>(sc);
    default: return run_search_lanes<DIM, SEARCH_DIGEST>(sc);
  }
}

cudaError_t launch_search(const SearchCtx& call, int dim, int mode) {
  if (call.boxes.q == 0) return cudaSuccess;
  SearchCtx sc = call;
  switch (dim) {
    case 1: return run_search_mode<1>(sc, mode);
    case 2: return run_search_mode<2>(sc, mode);
    case 3: return run_search_mode<3>(sc, mode);
    case 4: return run_search_mode<4>(sc, mode);
    default: return cudaErrorInvalidValue;
  }
}

// ------------------------------------------------------------ box order
//
// Boxes are processed in the order of the tree cell their centre falls in
// (the root-to-depth-D path of the centre, D = min(H, 16)), so the warps
// running at the same time walk neighbouring parts of the tree and share
// its nodes in L2.  The order only changes which warp does which box, never
// a box's result.  On the way down the pass also notes where the box's own walk
// may begin (100,000 small boxes: 254 -> 229 us).

constexpr int QO_BITS = 16;

template <int DIM>
__global__ void k_box_keys(Geom g, Table tab, Boxes b, uint32_t bits, uint32_t* __restrict__ keys,
                           uint32_t* __restrict__ hist, uint32_t* __restrict__ start) {
  chain_wait();
  const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= b.q) return;
  float lo[4] = {0.f, 0.f, 0.f, 0.f}, hi[4] = {0.f, 0.f, 0.f, 0.f}, ctr[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    lo[c] = b.lo[(uint64_t)c * b.stride + j];
    hi[c] = b.hi[(uint64_t)c * b.stride + j];
    ctr[c] = 0.5f * (lo[c] + hi[c]);
  }
  const uint32_t D = g.H < bits ? g.H : bits;
  uint32_t i = 0u, path = 0u, dep = 0u;
  uint32_t first = 0xffffffffu;  // the first node the box does not lie to one side of
  while (dep < D) {
    const uint32_t c = dep % DIM;
    const uint4 nd = __ldg(tab.nodes + i);
    const float v = sel4(c, __uint_as_float(nd.x), __uint_as_float(nd.y), __uint_as_float(nd.z), __uint_as_float(nd.w));
    const uint32_t right = (sel4(c, ctr[0], ctr[1], ctr[2], ctr[3]) < v) ? 0u : 1u;
    // (an empty box or a NaN bound: the walk answers it before it looks at its start)
    if (first == 0xffffffffu && !(right ? v < sel4(c, lo[0], lo[1], lo[2], lo[3]) : v > sel4(c, hi[0], hi[1], hi[2], hi[3])))
      first = i;
    path = (path << 1) | right;
    i = 2u * i + 1u + right;
    ++dep;
    if (i >= g.n) break;
  }
  if (start) start[j] = first != 0xffffffffu ? first : (i < g.n ? i : 0u);
  const uint32_t key = path << (bits - dep);
  keys[j] = key;
  atomicAdd(&hist[key], 1u);
}

__global__ void k_box_scatter(uint64_t q, const uint32_t* __restrict__ keys, unsigned long long* __restrict__ offs,
                              uint32_t* __restrict__ order) {
  chain_wait();
  const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= q) return;
  const unsigned long long pos = atomicAdd(&offs[keys[j]], 1ull);
  if (pos < q) order[pos] = (uint32_t)j;
}

size_t box_order_words(uint64_t q) {
  // keys (q) + hist (2^16) + offsets (2^16 + 1, 64-bit) + partials + order (q) + start (q)
  return q + (1u << QO_BITS) + 2ull * ((1u << QO_BITS) + 1) + 2ull * scan_partials_words(1u << QO_BITS) + 2ull * q + 16;
}

cudaError_t launch_box_order(const Geom& g, const Table& tab, const Boxes& b, int dim, uint32_t* scratch,
                             uint32_t** order_out, cudaStream_t stream, uint32_t** start_out, uint32_t* ticket) {
  *order_out = nullptr;
  if (start_out) *start_out = nullptr;
  if (b.q == 0 || g.n == 0) return cudaSuccess;
  // about four boxes per cell: few boxes need few cells, and a shorter scan
  uint32_t bits = (uint32_t)QO_BITS;
  while (bits > 8u && (4ull << bits) > b.q) --bits;
  uint32_t* keys = scratch;
  uint32_t* hist = keys + b.q;
  unsigned long long* offs = (unsigned long long*)(((uintptr_t)(hist + (1u << QO_BITS)) + 15) & ~(uintptr_t)15);
  unsigned long long* partials = offs + (1u << QO_BITS) + 1;
  uint32_t* order = (uint32_t*)(partials + scan_partials_words(1u << QO_BITS));
  uint32_t* start = start_out ? order + b.q : nullptr;
  cudaError_t e = cudaMemsetAsync(hist, 0, sizeof(uint32_t) << bits, stream);
  if (e != cudaSuccess) return e;
  const unsigned blocks = (unsigned)((b.q + 255) / 256);
  switch (dim) {
    case 1: FKD_CHAIN(k_box_keys<1>, dim3(blocks), dim3(256), 0, stream, g, tab, b, bits, keys, hist, start); break;
    case 2: FKD_CHAIN(k_box_keys<2>, dim3(blocks), dim3(256), 0, stream, g, tab, b, bits, keys, hist, start); break;
    case 3: FKD_CHAIN(k_box_keys<3>, dim3(blocks), dim3(256), 0, stream, g, tab, b, bits, keys, hist, start); break;
    default: FKD_CHAIN(k_box_keys<4>, dim3(blocks), dim3(256), 0, stream, g, tab, b, bits, keys, hist, start); break;
  }
  e = launch_scan_counts(hist, 1u << bits, (uint64_t*)offs, partials, stream, ticket);
  if (e != cudaSuccess) return e;
  FKD_CHAIN(k_box_scatter, dim3(blocks), dim3(256), 0, stream, b.q, keys, offs, order);
  *order_out = order;
  if (start_out) *start_out = start;
  return cudaGetLastError();
}

// ------------------------------------------------------------------- scan

constexpr int SCT = 256;
constexpr int SCIPT = 16;
constexpr int SCB = SCT * SCIPT;

size_t scan_partials_words(uint64_t q) { return (q + SCB - 1) / SCB + 1; }

__device__ __forceinline__ unsigned long long block_excl_scan64(unsigned long long v, unsigned long long* wsum,
                                                                unsigned long long* total) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  unsigned long long incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += y;
  }
  if (lane == 31u) wsum[warp] = incl;
  __syncthreads();
  unsigned long long base = 0ull, tot = 0ull;
  for (uint32_t k = 0; k < blockDim.x / 32u; ++k) {
    if (k < warp) base += wsum[k];
    tot += wsum[k];
  }
  __syncthreads();
  *total = tot;
  return base + incl - v;
}

__global__ void __launch_bounds__(SCT) k_scan_partials(const uint32_t* __restrict__ counts, uint64_t q,
                                                       unsigned long long* __restrict__ partials,
                                                       uint32_t* __restrict__ ticket, uint64_t* __restrict__ total) {
  chain_wait();
  __shared__ unsigned long long wsum[SCT / 32];
  __shared__ uint32_t s_last;
  const uint64_t b0 = (uint64_t)blockIdx.x * SCB;
  unsigned long long s = 0ull;
#pragma unroll
  for (int k = 0; k < SCIPT; ++k) {
    const uint64_t i = b0 + (uint64_t)k * SCT + threadIdx.x;
    if (i < q) s += counts[i];
  }
  unsigned long long tot;
  block_excl_scan64(s, wsum, &tot);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = tot;
    s_last = 0u;
    if (ticket) {
      __threadfence();
      s_last = atomicAdd(ticket, 1u) == gridDim.x - 1u ? 1u : 0u;
    }
  }
  if (!ticket) return;
  __syncthreads();
  if (!s_last) return;
  // the last CTA scans the partial sums (k_scan_top's work)
  __threadfence();
  unsigned long long carry = 0ull;
  for (uint32_t c0 = 0; c0 < gridDim.x; c0 += SCT) {
    const uint32_t i = c0 + threadIdx.x;
    const unsigned long long v = i < gridDim.x ? __ldcg(partials + i) : 0ull;
    const unsigned long long ex = block_excl_scan64(v, wsum, &tot);
    if (i < gridDim.x) partials[i] = carry + ex;
    carry += tot;
  }
  if (threadIdx.x == 0) {
    partials[gridDim.x] = carry;
    if (total) *total = carry;
  }
}

__global__ void __launch_bounds__(1024) k_scan_top(unsigned long long* __restrict__ partials, uint64_t nb,
                                                   uint64_t* __restrict__ total) {
  chain_wait();
  __shared__ unsigned long long wsum[32];
  unsigned long long carry = 0ull;
  for (uint64_t c0 = 0; c0 < nb; c0 += blockDim.x) {
    const uint64_t i = c0 + threadIdx.x;
    const unsigned long long v = i < nb ? partials[i] : 0ull;
    unsigned long long tot;
    const unsigned long long ex = block_excl_scan64(v, wsum, &tot);
    if (i < nb) partials[i] = carry + ex;
    carry += tot;
  }
  if (threadIdx.x == 0) {
    partials[nb] = carry;
    if (total) *total = carry;
  }
}

__global__ void __launch_bounds__(SCT) k_scan_down(const uint32_t* __restrict__ counts, uint64_t q,
                                                   const unsigned long long* __restrict__ partials,
                                                   uint64_t* __restrict__ offsets, uint64_t nb) {
  chain_wait();
  __shared__ unsigned long long wsum[SCT / 32];
  const uint64_t b0 = (uint64_t)blockIdx.x * SCB;
  // each thread owns SCIPT consecutive counts
  const uint64_t t0 = b0 + (uint64_t)threadIdx.x * SCIPT;
  uint32_t v[SCIPT];
  unsigned long long s = 0ull;
#pragma unroll
  for (int k = 0; k < SCIPT; ++k) {
    v[k] = (t0 + k < q) ? counts[t0 + k] : 0u;
    s += v[k];
  }
  unsigned long long tot;
  unsigned long long run = partials[blockIdx.x] + block_excl_scan64(s, wsum, &tot);
#pragma unroll
  for (int k = 0; k < SCIPT; ++k) {
    if (t0 + k < q) offsets[t0 + k] = run;
    run += v[k];
  }
  if (blockIdx.x == nb - 1 && threadIdx.x == 0) offsets[q] = partials[nb];
}

cudaError_t launch_scan_counts(const uint32_t* counts, uint64_t q, uint64_t* offsets, unsigned long long* partials,
                               cudaStream_t stream, uint32_t* ticket, uint64_t* total) {
  if (q == 0) return cudaMemsetAsync(offsets, 0, sizeof(uint64_t), stream);
  const uint64_t nb = (q + SCB - 1) / SCB;
  // the partial sums of up to 4M counts are scanned by the last CTA that made one; more by 1,024 threads
  if (nb > 1024u) ticket = nullptr;
  FKD_CHAIN(k_scan_partials, dim3((unsigned)nb), dim3(SCT), 0, stream, counts, q, partials, ticket, total);
  if (!ticket) FKD_CHAIN(k_scan_top, dim3(1), dim3(1024), 0, stream, partials, nb, total);
  FKD_CHAIN(k_scan_down, dim3((unsigned)nb), dim3(SCT), 0, stream, counts, q, partials, offsets, nb);
  return cudaGetLastError();
}

// ------------------------------------------------------ ordered results
//
// search_in_the_box and its BFS / branchless variants emit the in-box nodes
// level by level in frontier order, and the frontier of every level is sorted
// by heap index (children are appended in order), so their output is the
// in-box set sorted by heap index.  For that order the write pass stores heap
// indices, this kernel sorts each box's slice and replaces the indices by ids.

constexpr int OT = 256;
constexpr int ORUN = 8192;  // slice length sorted in shared memory

__device__ void bitonic_smem(uint32_t* a, uint32_t m) {  // m a power of two
  for (uint32_t k = 2; k <= m; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
        const uint32_t p = i ^ j;
        if (p > i) {
          const uint32_t x = a[i], y = a[p];
          const bool up = (i & k) == 0;
          if ((x > y) == up) {
            a[i] = y;
            a[p] = x;
          }
        }
      }
      __syncthreads();
    }
  }
}

// Merges sorted runs a[0,la) and b[0,lb) into o (distinct keys), CTA-wide by
// merge-path partitioning.
__device__ void merge_cta(const uint32_t* a, uint32_t la, const uint32_t* b, uint32_t lb, uint32_t* o) {
  const uint32_t total = la + lb;
  const uint32_t per = (total + blockDim.x - 1) / blockDim.x;
  const uint32_t k0 = min(total, threadIdx.x * per), k1 = min(total, k0 + per);
  if (k0 >= k1) return;
  // find i in [max(0,k0-lb), min(k0,la)] with a[i-1] < b[k0-i] and b[k0-i-1] < a[i]
  uint32_t lo = k0 > lb ? k0 - lb : 0u, hi = k0 < la ? k0 : la;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (a[mid] < b[k0 - mid - 1u])
      lo = mid + 1u;
    else
      hi = mid;
  }
  uint32_t i = lo, j = k0 - lo;
  for (uint32_t k = k0; k < k1; ++k) {
    if (j >= lb || (i < la && a[i] < b[j]))
      o[k] = a[i++];
    else
      o[k] = b[j++];
  }
}

__global__ void __launch_bounds__(OT) k_order(Geom g, Table tab, const uint64_t* __restrict__ offsets, uint64_t q,
                                              uint32_t* __restrict__ out, uint64_t capacity,
                                              uint32_t* __restrict__ tmp, uint32_t* __restrict__ err,
                                              const uint32_t* __restrict__ list,
                                              const unsigned long long* __restrict__ nlist) {
  chain_wait();
  __shared__ uint32_t buf[ORUN];
  if (nlist) q = *nlist;
  for (uint64_t qx = blockIdx.x; qx < q; qx += gridDim.x) {
    const uint64_t qj = list ? list[qx] : qx;
    const uint64_t s0 = offsets[qj], s1 = offsets[qj + 1];
    if (s1 < s0 || s1 > capacity) {  // a caller's offsets need not be those of the boxes
      if (threadIdx.x == 0) atomicOr(err, ERRB_INTERNAL);
      continue;
    }
    const uint32_t len = (uint32_t)(s1 - s0);
    uint32_t* seg = out + s0;
    uint32_t* alt = tmp + s0;
    if (len > 1u) {
      // sort runs of ORUN in shared memory
      for (uint32_t r0 = 0; r0 < len; r0 += ORUN) {
        const uint32_t rl = min((uint32_t)ORUN, len - r0);
        uint32_t m = 1u;
        while (m < rl) m <<= 1;
        for (uint32_t i = threadIdx.x; i < m; i += OT) buf[i] = i < rl ? seg[r0 + i] : 0xffffffffu;
        __syncthreads();
        bitonic_smem(buf, m);
        for (uint32_t i = threadIdx.x; i < rl; i += OT) seg[r0 + i] = buf[i];
        __syncthreads();
      }
      // merge runs pairwise, ping-ponging between out and tmp
      uint32_t* src = seg;
      uint32_t* dst = alt;
      for (uint32_t w = ORUN; w < len; w <<= 1) {
        for (uint32_t a0 = 0; a0 < len; a0 += 2u * w) {
          const uint32_t la = min(w, len - a0);
          const uint32_t lb = (a0 + w < len) ? min(w, len - a0 - w) : 0u;
          merge_cta(src + a0, la, src + a0 + la, lb, dst + a0);
        }
        __syncthreads();
        uint32_t* t = src;
        src = dst;
        dst = t;
      }
      if (src != seg) {
        for (uint32_t i = threadIdx.x; i < len; i += OT) seg[i] = src[i];
        __syncthreads();
      }
    }
    for (uint32_t i = threadIdx.x; i < len; i += OT) {
      const uint32_t hidx = seg[i];
      if (hidx < g.n) {
        seg[i] = __ldg(tab.ids + hidx);
      } else {
        seg[i] = 0xffffffffu;
        atomicOr(err, ERRB_INTERNAL);
      }
    }
    __syncthreads();
  }
}

cudaError_t launch_order_results(const Geom& g, const Table& tab, const uint64_t* offsets, uint64_t q, uint32_t* out,
                                 uint64_t capacity, uint32_t* tmp, uint32_t* err, cudaStream_t stream, const uint32_t* list,
                                 const unsigned long long* nlist) {
  if (q == 0) return cudaSuccess;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const uint64_t blocks = q < (uint64_t)sms * 8 ? q : (uint64_t)sms * 8;
  FKD_CHAIN(k_order, dim3((unsigned)blocks), dim3(OT), 0, stream, g, tab, offsets, q, out, capacity, tmp, err, list, nlist);
  return cudaGetLastError();
}

// One box with a host round trip (a caller that searches box by box, as the
// reference's driver does from its TBB loop, main.cpp:351-359): a single warp
// walks the tree level by level like search_in_the_box (FKDTree_cpu.h:
// 123-169) -- the frontier of each depth in ascending heap order, the left
// child visited when min <= split value, the right when split value <= max --
// so the in-box nodes come out in ascending heap order, the reference's list,
// with no count pass, scan or sort.  out[0] = results (all of them, also past
// cap), out[1] = 1 when a depth's frontier outgrew ONE_FRONTIER (the caller
// then takes the general path), out[4 ..] = the first cap ids.
constexpr uint32_t ONE_FRONTIER = 2048;
template <int DIM>
__global__ void __launch_bounds__(32) k_one(Table tab, uint32_t n, OneBox bx, uint32_t* __restrict__ out,
                                            uint32_t cap) {
  __shared__ uint32_t fr[2][ONE_FRONTIER];
  const uint32_t lane = threadIdx.x;
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t nf = n ? 1u : 0u, total = 0u, cur = 0u;
  bool ovf = false;
  if (lane == 0) fr[0][0] = 0u;
  __syncwarp();
  for (uint32_t d = 0; nf > 0u && !ovf; ++d) {
    const uint32_t c = d % DIM;
    uint32_t nn = 0u;
    for (uint32_t b0 = 0; b0 < nf; b0 += 32u) {
      const uint32_t i = b0 + lane;
      const bool v = i < nf;
      const uint32_t node = v ? fr[cur][i] : 0u;
      uint4 p = make_uint4(0u, 0u, 0u, 0u);
      if (v) p = __ldg(tab.nodes + node);
      const float x[4] = {__uint_as_float(p.x), __uint_as_float(p.y), __uint_as_float(p.z), __uint_as_float(p.w)};
      bool in = v;
#pragma unroll
      for (int w = 0; w < DIM; ++w) in &= bx.lo[w] <= x[w] && x[w] <= bx.hi[w];
      const float sv = sel4(c, x[0], x[1], x[2], x[3]);
      const float lo = sel4(c, bx.lo[0], bx.lo[1], bx.lo[2], bx.lo[3]);
      const float hi = sel4(c, bx.hi[0], bx.hi[1], bx.hi[2], bx.hi[3]);
      const bool l = v && 2ull * node + 1ull < n && lo <= sv;
      const bool r = v && 2ull * node + 2ull < n && sv <= hi;
      const uint32_t bin = __ballot_sync(0xffffffffu, in);
      const uint32_t at = total + __popc(bin & lt);
      if (in && at < cap) out[4 + at] = __ldg(tab.ids + node);
      total += __popc(bin);
      // children in lane order, left before right: ascending heap order
      const uint32_t k = (l ? 1u : 0u) + (r ? 1u : 0u);
      uint32_t incl = k;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
      }
      const uint32_t q0 = nn + incl - k;
      const uint32_t add = __shfl_sync(0xffffffffu, incl, 31);
      if (nn + add > ONE_FRONTIER) {
        ovf = true;  // warp-uniform
        break;
      }
      uint32_t q = q0;
      if (l) fr[cur ^ 1u][q++] = 2u * node + 1u;
      if (r) fr[cur ^ 1u][q] = 2u * node + 2u;
      nn += add;
    }
    __syncwarp();
    cur ^= 1u;
    nf = nn;
  }
  if (lane == 0) {
    out[0] = total;
    out[1] = ovf ? 1u : 0u;
  }
}

cudaError_t launch_one(const Table& tab, uint32_t n, int dim, const OneBox& bx, uint32_t* out, uint32_t cap,
                       cudaStream_t stream) {
  switch (dim) {
    case 1: k_one<1><<<1, 32, 0, stream>>>(tab, n, bx, out, cap); break;
    case 2: k_one<2><<<1, 32, 0, stream>>>(tab, n, bx, out, cap); break;
    case 3: k_one<3><<<1, 32, 0, stream>>>(tab, n, bx, out, cap); break;
    case 4: k_one<4><<<1, 32, 0, stream>>>(tab, n, bx, out, cap); break;
    default: return cudaErrorInvalidValue;
  }
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace fkd
