// fkd_packet.cu -- count and digest search of neighbouring boxes together
// (sm_100a).
//
// Semantics: those of fkd_search.cu (FKDTree_cpu.h:123-169): a box visits the
// left child unless v < box.lo[c], the right child when v < box.lo[c] or
// box.lo[c] <= v <= box.hi[c], and counts exactly the points inside the closed box.
//
// Shape: boxes are put in the order of the tree cell their centre falls in
// and handed out 32 at a time (a packet); a warp walks the tree once for the
// packet, one box per lane.  The nodes, their subtrees' bounding boxes
// (fkd_tables.cu), sizes and digests are the same for all lanes (one broadcast
// load); each lane only tests its own bounds, and no lane ever diverges from
// the others.  A subtree whose bounding box lies outside a lane's box or
// inside it is done for that lane; it is entered while any lane's box cuts it.
// Subtrees of height BB_HEIGHT are not walked: their points, one per lane, are
// tested box by box (few boxes cut the bucket) or side by side (many).
//
// Sharing pays while several lanes cut the same buckets.  A packet whose
// buckets are cut by fewer than PKT_LANES lanes on average (boxes too far
// apart for their size) gives up and lists its boxes for the search that walks
// each box alone (fkd_walk.cu).
//
// Bound by issue slots (72% of them, 46% of the warps; 0.79 ms of the counts of 10^6
// boxes of 100 results of 10^6 points) and the latency of the node loads.
// Measured on one B200: the digest search of 1,024 events (33.6M boxes of half-width
// 0.01, a quarter of the events 4-D) 12.6 ms and 1.7 ms for the boxes' order and the
// packets left over, against 70.0 ms with two lanes per box.  Before the bounding
// boxes (cells of split values, a mask of the box's sides per lane, every side compared
// for every point): 27 ms.  fkd_capi.cu has the counts where a warp per box is faster.
#include <math.h>

#include "fkd_walk.cuh"

namespace fkd {
namespace {

constexpr int KT = 128;  // threads per CTA
constexpr int KW = KT / 32;
constexpr int PSTACK = 32;  // pending right children: at most one per depth, depths below 31
// (1 / 2 / 4 / 6 lanes: 23.5 / 23.8 / 24.0 / 24.5 ms of the 1,024 events; below 2 a packet
// of boxes all over a large tree never gives up)
constexpr uint32_t PKT_LANES = 2;
constexpr uint32_t PKT_TRIAL = 24;  // buckets before a packet may give up
// a bucket's cost box by box (per box) and side by side (per side), in the same unit:
// (2 / 4 / 8: 25.2 / 25.4 / 26.6 ms of the 1,024 events)
constexpr uint32_t PKT_TBOX = 1, PKT_TSIDE = 2;
// resident CTAs: 6 / 8 / 10 -> 25.4 / 25.5 / 27.0 ms of the 1,024 events
constexpr int PKT_MINB = 8;

template <int DIM, bool DIG>
__global__ void __launch_bounds__(KT, PKT_MINB) k_packet(SearchCtx sc, uint64_t nslots) {
  chain_wait();
  __shared__ float2 s_box[KW][DIM][32];                                   // (lo, hi) of every lane's box
  __shared__ __align__(16) float s_x[KW][DIM][32];                        // a bucket's points
  __shared__ __align__(16) unsigned long long s_dig[DIG ? KW : 1][32];    // their digests
  __shared__ __align__(16) unsigned long long s_sum[DIG ? KW : 1][8][16]; // sums of 4 points' subsets
  __shared__ uint2 s_stack[KW][PSTACK];                                   // pending (node, lanes that cut it)
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t cur_ev = 0u;  // batched: the event of the last packet (slots come in increasing order)
  for (;;) {
    uint32_t slot = 0u;
    if (lane == 0) slot = atomicAdd(sc.qcounter, 1u);
    slot = __shfl_sync(0xffffffffu, slot, 0);
    if ((uint64_t)slot >= nslots) break;
    Geom g = sc.g;
    Table tab = sc.tab;
    const float *blo = sc.boxes.lo, *bhi = sc.boxes.hi;
    uint64_t bstride = sc.boxes.stride, q0 = (uint64_t)slot * 32u, q1 = sc.boxes.q, qbase = 0u, qout = 0u;
    if (sc.evs) {
      // event e's packets take the slots from (qbase_e / 32) + e on
      while (cur_ev + 1u < sc.nev && (uint64_t)slot >= (sc.evs[cur_ev + 1u].qbase >> 5) + cur_ev + 1u) ++cur_ev;
      const EvDesc& ev = sc.evs[cur_ev];
      g = ev.g;
      tab.nodes += ev.base;
      tab.ids += ev.base;
      if (tab.ipts) tab.ipts += ev.base;
      tab.bb += 2u * bb_base(ev.base, cur_ev);
      if (DIM > 3) tab.dids += ev.base;
      if (DIG) tab.sdig += ev.base;
      blo += ev.qcbase;
      bhi += ev.qcbase;
      bstride = ev.nq;
      qbase = ev.qbase;
      qout = ev.qout;
      q0 = qbase + 32ull * (slot - (uint32_t)((qbase >> 5) + cur_ev));
      q1 = qbase + ev.nq;
    }
    if (q0 >= q1) continue;
    const bool have = q0 + lane < q1;
    uint64_t bj = 0u;  // this lane's box within its event
    BoxShape<DIM> box;
#pragma unroll
    for (int c = 0; c < DIM; ++c) box.lo[c] = box.hi[c] = 0.f;
    bool ok = have && g.n != 0u;
    if (have) {
      bj = sc.order[q0 + lane] - qbase;
      ok = box.load(blo, bhi, bstride, bj) && ok;
    }
    __syncwarp();  // the last packet's reads
#pragma unroll
    for (int c = 0; c < DIM; ++c) s_box[warp][c][lane] = make_float2(box.lo[c], box.hi[c]);
    __syncwarp();
    const float4* bb = tab.bb;
    uint32_t cnt = 0u;
    unsigned long long dig = 0ull;
    const uint32_t bdep = g.H > BB_HEIGHT ? g.H - BB_HEIGHT : 0u;
    uint32_t i = 0u, dep = 0u, sp = 0u;
    uint32_t nbuckets = 0u, ncut = 0u;
    bool loose = false;
    uint32_t R = __ballot_sync(0xffffffffu, ok);  // lanes whose box cuts subtree i
    if (R) {
      uint32_t out, cut;
      box.place(__ldg(bb), __ldg(bb + 1), out, cut);
      if (ok && !neg(cut)) {  // the whole tree
        cnt = g.n;
        if (DIG) dig = __ldg(tab.sdig);
      }
      R = __ballot_sync(0xffffffffu, ok && neg(cut) && !neg(out));
    }
    while (R) {
      if (dep == bdep) {
        // leaf bucket: the in-order range of subtree i, one point per lane
        const uint32_t t = i + 1u - (1u << dep);
        const uint32_t S = seg_start(g, dep, t), len = seg_len(g, dep, t);
        uint4 p = make_uint4(0u, 0u, 0u, 0u);
        if (lane < len) p = inorder_point(tab, g, S + lane);
        const float4 mn = __ldg(bb + 2u * i), mx = __ldg(bb + 2u * i + 1u);
        const float4 pf = as_float4(p);
        const bool mine = (R >> lane) & 1u;
        // the sides of this lane's box that leave points of the bucket out
        uint32_t nm = 0u;
#pragma unroll
        for (int c = DIM - 1; c >= 0; --c) {
          nm = __funnelshift_l(diff(box.hi[c], word(mx, c)), nm, 1);
          nm = __funnelshift_l(diff(word(mn, c), box.lo[c]), nm, 1);
        }
        if (!mine) nm = 0u;
        const uint32_t need = __reduce_or_sync(0xffffffffu, nm);
        uint32_t hits = 0u;  // bit 31 - k: the bucket's point k is inside this lane's box
        if (__popc(R) * PKT_TBOX <= __popc(need) * PKT_TSIDE) {
          // few boxes: box by box, every lane tests its own point
          for (uint32_t rest = R; rest != 0u; rest &= rest - 1u) {
            const uint32_t k = (uint32_t)__ffs(rest) - 1u;
            const uint32_t bm = __shfl_sync(0xffffffffu, nm, k);
            uint32_t o = 0u;
#pragma unroll
            for (int c = 0; c < DIM; ++c) {
              if ((bm >> (2 * c)) & 3u) {
                const float2 b = s_box[warp][c][k];
                o |= diff(word(pf, c), b.x) | diff(b.y, word(pf, c));
              }
            }
            const uint32_t bal = __ballot_sync(0xffffffffu, !neg(o));
            if (lane == k) hits = bal;
          }
          hits = __brev(hits);
        } else {
          // many boxes: side by side, every lane tests every point against its own box
#pragma unroll
          for (int c = 0; c < DIM; ++c)
            if ((need >> (2 * c)) & 3u) s_x[warp][c][lane] = word(pf, c);
          __syncwarp();
          uint32_t o = 0u;
#pragma unroll
          for (int c = 0; c < DIM; ++c) {
            const float4* xs = reinterpret_cast<const float4*>(s_x[warp][c]);
            if ((need >> (2 * c)) & 1u) {
              uint32_t h = 0u;
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                const float4 v = xs[k];
                h = __funnelshift_l(diff(v.x, box.lo[c]), h, 1);
                h = __funnelshift_l(diff(v.y, box.lo[c]), h, 1);
                h = __funnelshift_l(diff(v.z, box.lo[c]), h, 1);
                h = __funnelshift_l(diff(v.w, box.lo[c]), h, 1);
              }
              o |= h;
            }
            if ((need >> (2 * c)) & 2u) {
              uint32_t h = 0u;
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                const float4 v = xs[k];
                h = __funnelshift_l(diff(box.hi[c], v.x), h, 1);
                h = __funnelshift_l(diff(box.hi[c], v.y), h, 1);
                h = __funnelshift_l(diff(box.hi[c], v.z), h, 1);
                h = __funnelshift_l(diff(box.hi[c], v.w), h, 1);
              }
              o |= h;
            }
          }
          __syncwarp();
          hits = mine ? ~o : 0u;
        }
        hits &= len < 32u ? ~(0xffffffffu >> len) : 0xffffffffu;
        cnt += __popc(hits);
        if (DIG && __any_sync(0xffffffffu, hits != 0u)) {
          // the sum over a lane's hits from tables of the sums of all subsets of 4 points
          const uint32_t id = DIM <= 3 ? p.w : (lane < len ? __ldg(tab.dids + S + lane) : 0u);
          s_dig[warp][lane] = mix64(id);
          __syncwarp();
          {
            const uint32_t q = lane >> 2, r = lane & 3u;
            const unsigned long long u = ((r & 2u) ? s_dig[warp][4u * q] : 0ull) +
                                         ((r & 1u) ? s_dig[warp][4u * q + 1u] : 0ull);
            const unsigned long long a = s_dig[warp][4u * q + 3u], b = s_dig[warp][4u * q + 2u];
            s_sum[warp][q][4u * r] = u;
            s_sum[warp][q][4u * r + 1u] = u + a;
            s_sum[warp][q][4u * r + 2u] = u + b;
            s_sum[warp][q][4u * r + 3u] = u + a + b;
          }
          __syncwarp();
#pragma unroll
          for (int q = 0; q < 8; ++q) dig += s_sum[warp][q][(hits >> (28 - 4 * q)) & 15u];
          __syncwarp();
        }
        ++nbuckets;
        ncut += (uint32_t)__popc(R);
        if (nbuckets >= PKT_TRIAL && ncut < PKT_LANES * nbuckets) {
          loose = true;
          break;
        }
      } else {
        // an inner node: its own point, then both children's bounding boxes
        const uint32_t l = 2u * i + 1u;
        const uint4 nd = __ldg(tab.nodes + i);
        const float4 mnL = __ldg(bb + 2u * l), mxL = __ldg(bb + 2u * l + 1u);
        const float4 mnR = __ldg(bb + 2u * l + 2u), mxR = __ldg(bb + 2u * l + 3u);
        const bool mine = (R >> lane) & 1u;
        const bool emit = mine && !neg(box.outside(as_float4(nd)));
        uint32_t outL, cutL, outR, cutR;
        box.place(mnL, mxL, outL, cutL);
        box.place(mnR, mxR, outR, cutR);
        const uint32_t RL = __ballot_sync(0xffffffffu, mine && neg(cutL) && !neg(outL));
        const uint32_t RR = __ballot_sync(0xffffffffu, mine && neg(cutR) && !neg(outR));
        const bool inL = mine && !neg(cutL), inR = mine && !neg(cutR);
        cnt += emit ? 1u : 0u;
        if (DIG && __any_sync(0xffffffffu, emit)) {
          const unsigned long long x = mix64(DIM <= 3 ? nd.w : __ldg(tab.ids + i));
          if (emit) dig += x;
        }
        if (__any_sync(0xffffffffu, inL || inR)) {
          const uint32_t t = l + 1u - (1u << (dep + 1u));
          const uint32_t szL = seg_len(g, dep + 1u, t), szR = seg_len(g, dep + 1u, t + 1u);
          if (inL) cnt += szL;
          if (inR) cnt += szR;
          if (DIG) {
            const unsigned long long xL = __ldg(tab.sdig + l), xR = __ldg(tab.sdig + l + 1u);
            if (inL) dig += xL;
            if (inR) dig += xR;
          }
        }
        if (RL) {
          if (RR) {
            if (lane == 0) s_stack[warp][sp] = make_uint2(l + 1u, RR);
            ++sp;
          }
          i = l;
          R = RL;
          ++dep;
          continue;
        }
        if (RR) {
          i = l + 1u;
          R = RR;
          ++dep;
          continue;
        }
      }
      if (sp == 0u) break;
      --sp;
      __syncwarp();
      const uint2 top = s_stack[warp][sp];
      i = top.x;
      R = top.y;
      dep = floor_log2_u32(i + 1u);
    }
    __syncwarp();
    if (!loose) {
      if (have) {
        sc.counts[qout + bj] = cnt;
        if (DIG) sc.digests[qout + bj] = dig;
      }
    } else {
      // the boxes of a packet that gave up, for the search that walks each box alone
      const uint32_t nh = (uint32_t)__popc(__ballot_sync(0xffffffffu, have));
      unsigned long long at = 0ull;
      if (lane == 0) at = atomicAdd(sc.loose_ctr, (unsigned long long)nh);
      at = __shfl_sync(0xffffffffu, at, 0);
      if (have) sc.loose[at + lane] = (uint32_t)(qbase + bj);
    }
  }
}

template <int DIM, bool DIG>
cudaError_t run_packet(SearchCtx& sc) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_packet<DIM, DIG>, KT, 0);
  if (e != cudaSuccess) return e;
  if (per < 1) per = 1;
  const uint64_t nslots = (sc.boxes.q + 31u) / 32u + (sc.evs ? sc.nev + 1u : 0u);
  uint64_t blocks = (uint64_t)sms * per;
  const uint64_t need = (nslots + KW - 1) / KW;
  if (blocks > need) blocks = need;
  if (!sc.qready) e = cudaMemsetAsync(sc.loose_ctr, 0, sizeof(unsigned long long), sc.stream);
  SearchCtx pk = sc;
  if (e == cudaSuccess) e = work_counter(pk, QC_PACKET);
  if (e != cudaSuccess) return e;
  FKD_CHAIN(k_packet<DIM, DIG>, dim3((unsigned)blocks), dim3(KT), 0, sc.stream, pk, nslots);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  SearchCtx left = sc;
  left.order = sc.loose;
  left.qdev = sc.loose_ctr;
  return launch_walk(left, DIM, DIG ? SEARCH_DIGEST : SEARCH_COUNT);
}

__device__ __forceinline__ float pick4(uint32_t c, float a, float b, float d, float e) {
  return c == 0 ? a : (c == 1 ? b : (c == 2 ? d : e));
}

// -------------------------------------------- order of a batch's boxes
//
// The boxes of event e in the order of the cell of its tree their centre
// falls in: D = H - 5 levels, cells of 32 to 63 points.  The cells of all
// events are numbered through -- event e's from (base_e / 32) + e on, which
// leaves at least 2^D of them -- so that a counting sort by cell keeps every
// event's boxes in its own range [qbase, qbase + nq).
constexpr uint32_t CELL_BITS = 5;

__device__ __forceinline__ uint32_t event_of(const EvDesc* __restrict__ evs, uint32_t nev, uint64_t j) {
  uint32_t a = 0u, b = nev;  // evs[a].qbase <= j < evs[b].qbase
  while (b - a > 1u) {
    const uint32_t mid = (a + b) >> 1;
    if (evs[mid].qbase <= j)
      a = mid;
    else
      b = mid;
  }
  return a;
}

template <int DIM>
__global__ void k_event_keys(const EvDesc* __restrict__ evs, uint32_t nev, const uint4* __restrict__ nodes,
                             const float* __restrict__ lo, const float* __restrict__ hi, uint64_t q,
                             uint32_t* __restrict__ keys, uint32_t* __restrict__ hist) {
  chain_wait();
  const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= q) return;
  const uint32_t e = event_of(evs, nev, j);
  const EvDesc& ev = evs[e];
  const uint64_t bj = j - ev.qbase;
  float ctr[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int c = 0; c < DIM; ++c)
    ctr[c] = 0.5f * (lo[ev.qcbase + (uint64_t)c * ev.nq + bj] + hi[ev.qcbase + (uint64_t)c * ev.nq + bj]);
  const uint4* nd0 = nodes + ev.base;
  const uint32_t D = ev.g.H > CELL_BITS ? ev.g.H - CELL_BITS : 0u;
  uint32_t i = 0u;
  for (uint32_t dep = 0; dep < D; ++dep) {  // every node above depth D <= H - 1 exists
    const uint32_t c = dep % (uint32_t)DIM;
    const uint4 nd = __ldg(nd0 + i);
    const float v = pick4(c, __uint_as_float(nd.x), __uint_as_float(nd.y), __uint_as_float(nd.z),
                          __uint_as_float(nd.w));
    i = 2u * i + 1u + (pick4(c, ctr[0], ctr[1], ctr[2], ctr[3]) < v ? 0u : 1u);
  }
  const uint32_t key = (ev.base >> CELL_BITS) + e + (i + 1u - (1u << D));
  keys[j] = key;
  atomicAdd(&hist[key], 1u);
}

__global__ void k_event_scatter(uint64_t q, const uint32_t* __restrict__ keys, unsigned long long* __restrict__ offs,
                                uint32_t* __restrict__ order) {
  chain_wait();
  const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= q) return;
  const unsigned long long pos = atomicAdd(&offs[keys[j]], 1ull);
  if (pos < q) order[pos] = (uint32_t)j;
}

struct OrderLayout {
  size_t keys, order, hist, offs, partials, words;
};
OrderLayout order_layout(uint64_t npts, uint32_t nev, uint64_t q) {
  const uint64_t cells = (npts >> CELL_BITS) + nev + 1u;
  auto up4 = [](size_t w) { return (w + 3u) & ~(size_t)3u; };
  OrderLayout L;
  L.keys = 0;
  L.order = up4(q);
  L.hist = L.order + up4(q);
  L.offs = L.hist + up4(cells);
  L.partials = L.offs + up4(2u * (cells + 1u));
  L.words = L.partials + up4(2u * scan_partials_words(cells));
  return L;
}

}  // namespace

size_t event_order_words(uint64_t npts, uint32_t nev, uint64_t q) { return order_layout(npts, nev, q).words; }

cudaError_t launch_event_order(const EvDesc* evs, uint32_t nev, uint64_t npts, const Table& tab, const Boxes& b, int dim,
                               uint32_t* scratch, uint32_t** order_out, cudaStream_t stream) {
  *order_out = nullptr;
  if (b.q == 0) return cudaSuccess;
  const OrderLayout L = order_layout(npts, nev, b.q);
  const uint64_t cells = (npts >> CELL_BITS) + nev + 1u;
  uint32_t* keys = scratch + L.keys;
  uint32_t* hist = scratch + L.hist;
  unsigned long long* offs = (unsigned long long*)(scratch + L.offs);
  cudaError_t e = cudaMemsetAsync(hist, 0, cells * sizeof(uint32_t), stream);
  if (e != cudaSuccess) return e;
  const unsigned blocks = (unsigned)((b.q + 255u) / 256u);
  switch (dim) {
    case 1: FKD_CHAIN(k_event_keys<1>, dim3(blocks), dim3(256), 0, stream, evs, nev, tab.nodes, b.lo, b.hi, b.q, keys, hist); break;
    case 2: FKD_CHAIN(k_event_keys<2>, dim3(blocks), dim3(256), 0, stream, evs, nev, tab.nodes, b.lo, b.hi, b.q, keys, hist); break;
    case 3: FKD_CHAIN(k_event_keys<3>, dim3(blocks), dim3(256), 0, stream, evs, nev, tab.nodes, b.lo, b.hi, b.q, keys, hist); break;
    default: FKD_CHAIN(k_event_keys<4>, dim3(blocks), dim3(256), 0, stream, evs, nev, tab.nodes, b.lo, b.hi, b.q, keys, hist); break;
  }
  e = launch_scan_counts(hist, cells, (uint64_t*)offs, (unsigned long long*)(scratch + L.partials), stream);
  if (e != cudaSuccess) return e;
  FKD_CHAIN(k_event_scatter, dim3(blocks), dim3(256), 0, stream, b.q, keys, offs, scratch + L.order);
  *order_out = scratch + L.order;
  return cudaGetLastError();
}

cudaError_t launch_packets(SearchCtx& sc, int dim, int mode) {
  const bool dig = mode == SEARCH_DIGEST;
  switch (dim) {
    case 1: return dig ? run_packet<1, true>(sc) : run_packet<1, false>(sc);
    case 2: return dig ? run_packet<2, true>(sc) : run_packet<2, false>(sc);
    case 3: return dig ? run_packet<3, true>(sc) : run_packet<3, false>(sc);
    case 4: return dig ? run_packet<4, true>(sc) : run_packet<4, false>(sc);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fkd
