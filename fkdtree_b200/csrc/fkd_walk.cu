// fkd_walk.cu -- searches that walk the tree for one box (or ball) with a
// warp, 32 subtrees at a time (sm_100a).
//
// Semantics: those of fkd_search.cu (FKDTree_cpu.h:123-169): exactly the
// points inside the closed box; the ordered list is the reference's (level by
// level, ascending heap index).
//
// k_walk.  The warp enters a node by testing, one per lane, the bounding
// boxes of all its descendants WIDE levels below (neighbours in heap order: one
// coalesced load) and the points of the nodes in between.  Descendants inside
// the box are counted in closed form, those outside dropped, those the box
// cuts entered in turn, from left to right; at the bottom a descendant is a
// leaf bucket (height BB_HEIGHT, at most 31 points) and its points are tested
// one per lane.  A box on a tree of 16M points thus waits for 4 to 5
// dependent loads per path, not for 24.
//
// A bucket that reaches into the tree's last level holds 16 to 31 points, the
// others 15: of 2^24 points, a tree whose last level is all but empty, nearly
// all.  Two of those share a step, half a warp each.  Counts of 131,072 boxes on
// 2^24 uniform points, us, one by one / in pairs (a walk of single nodes with
// buckets of 31): 1,000 results 985 / 756 (889), 10,000 results 3,580 / 2,588
// (2,800), in 4-D 7,190 / 5,103 (5,545); digests of 10,000 5,305 / 3,502 (4,257);
// on 10^6 points, where nearly all buckets are full, 2,132 / 2,184 (2,859).
//
// Because the walk goes from left to right it meets the box's points in in-order
// position, and records them as a list of entries in that order: runs of
// consecutive positions (contained subtrees with the nodes between them) and
// windows (the hits of a bucket as a bit mask; where the list's order does not
// matter, their ids).  The in-order position of a point tells its depth: with v the position counted from 1 in the perfect
// tree it belongs to, depth = H - (number of trailing zeros of v).  The
// reference's order -- by depth, then from left to right -- is therefore a
// stable distribution of the list over the tree's depths: the walk counts the
// results per depth as it goes (closed form for contained subtrees, popcounts
// for windows), and k_emit copies every window, and every 32 positions of a
// run, to the cursors of their depths.  No sort, and the ids are read and
// written nearly in sequence.
//
// Both are bound by issue slots and the latency of their dependent loads (walk 69%
// of the issue slots and 47% of the warps -- 64 registers --, emission 56% and 56%).
// Measured on one B200, 2^24 clustered points: 65,536 boxes (2.76e8 ids, ordered)
// walk 1.12 + emit 1.04 ms, against 1.50 for a recording walk of single nodes, 0.85
// for its copy and 27.4 for the sort by heap index; 1,048,576 boxes (4.43e9 ids)
// unordered 12.1 + 8.5 ms (21.4 + 9.3), ordered 15.3 + 13.9; 100,000 boxes of 1.8
// results 0.12 + 0.04 ms against 0.20 + 0.06 + 0.19; 100,000 balls of 137 points on
// 10^6 0.30 + 0.13 ms against 0.30 + 0.35 for walks node by node and 1.22 for the
// sort; counts of 1,048,576 boxes of 4,200 results 5.2 ms against 8.5.  k_emit
// counting the depths itself, and windows at 32-aligned positions for runs too:
// 1.76 ms of the 65,536 lists.
#include <math.h>

#include <initializer_list>

#include "fkd_walk.cuh"

namespace fkd {
namespace {

constexpr int WT = 128;  // threads per CTA
constexpr uint32_t WIDE = 5;        // levels per step: 32 descendants, one per lane
constexpr int WLEV = 7;             // steps per path (depths below 31)
constexpr uint32_t EBUF = 128;      // entries buffered per warp
constexpr uint32_t EBLK = 256;     // pool entries a warp reserves at a time
constexpr uint32_t E_WINDOW = 0x80000000u, E_UPPER = 0x40000000u, E_LINK = 0xffffffffu, E_IDS = 0xfffffffeu;
constexpr uint32_t NO_RECORD = 0xffffffffu;  // first entry of a box whose record did not fit (no entry is numbered so)
constexpr uint32_t NONE = 32u;      // no descendant, no step
// Descendants to enter from which a step is divided.  Counts, us, from 16 with eight warps, 8 with
// four, 4 with two / from 12 / from 20: 1,000 boxes of 50,000 results of 2^24 points 332 / 247 / 269, in
// 4-D 683 / 499 / 510, of 10,000 of 10^6 90 / 77 / 85; 3,000 of 1,000 in 4-D 123 / 139 / 147.
constexpr int SHARE = 12;
constexpr uint32_t IBUF = 160;      // ids buffered per warp (a bucket adds at most 31)
// resident CTAs: 6 / 8 / 10 -> 2.71 / 2.63 / 2.69 ms of the counts of 131,072 boxes of 10,000 results
constexpr int WALK_MINB = 8;
enum { WALK_COUNT = 0, WALK_DIGEST = 1, WALK_RECORD = 2, WALK_RECORD_ORDERED = 3 };

// bits b of a 32-bit window (b = 0 apart) with c trailing zeros; none for c > 4
__device__ __forceinline__ uint32_t window_class(uint32_t c) {
  return c == 0u   ? 0xaaaaaaaau
         : c == 1u ? 0x44444444u
         : c == 2u ? 0x10101010u
         : c == 3u ? 0x01000100u
                   : (c == 4u ? 0x00010000u : 0u);
}

constexpr int walk_threads(int split) { return split ? 32 * split : WT; }

// SPLIT (counts and digests): a CTA of so many warps per box.  All of them take the
// same steps until one has SHARE descendants to enter, or is the last: those they
// divide among themselves, and each enters its own alone.
//
// PAIRS: whether buckets without points of the last level are tested in pairs.
template <int DIM, int KIND, template <int> class SHAPE, int SPLIT = 0, bool PAIRS = true>
__global__ void __launch_bounds__(walk_threads(SPLIT), WALK_MINB * WT / walk_threads(SPLIT)) k_walk(SearchCtx sc, uint32_t grab) {
  chain_wait();
  constexpr bool ORD = KIND == WALK_RECORD_ORDERED, REC = KIND == WALK_RECORD || ORD, DIG = KIND == WALK_DIGEST;
  constexpr int WW = SPLIT ? SPLIT : WT / 32;  // warps
  __shared__ uint4 s_lv[WW][WLEV];  // pending steps: (first descendant, those still to enter, contained, nodes inside)
  __shared__ uint32_t s_from[WW][WLEV];
  __shared__ uint2 s_ent[REC ? WW : 1][EBUF];
  __shared__ __align__(8) uint32_t s_ids[KIND == WALK_RECORD ? WW : 1][IBUF];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const uint64_t nq = sc.qdev ? *sc.qdev : sc.boxes.q;
  uint32_t cur_ev = 0u;
  uint32_t e_cur = 0u, e_end = 0u;  // this warp's block of the entry pool
  uint32_t qi = 0u, qend = 0u;      // this warp's boxes
  static_assert(!SPLIT || !REC, "a list is recorded by one warp");
  __shared__ uint32_t s_acc[SPLIT ? SPLIT : 1];
  __shared__ unsigned long long s_dig[SPLIT && DIG ? SPLIT : 1];
  for (;; ++qi) {
    if (SPLIT) {
      if (qend) break;
      qi = blockIdx.x;
      qend = ~0u;
    } else if (qi == qend) {
      if (lane == 0) qi = atomicAdd(sc.qcounter, grab);
      qi = __shfl_sync(0xffffffffu, qi, 0);
      qend = qi + grab;
    }
    if ((uint64_t)qi >= nq) break;
    uint32_t qj = sc.order ? sc.order[qi] : qi;
    if (sc.evsel) qj = select_box(sc, qi, cur_ev);
    uint64_t oj = qj, bj = qj, bstride = sc.boxes.stride;
    Geom g = sc.g;
    Table tab = sc.tab;
    const float *blo = sc.boxes.lo, *bhi = sc.boxes.hi;
    if (sc.evs) {
      while (cur_ev > 0u && (uint64_t)qj < sc.evs[cur_ev].qbase) --cur_ev;  // (a list of loose boxes)
      while (cur_ev + 1u < sc.nev && (uint64_t)qj >= sc.evs[cur_ev + 1u].qbase) ++cur_ev;
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
      bj = qj - ev.qbase;
      oj = ev.qout + bj;
    }
    const float4* bb = tab.bb;
    const uint32_t bdep = g.H > BB_HEIGHT ? g.H - BB_HEIGHT : 0u;
    const uint32_t pair0 = PAIRS ? (g.M + 15u) >> BB_HEIGHT : ~0u;  // buckets from here on hold no point of the last level
    SHAPE<DIM> box;
    const bool ok = box.load(blo, bhi, bstride, bj) && g.n != 0u;
    uint32_t acc = 0u;  // this lane's share of the count; ordered: the results at depth `lane`
    unsigned long long dig = 0ull;
    // the bits of a window at depth `lane` (H - its class, one less past 2M)
    const uint32_t dpat = ORD ? window_class(g.H - lane) : 0u, dpatU = ORD ? window_class(g.H - 1u - lane) : 0u;
    // recording
    uint32_t nbuf = 0u, etotal = 0u, efirst = e_cur;
    bool recfail = false;
    // room for k entries in a row; one entry of a block is left for the link to the next
    auto room = [&](uint32_t k) {
      if (!recfail && e_cur + k + 1u > e_end) {
        const uint32_t want = EBLK > k + 1u ? EBLK : k + 1u;
        unsigned long long b = 0ull;
        if (lane == 0) b = atomicAdd(sc.ent_ctr, (unsigned long long)want);
        b = __shfl_sync(0xffffffffu, b, 0);
        if (b + want <= sc.ent_cap) {
          if (etotal) {
            if (lane == 0) sc.ents[e_cur] = make_uint2(E_LINK, (uint32_t)b);
          } else {
            efirst = (uint32_t)b;
          }
          e_cur = (uint32_t)b;
          e_end = (uint32_t)(b + want);
        } else {
          recfail = true;
          e_cur = e_end = 0u;
        }
      } else if (recfail && lane == 0) {
        atomicAdd(sc.ent_ctr, (unsigned long long)k);  // the next call's pool is sized by the demand
      }
    };
    auto flush = [&]() {  // buffered entries to the pool
      if (nbuf == 0u) return;
      __syncwarp();
      room(nbuf);
      if (!recfail) {
        for (uint32_t e = lane; e < nbuf; e += 32u) sc.ents[e_cur + e] = s_ent[warp][e];
        e_cur += nbuf;
        etotal += nbuf;
      }
      nbuf = 0u;
      __syncwarp();
    };
    uint32_t nids = 0u;  // not ordered: the buckets' hits are recorded by their ids
    auto flush_ids = [&]() {  // ids to the pool, two per entry, under a heading entry
      if (nids == 0u) return;
      __syncwarp();
      const uint32_t k = (nids + 1u) >> 1;
      room(k + 1u);
      if (!recfail) {
        if (lane == 0) sc.ents[e_cur] = make_uint2(E_IDS, nids);
        for (uint32_t e = lane; e < k; e += 32u)
          sc.ents[e_cur + 1u + e] = reinterpret_cast<const uint2*>(s_ids[warp])[e];
        e_cur += k + 1u;
        etotal += k + 1u;
      }
      nids = 0u;
      __syncwarp();
    };

    // This lane's point of a leaf bucket, p at in-order position pos; the lanes whose point is inside.
    auto scan = [&](bool have, uint32_t pos, const uint4& p) {
      const bool in = have && !neg(box.outside(as_float4(p)));
      if (!ORD) acc += in ? 1u : 0u;
      if (DIG && in) dig += mix64(DIM <= 3 ? p.w : __ldg(tab.dids + pos));
      if (!REC) return 0u;
      const uint32_t bal = __ballot_sync(0xffffffffu, in);
      if (KIND == WALK_RECORD) {
        if (in) s_ids[warp][nids + __popc(bal & lt)] = DIM <= 3 ? p.w : __ldg(tab.dids + pos);
        nids += __popc(bal);
        if (nids > IBUF - 32u) flush_ids();
      }
      return bal;
    };
    // Ordered lists: the windows of the bucket at [S, S + len), bit k of bal its k-th point.
    auto windows = [&](uint32_t S, uint32_t len, uint32_t bal) {
      // v = position + 1 up to 2M (the part of the tree with its last level), position - M + 1 past it
      const uint32_t c1 = S >= 2u * g.M ? 0u : min(len, 2u * g.M - S);
      const uint32_t m1 = c1 < 32u ? bal & ((1u << c1) - 1u) : bal;
      const uint32_t m2 = c1 < 32u ? bal >> c1 : 0u;
      if (m1) {
        const uint32_t v0 = S + 1u, m = m1 << (v0 & 31u);
        if (lane == 0) s_ent[warp][nbuf] = make_uint2(E_WINDOW | (v0 >> 5), m);
        acc += __popc(m & dpat);
        ++nbuf;
      }
      if (m2) {
        const uint32_t v0 = S + c1 - g.M + 1u, m = m2 << (v0 & 31u);
        if (lane == 0) s_ent[warp][nbuf] = make_uint2(E_WINDOW | E_UPPER | (v0 >> 5), m);
        acc += __popc(m & dpatU);
        ++nbuf;
      }
      if (nbuf > EBUF - 34u) flush();
    };

    // the wide step that holds the node all results lie below (the root's, if it is not known)
    const uint32_t w0 = bdep ? (bdep - 1u) % WIDE + 1u : 0u;  // levels of the first step; the others take WIDE
    uint32_t lv0 = 0u, t00 = 0u;
    if (sc.start && bdep) {
      const uint32_t r = sc.start[qj];
      const uint32_t rd = floor_log2_u32(r + 1u);
      if (rd >= w0) {
        const uint32_t steps = min((rd - w0) / WIDE, (bdep - w0) / WIDE - (bdep > w0 ? 1u : 0u));
        const uint32_t d = w0 + WIDE * steps;  // its depth, above the buckets
        if (d < bdep) {
          lv0 = steps + 1u;
          t00 = ((r + 1u) >> (rd - d)) - (1u << d);
        }
      }
    }
    uint32_t rootcut = 0u;
    if (ok && lv0 != 0u) {
      rootcut = 0x80000000u;  // its step decides
    } else if (ok) {
      uint32_t out;
      box.place(__ldg(bb), __ldg(bb + 1), out, rootcut);
      if (!neg(rootcut)) {  // the whole tree
        if (lane == 0) {
          acc = g.n;
          if (DIG) dig = __ldg(tab.sdig);
          if (REC) s_ent[warp][0] = make_uint2(0u, g.n);
        }
        if (REC) nbuf = 1u;
        if (ORD) acc = lane < g.H ? 1u << lane : (lane == g.H ? g.M : 0u);
      }
      if (neg(out)) rootcut = 0u;
    }
    if (neg(rootcut) && bdep == 0u) {
      const uint4 p = lane < g.n ? inorder_point(tab, g, lane) : make_uint4(0u, 0u, 0u, 0u);
      const uint32_t bal = scan(lane < g.n, lane, p);
      if (ORD) windows(0u, g.n, bal);
    } else if (neg(rootcut)) {
      uint32_t lv = lv0, t0 = t00 << (lv0 ? WIDE : 0u), from = 0u;
      uint32_t X = 0u, C = 0u, P = 0u;     // descendants to enter, contained; nodes in between inside the box
      uint32_t lvs = NONE;                 // the step whose descendants the warps have divided
      uint32_t SM = 0u, rs = 0u, rl = 0u;  // recording: lanes that start a run, this lane's run
      // the runs of consecutive positions of a step: descendant k sits at [S_k, S_k + len), the node
      // after it at S_{k+1} - 1
      auto runs = [&](uint32_t dc) {
        const uint32_t c = (C >> lane) & 1u, q = (P >> lane) & 1u;
        const bool cs = c && !(lane && ((P >> (lane - 1u)) & 1u)), ps = q && !c;
        SM = __ballot_sync(0xffffffffu, cs || ps);
        if (SM == 0u) return;
        rs = cs ? seg_start(g, dc, t0 + lane) : seg_start(g, dc, t0 + lane + 1u) - 1u;
        const uint32_t k0 = cs ? lane : lane + 1u;
        const uint32_t k = k0 + (uint32_t)__ffs((~(C & P)) >> (k0 & 31u)) - 1u;  // (node 31 is not of this step: P < 2^31)
        rl = (((C >> (k & 31u)) & 1u) ? seg_start(g, dc, t0 + k + 1u) - 1u : seg_start(g, dc, t0 + k)) - rs;
      };
      auto put_runs = [&](uint32_t sel) {
        if (sel == 0u) return;
        if ((sel >> lane) & 1u) s_ent[warp][nbuf + __popc(sel & lt)] = make_uint2(rs, rl);
        nbuf += __popc(sel);
        if (nbuf > EBUF - 34u) flush();
      };
      auto enter = [&](uint32_t dc, uint32_t w) {
        const uint32_t t = t0 + lane, nch = 1u << w;
        const bool have = lane < nch, havep = lane + 1u < nch;
        const uint32_t r = (1u << dc) - 1u + t;
        const uint32_t z = (uint32_t)__ffs(lane + 1u);  // the node after descendant k: z levels up
        const uint32_t hp = (1u << (dc - (havep ? z : 0u))) - 1u + (t >> z);
        float4 mn = make_float4(0.f, 0.f, 0.f, 0.f), mx = mn;
        uint4 nd = make_uint4(0u, 0u, 0u, 0u);
        if (have) {
          mn = __ldg(bb + 2u * r);
          mx = __ldg(bb + 2u * r + 1u);
        }
        if (havep) nd = __ldg(tab.nodes + hp);
        uint32_t out, cut;
        box.place(mn, mx, out, cut);
        const bool all = SPLIT && lv <= lvs;      // a step that all warps take:
        const bool mine = !all || warp == 0u;     // what they find counts once
        const bool in = mine && havep && !neg(box.outside(as_float4(nd)));
        const bool cont = mine && have && !neg(cut);
        X = __ballot_sync(0xffffffffu, have && neg(cut) && !neg(out));
        if (all && (dc == bdep || __popc(X) >= SHARE)) {
          X = __ballot_sync(0xffffffffu, ((X >> lane) & 1u) && (__popc(X & lt) + t0) % (SPLIT ? SPLIT : 1) == warp);
          lvs = lv;
        }
        if (KIND == WALK_COUNT && DIM == 4 && dc == bdep && tab.ipts && ((X >> lane) & 1u)) {
          // a 4-D box cuts many buckets of a step, often not in L2: all on their way at once (8,000 boxes
          // of 10,000 results of 2^24 points 649 -> 597 us; other kinds and dimensions lose: 2.63 -> 2.83 ms
          // of 131,072 boxes in 3-D, 8.06 -> 8.41 of digests in 4-D)
          const uint4* q = tab.ipts + seg_start(g, bdep, t);
          const uint32_t len = seg_len(g, bdep, t);
#pragma unroll
          for (uint32_t i = 0u; i < 32u; i += 8u)
            if (i < len) asm volatile("prefetch.global.L2 [%0];" ::"l"(q + i));
        }
        if (!ORD) {
          if (cont) acc += seg_len(g, dc, t);
          acc += in ? 1u : 0u;
        }
        if (DIG) {
          if (cont) dig += __ldg(tab.sdig + r);
          if (in) dig += mix64(DIM <= 3 ? nd.w : __ldg(tab.ids + hp));
        }
        if (REC) {
          C = __ballot_sync(0xffffffffu, cont);
          P = __ballot_sync(0xffffffffu, in);
          if (ORD) {
            // a contained descendant has 2^k nodes k levels below it, down to the last but one level
            const uint32_t full = (1u << (g.H - dc)) - 1u;
            if (C) {
              const uint32_t last = __reduce_add_sync(0xffffffffu, cont ? seg_len(g, dc, t) - full : 0u);
              if (lane >= dc && lane < g.H) acc += (uint32_t)__popc(C) << (lane - dc);
              if (lane == g.H) acc += last;
            }
            if (P) acc += __popc(P & (window_class(dc - 1u - lane) >> 1));  // the node after descendant k: see z
          }
          runs(dc);
        }
        from = 0u;
      };
      enter(w0 + WIDE * lv, lv ? WIDE : w0);
      for (;;) {
        const uint32_t dc = w0 + WIDE * lv;
        if (dc == bdep) {
          // the cut leaf buckets, the next one's points loaded before this one's are tested: those that
          // hold points of the last level one by one, the others in pairs, half a warp each
          auto runs_to = [&](uint32_t kx) {
            put_runs(SM & ((1u << kx) - 1u) & ~((1u << from) - 1u));
            from = kx;
          };
          uint32_t XS = 0u;
          if (PAIRS) {
            const uint32_t nlong = pair0 > t0 ? pair0 - t0 : 0u;
            XS = nlong < 32u ? X >> nlong << nlong : 0u;
            X ^= XS;
          }
          uint32_t k = 0u, len = 0u, S = 0u;
          uint4 p = make_uint4(0u, 0u, 0u, 0u);
          auto fetch = [&]() {
            k = (uint32_t)__ffs(X) - 1u;
            S = PAIRS ? 32u * (t0 + k) : seg_start(g, bdep, t0 + k);
            len = PAIRS ? min(31u, 15u + g.M - 16u * (t0 + k)) : seg_len(g, bdep, t0 + k);
            if (lane < len) p = inorder_point(tab, g, S + lane);
          };
          if (X) fetch();
          while (X) {
            const uint32_t S1 = S, k1 = k, len1 = len;
            const uint4 p1 = p;
            X &= X - 1u;
            if (X) fetch();
            if (REC) runs_to(k1);
            const uint32_t bal = scan(lane < len1, S1 + lane, p1);
            if (ORD) windows(S1, len1, bal);
          }
          if (PAIRS && XS) {
            const uint32_t base = 16u * t0 + g.M;  // bucket t at 16 t + M, 15 points
            uint32_t k2 = NONE, pos = 0u;
            bool mine = false, more = true;
            auto fetch2 = [&]() {
              k = (uint32_t)__ffs(XS) - 1u;
              XS &= XS - 1u;
              k2 = XS ? (uint32_t)__ffs(XS) - 1u : NONE;
              XS &= XS - 1u;
              const uint32_t kk = lane < 16u ? k : k2;
              pos = base + 16u * kk + (lane & 15u);
              mine = (lane & 15u) != 15u && kk != NONE;
              if (mine) p = inorder_point(tab, g, pos);
            };
            fetch2();
            while (more) {
              const uint32_t ka = k, kb = k2, pos1 = pos;
              const bool mine1 = mine;
              const uint4 p1 = p;
              more = XS != 0u;
              if (more) fetch2();
              uint32_t bal = scan(mine1, pos1, p1);
              if (REC) {
                // (a loop: the code written out twice costs 100,000 small boxes 4 us of 117, and saves 65,536
                // large ones 60 of 1,119)
                uint32_t kx = ka;
#pragma unroll 1
                for (;;) {
                  runs_to(kx);
                  if (ORD) windows(base + 16u * kx, 15u, bal & 0xffffu);
                  if (kx == kb || kb == NONE) break;
                  kx = kb;
                  bal >>= 16;
                }
              }
            }
          }
        } else if (X) {
          const uint32_t k = (uint32_t)__ffs(X) - 1u;
          X &= X - 1u;
          if (REC) {
            put_runs(SM & ((1u << k) - 1u) & ~((1u << from) - 1u));
            from = k;
          }
          if (lane == 0) {
            s_lv[warp][lv] = make_uint4(t0, X, C, P);
            if (REC) s_from[warp][lv] = from;
          }
          t0 = (t0 + k) << WIDE;
          ++lv;
          enter(dc + WIDE, WIDE);
          continue;
        }
        if (REC) put_runs(SM & ~((1u << from) - 1u));
        // back to the last step that has descendants left to enter (or, recording, runs)
        if (lv == lv0) break;
        --lv;
        if (SPLIT && lv < lvs) lvs = NONE;
        __syncwarp();
        const uint4 e = s_lv[warp][lv];
        t0 = e.x;
        X = e.y;
        if (REC) {
          C = e.z;
          P = e.w;
          from = s_from[warp][lv];
          runs(w0 + WIDE * lv);
        }
        __syncwarp();
      }
    }
    if (REC) {
      if (KIND == WALK_RECORD) flush_ids();
      flush();
      if (lane == 0) sc.erec[oj] = recfail ? make_uint2(NO_RECORD, 0u) : make_uint2(efirst, etotal);
      if (recfail && lane == 0) sc.flags[atomicAdd(sc.flag_ctr, 1u)] = qj;
    }
    if (ORD) {
      // where the box's results of every depth start in its list
      uint32_t incl = acc;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
      }
      if (etotal) sc.ehist[oj * 32u + lane] = incl - acc;
      acc = __shfl_sync(0xffffffffu, incl, 31);
    } else {
      acc = __reduce_add_sync(0xffffffffu, acc);
    }
    if (DIG) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) dig += __shfl_xor_sync(0xffffffffu, dig, o);
    }
    if (SPLIT) {
      // (a box that no step was taken for, the whole tree or a small one: every warp has all of it)
      const bool whole = !neg(rootcut) || bdep == 0u;
      if (lane == 0) {
        s_acc[warp] = acc;
        if (DIG) s_dig[warp] = dig;
      }
      __syncthreads();
      if (warp) break;
      if (!whole) {
        for (int w = 1; w < SPLIT; ++w) {
          acc += s_acc[w];
          if (DIG) dig += s_dig[w];
        }
      }
    }
    if (lane == 0) {
      sc.counts[oj] = acc;
      if (DIG) sc.digests[oj] = dig;
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------- emission

// resident CTAs: 4 / 5 / 6 -> 2.55 / 2.48 / 2.55 ms of the 65,536-box search
constexpr int EMIT_MINB = 5;
constexpr int MT = 256;

// Writes every recorded box's ids to its slice: in the reference's order
// (ORDERED; ehist holds where each depth's results start), else in in-order
// position.  A warp per box; every step's ids are stored when the next step's
// loads are under way.
template <bool ORDERED>
__global__ void __launch_bounds__(MT, EMIT_MINB) k_emit(SearchCtx sc, uint32_t grab) {
  chain_wait();
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lt = (1u << lane) - 1u;
  const Geom g = sc.g;
  const uint32_t* __restrict__ ids = sc.tab.dids;
  // this lane's bit of a window: its depth (modulo 32), and the bits of the same depth before it
  const uint32_t myc = lane ? (uint32_t)__ffs(lane) - 1u : 0u;
  const uint32_t myd = g.H - myc;
  const uint32_t mypat = ORDERED ? window_class(myc) & lt : lt;
  // lane as a depth: the bits of a window at it
  const uint32_t dpat = ORDERED ? window_class(g.H - lane) : 0xffffffffu;
  const uint32_t dpatU = ORDERED ? window_class(g.H - 1u - lane) : 0xffffffffu;
  uint32_t qi = 0u, qend = 0u;  // this warp's boxes
  for (;; ++qi) {
    if (qi == qend) {
      if (lane == 0) qi = atomicAdd(sc.qcounter, grab);
      qi = __shfl_sync(0xffffffffu, qi, 0);
      qend = qi + grab;
    }
    if ((uint64_t)qi >= sc.boxes.q) break;
    const uint32_t j = sc.order ? sc.order[qi] : qi;
    const uint2 rec = sc.erec[j];
    const uint64_t base = sc.offsets[j], end = sc.offsets[j + 1u];
    const uint64_t space = (end < sc.capacity ? end : sc.capacity) - base;
    const uint32_t room = space < 0xfffffffeull ? (uint32_t)space : 0xfffffffeu;
    const uint32_t want = (uint32_t)(end - base);
    // ordered: where lane d writes the next id of depth d; else, in every lane, where the next id goes
    uint32_t cur = ORDERED ? sc.ehist[(uint64_t)j * 32u + lane] : 0u;
    if (rec.x == NO_RECORD && rec.y == 0u) continue;  // the traversing pass writes it
    if (end < base || sc.capacity < base || (end - base) >> 32) {  // not the slice of any box
      if (lane == 0) atomicOr(sc.err, ERRB_INTERNAL | (rec.y && (end < base || sc.capacity < base) ? ERRB_CAPACITY : 0u));
      continue;
    }
    uint32_t* out = sc.out + base;
    uint32_t written = 0u;
    bool failed = false;
    // the ids and places (0xffffffff: none) of the last two steps
    uint32_t v1 = 0u, p1 = 0xffffffffu, v2 = 0u, p2 = 0xffffffffu;
    auto step = [&](uint32_t p, bool hit, uint32_t pos) {
      uint32_t id = 0u;
      if (hit) id = __ldg(ids + p);
      if (p2 < room)
        out[p2] = v2;
      else if (p2 != 0xffffffffu)
        failed = true;
      v2 = v1;
      p2 = p1;
      v1 = id;
      p1 = hit ? pos : 0xffffffffu;
    };
    auto span = [&](uint32_t v0, uint32_t vz, bool up) {  // v in (v0, vz]
      if (v0 == vz) return;
      const uint32_t hr = g.H - (up ? 1u : 0u), off = up ? g.M - 1u : 0xffffffffu;
      for (uint32_t w = v0; w < vz; w += 32u) {
        const uint32_t v = w + 1u + lane;
        uint32_t pos;
        if (ORDERED) {
          // 2^c the largest power of two in v: the odd multiples of it in (v0, v)
          const uint32_t c = (uint32_t)__ffs(v) - 1u;
          pos = __shfl_sync(0xffffffffu, cur, (hr - c) & 31u) + ((v >> c) >> 1) - (((v0 >> c) + 1u) >> 1);
        } else {
          pos = cur + (v - v0 - 1u);
        }
        step(v + off, v <= vz, pos);
      }
      if (ORDERED) {
        const uint32_t c = hr - lane;
        if (c < 32u) cur += (((vz >> c) + 1u) >> 1) - (((v0 >> c) + 1u) >> 1);
      } else {
        cur += vz - v0;
      }
    };
    uint32_t at = rec.x, left = rec.y;
    while (left) {
      uint2 e = make_uint2(0u, 0u);
      if ((uint64_t)at + lane < sc.ent_cap) e = sc.ents[at + lane];
      // up to the first entry that is not a result itself: a link to the next block, a heading of ids
      const uint32_t heads = __ballot_sync(0xffffffffu, e.x >= E_IDS && lane < left);
      const uint32_t nv = heads ? (uint32_t)__ffs(heads) - 1u : min(left, 32u);
      const uint32_t head = __shfl_sync(0xffffffffu, e.x, nv & 31u), next = __shfl_sync(0xffffffffu, e.y, nv & 31u);
      for (uint32_t k = 0; k < nv; ++k) {
        const uint32_t x = __shfl_sync(0xffffffffu, e.x, k), y = __shfl_sync(0xffffffffu, e.y, k);
        if (x & E_WINDOW) {
          const bool up = (x & E_UPPER) != 0u;
          const uint32_t v = 32u * (x & (E_UPPER - 1u)) + lane;
          const uint32_t b = ORDERED ? __shfl_sync(0xffffffffu, cur, (myd - (up ? 1u : 0u)) & 31u) : cur;
          const uint32_t pos = b + __popc(y & mypat);
          cur += __popc(y & (up ? dpatU : dpat));
          step(up ? v + g.M - 1u : v - 1u, (y >> lane) & 1u, pos);
          written += __popc(y);
        } else {
          const uint32_t m2 = 2u * g.M;
          span(min(x, m2), min(x + y, m2), false);
          span(max(x, m2) - g.M, max(x + y, m2) - g.M, true);
          written += y;
        }
      }
      left -= nv;
      at += nv;
      if (heads && head == E_LINK) {
        at = next;
      } else if (heads) {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(sc.ents + at + 1u);
        for (uint32_t k = lane; k < next; k += 32u) {
          const uint32_t pos = cur + k;
          if (pos < room)
            out[pos] = src[k];
          else
            failed = true;
        }
        cur += next;
        written += next;
        left -= 1u + ((next + 1u) >> 1);
        at += 1u + ((next + 1u) >> 1);
      }
    }
    step(0u, false, 0u);
    step(0u, false, 0u);
    // the traversing pass's verdicts (k_search_write): no room for a result, or not the slice of this box
    // (each behind a branch of its own, 64 bits wide: 77 us of 100,000 boxes of 1.8 results instead of 43)
    const bool cut = __any_sync(0xffffffffu, failed);
    if ((cut || written != want) && lane == 0) atomicOr(sc.err, cut ? ERRB_CAPACITY : ERRB_INTERNAL);
  }
}

// A grid of resident CTAs whose warps take boxes from the call's counter, `grab`
// at a time: where a warp takes sixteen times or more, two -- one counter serves
// about one atomic a clock, which holds up small boxes, while large boxes want an
// even end (1 / 2 / 4 / 8: 258 / 229 / 230 / 229 us of 100,000 boxes of 1.8 results,
// 6.62 / 6.73 / 6.86 / 7.10 ms of the count of 1M boxes of 4,300, before pairs of buckets).
//
// Counts and digests of so few boxes that a warp each leaves the chip idle split
// a box over a CTA of eight, four or two warps: one warp's chain of dependent loads
// is all such a call waits for.  A form is taken up to `waves` times the boxes
// resident at once (592, 1,184 and 2,368 on 148 SMs): one wave, as in more of them the
// steps that all warps take and the smaller boxes cost what the largest save (of 2^24
// points in 3-D, a warp each / two: 3,000 boxes of 10,000 results 223 / 246 us, of
// 1,000 86 / 85, 8,000 of 1,000 133 / 142); in 4-D, where a box cuts far more
// subtrees, four (3,000 of 10,000 461 a warp each, 394 four; 8,000 686, 649 two).
// Counts of 2^24 uniform points, us, with the walk of single nodes / with this walk,
// four or two warps sharing a box's second step / as it is now: 500 boxes of 10,000
// results 137 / 221 / 71, 1,000 178 / 307 / 123, 2,000 181 / 297 / 160, 1,000 of 1,000
// 70 / 73 / 49, 1,000 of 10,000 in 4-D 354 / 555 / 225, 3,000 370 / 666 / 361, 2,000 of 5
// 46 / 36 / 40; the corner that is left is 3,000 of 10,000 in 3-D, 193 / 323 / 226.
template <class K>
struct Split {
  int warps;
  K kernel;
  int waves;
};

template <class K>
cudaError_t launch_boxes(K kernel, int threads, SearchCtx sc, int which,
                         std::initializer_list<Split<K>> splits = {}) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, 0);
  if (e != cudaSuccess) return e;
  if (per < 1) per = 1;
  const uint64_t q = sc.boxes.q;
  uint64_t blocks = (uint64_t)sms * per;
  const uint64_t need = (q * 32u + threads - 1u) / threads;
  if (blocks > need) blocks = need ? need : 1u;
  for (const Split<K>& f : splits) {
    if (sc.qdev || sc.evs) break;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f.kernel, 32 * f.warps, 0);
    if (e != cudaSuccess) return e;
    if (q <= (uint64_t)sms * per * f.waves)
      return chain_launch(f.kernel, dim3((unsigned)q), dim3(32 * f.warps), 0, sc.stream, sc, 0u);
  }
  uint64_t grab = q / (blocks * (uint64_t)(threads / 32) * 8u);
  if (grab > 2u) grab = 2u;
  if (grab < 1u) grab = 1u;
  e = work_counter(sc, which);
  if (e != cudaSuccess) return e;
  return chain_launch(kernel, dim3((unsigned)blocks), dim3(threads), 0, sc.stream, sc, (uint32_t)grab);
}

// In pairs unless less than an eighth of the buckets are short: then the second form
// of a step's tests costs more than it saves (2.18 against 2.13 ms of 131,072 counts
// of 10,000 results of 10^6 points, 329 / 319 us of 72,527 lists of balls in 2-D).
inline bool in_pairs(const SearchCtx& sc) { return sc.evs || sc.g.M < (7ull << sc.g.H >> 3); }

template <int DIM, int KIND, template <int> class SHAPE>
cudaError_t launch_records(const SearchCtx& sc) {
  return launch_boxes(in_pairs(sc) ? k_walk<DIM, KIND, SHAPE> : k_walk<DIM, KIND, SHAPE, 0, false>, WT, sc,
                      sc.qdev ? QC_LEFT : QC_WALK);
}

template <int DIM, int KIND, template <int> class SHAPE>
cudaError_t launch_counts(const SearchCtx& sc) {
  constexpr int waves = DIM == 4 ? 4 : 1;
  using K = void (*)(SearchCtx, uint32_t);
  return launch_boxes<K>(in_pairs(sc) ? k_walk<DIM, KIND, SHAPE> : k_walk<DIM, KIND, SHAPE, 0, false>, WT, sc,
                         sc.qdev ? QC_LEFT : QC_WALK,
                         {{8, k_walk<DIM, KIND, SHAPE, 8>, 1},
                          {4, k_walk<DIM, KIND, SHAPE, 4>, waves},
                          {2, k_walk<DIM, KIND, SHAPE, 2>, waves}});
}

template <int DIM>
cudaError_t walk_dim(const SearchCtx& sc, int mode) {
  if (mode == SEARCH_DIGEST) return launch_counts<DIM, WALK_DIGEST, BoxShape>(sc);
  if (!sc.ents) return launch_counts<DIM, WALK_COUNT, BoxShape>(sc);
  return sc.ehist ? launch_records<DIM, WALK_RECORD_ORDERED, BoxShape>(sc) : launch_records<DIM, WALK_RECORD, BoxShape>(sc);
}

template <int DIM>
cudaError_t walk_balls_dim(const SearchCtx& sc) {
  if (!sc.ents) return launch_counts<DIM, WALK_COUNT, BallShape>(sc);
  return launch_records<DIM, WALK_RECORD_ORDERED, BallShape>(sc);
}

}  // namespace

cudaError_t launch_walk(const SearchCtx& sc, int dim, int mode) {
  if (sc.boxes.q == 0) return cudaSuccess;
  switch (dim) {
    case 1: return walk_dim<1>(sc, mode);
    case 2: return walk_dim<2>(sc, mode);
    case 3: return walk_dim<3>(sc, mode);
    case 4: return walk_dim<4>(sc, mode);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_walk_balls(const SearchCtx& sc, int dim) {
  if (sc.boxes.q == 0) return cudaSuccess;
  switch (dim) {
    case 1: return walk_balls_dim<1>(sc);
    case 2: return walk_balls_dim<2>(sc);
    case 3: return walk_balls_dim<3>(sc);
    case 4: return walk_balls_dim<4>(sc);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_emit(const SearchCtx& sc, int ordered) {
  if (sc.boxes.q == 0) return cudaSuccess;
  return ordered ? launch_boxes(k_emit<true>, MT, sc, QC_EMIT) : launch_boxes(k_emit<false>, MT, sc, QC_EMIT);
}

}  // namespace fkd
