// fkd_mid.cu -- the last global levels of a build, one CTA per segment.
//
// A segment of at most MIDN points fits one CTA's shared memory, so the levels
// between it and the subtree kernel's size (three or four of them) are split
// there: the records are read once and written once, instead of a select, a
// partition and a tie launch per level that read and write every record.
//
// Split of the work: the CTA starts as one group of T threads on the whole
// segment; after each level its halves are groups of their own, one per child,
// with their own barrier (bar.sync by id), so that a thread keeps about eight
// points at every level and no group waits for another.  A level of a group:
// the range of the split coordinate's order bits, a histogram of it in 2 T
// bins (narrowed until at most MCAND candidates hold the pivot's rank; the
// id's range is binned once a single value is left), the candidates ranked by
// the full key (coordinate, then id: FKDTree_cpu.h:246-252), and the move:
// every thread knows where its points go, so the records move word by word in
// place, the last level straight to global memory.
//
// Bound by the issue of integer compares and selects (one CTA of 1,024 threads
// fills the SM's registers; 8,192 points are 14 waves of a 16.8M-point build),
// not by its 0.5 GB of traffic: 389 us there, where the launches of the three
// levels took about 550 us.  Measured against the launches: build of 16.8M
// points 4,327 -> 4,133 us, of 100,000 237 -> 209 us, of 1.23M 4-D points
// 857 -> 812 us.  Segments of 4,096 points, three CTAs per SM: 4,209 us (one
// more level by launches).  A list of 128 candidates instead of 32 saves a
// third of the histogram passes but its ranking costs more (16.8M: +60 us).
#include "fkd_internal.h"

namespace fkd {

namespace {

constexpr int MIDN = 8192;
constexpr int PP = 8;           // points per thread
constexpr int MT = MIDN / PP;   // threads
constexpr int MSLOTS = 15;      // groups of four levels: 1 + 2 + 4 + 8
constexpr uint32_t MCAND = 32;  // candidates a group ranks by their full keys
static_assert(MCAND <= MT / 8, "a group's bins hold its candidates' keys");

struct MidGroup {
  uint32_t lo, hi;     // the candidates' interval (order bits of the value, or ids)
  uint32_t krem, cnt;  // the pivot's rank among the candidates, their number
  uint32_t ncand;
  uint32_t cur;        // points moved left | right << 16
  uint32_t dup;        // tickets of points with the pivot's very key
};

// one word, global to shared memory, not waited for
__device__ __forceinline__ void copy_word(uint32_t* to, const uint32_t* from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from)
               : "memory");
}

template <int DIM>
constexpr size_t mid_smem() {
  return ((size_t)(DIM + 1) * MIDN + 2 * MT) * 4;
}

}  // namespace

template <int DIM>
__global__ void __launch_bounds__(MT, 1) k_mid(const EvDesc* __restrict__ evs,
                                                          const uint2* __restrict__ mids, CSoA src_in, SoA buf0,
                                                          SoA buf1, Table tab_all, uint32_t* __restrict__ err) {
  chain_wait();
  extern __shared__ __align__(16) uint32_t rec[];  // [DIM + 1][MIDN], then 2 MT bins
  uint32_t* const hist = rec + (size_t)(DIM + 1) * MIDN;
  __shared__ MidGroup grp[MSLOTS];
  __shared__ uint32_t wsum[MT / 32];

  const uint2 sb = mids[blockIdx.x];
  const EvDesc ev = evs[sb.x];
  const Geom g = ev.g;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t base = seg_start(g, ev.dm, sb.y);
  const uint32_t nloc = seg_len(g, ev.dm, sb.y);
  if (nloc > (uint32_t)MIDN || ev.d0 > ev.dm + 4u) {
    if (threadIdx.x == 0) atomicOr(err, ERRB_INTERNAL);
    return;
  }
  // where the records sit after the event's first dm levels, and where the subtree kernel reads them
  const CSoA b0{buf0.base, buf0.ids, buf0.stride}, b1{buf1.base, buf1.ids, buf1.stride};
  const CSoA src = ev.dm == 0u ? src_in : ((ev.dm & 1u) ? b0 : b1);
  const SoA dst = (ev.d0 & 1u) ? buf0 : buf1;
  const uint64_t gb = (uint64_t)ev.base + base;
  const Table tab{tab_all.nodes + ev.base, tab_all.ids + ev.base};
  if (threadIdx.x < (uint32_t)MSLOTS) grp[threadIdx.x] = MidGroup{0xffffffffu, 0u, 0u, 0u, 0u, 0u, 0u};
  // the first level's split coordinate, then the other words, which that level's select does not wait for
  const uint32_t c0 = ev.dm % DIM;
#pragma unroll
  for (int w = 0; w <= DIM; ++w) {
    const uint32_t x = w < DIM ? (c0 + w) % DIM : DIM;
    const uint32_t* from = w < DIM ? src.base + (uint64_t)x * src.stride + gb : src.ids + gb;
#pragma unroll
    for (int k = 0; k < PP; ++k) {
      const uint32_t p = threadIdx.x + k * MT;
      if (p < nloc) copy_word(rec + x * MIDN + p, from + p);
    }
    if (w == 0) asm volatile("cp.async.commit_group;" ::: "memory");
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 1;" ::: "memory");
  __syncthreads();

  uint32_t t = sb.y, gi = 0u, gt = MT, tg = threadIdx.x;
  const uint32_t lt = (1u << lane) - 1u;
  bool pending = true;  // the other words are still on their way
  for (uint32_t d = ev.dm; d < ev.d0; ++d) {
    const uint32_t slot = (1u << (d - ev.dm)) - 1u + gi;
    MidGroup* const S = grp + slot;
    const uint32_t ls = seg_start(g, d, t) - base, m = seg_len(g, d, t), rank = seg_rank(g, d, t);
    const uint32_t c = d % DIM;
    const uint32_t* X = rec + (size_t)c * MIDN + ls;
    const uint32_t* I = rec + (size_t)DIM * MIDN + ls;
    uint32_t* const H = hist + 2u * (threadIdx.x - tg);  // the group's 2 gt bins
    const uint32_t w0 = (threadIdx.x - tg) >> 5;         // its first warp
    const bool last = d + 1u == ev.d0;
    unsigned long long* const K = reinterpret_cast<unsigned long long*>(H);  // later the candidates' keys
    auto gsync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(slot + 1u), "r"(gt) : "memory"); };
    auto arrive = [&]() {  // CTA-wide: only the first level's group meets words that are on their way
      if (!pending) return;
      pending = false;
      asm volatile("cp.async.wait_all;" ::: "memory");
      if (d == 0u) {  // deeper levels move the records level 0 checked
        bool nan = false;
#pragma unroll
        for (int w = 0; w < DIM; ++w) {
#pragma unroll
          for (int k = 0; k < PP; ++k)
            if (tg + k * gt < m) nan |= is_nan_bits(rec[w * MIDN + tg + k * gt]);
        }
        if (nan) atomicOr(err, ERRB_NAN);
      }
      gsync();
    };
    // this thread's points: positions tg + k gt below m, the bits of vm
    const uint32_t nv = tg < m ? min((uint32_t)PP, (m - tg + gt - 1u) / gt) : 0u;
    const uint32_t vm = (1u << nv) - 1u;
    // the range of the split coordinate (a thread short of points repeats one of the segment)
    uint32_t kv[PP];
    {
      const uint32_t fill = X[0];
#pragma unroll
      for (int k = 0; k < PP; ++k) kv[k] = mono_bits((vm >> k) & 1u ? X[tg + k * gt] : fill);
      uint32_t mn = kv[0], mx = kv[0];
#pragma unroll
      for (int k = 1; k < PP; ++k) {
        mn = min(mn, kv[k]);
        mx = max(mx, kv[k]);
      }
      *reinterpret_cast<uint2*>(H + 2u * tg) = make_uint2(0u, 0u);
      mn = __reduce_min_sync(0xffffffffu, mn);
      mx = __reduce_max_sync(0xffffffffu, mx);
      if (lane == 0u) {
        atomicMin(&S->lo, mn);
        atomicMax(&S->hi, mx);
      }
    }
    gsync();
    uint32_t lo = S->lo, hi = S->hi, cnt = m, krem = rank, v0 = 0u;
    bool idmode = false;  // one value left, v0: [lo, hi] is a range of ids
    const uint32_t lb = 31u - (uint32_t)__clz(2u * gt);  // log2 of the bins
    for (int guard = 0; guard < 12 && cnt > MCAND; ++guard) {
      if (guard || lo >= hi) arrive();
      if (lo >= hi) {
        if (idmode) break;  // more than MCAND points share the pivot's key
        idmode = true;
        v0 = lo;
        gsync();
        if (tg == 0u) {
          S->lo = 0xffffffffu;
          S->hi = 0u;
        }
        gsync();
        uint32_t mn = 0xffffffffu, mx = 0u;
#pragma unroll
        for (int k = 0; k < PP; ++k) {
          if (((vm >> k) & 1u) && kv[k] == v0) {
            const uint32_t id = I[tg + k * gt];
            mn = min(mn, id);
            mx = max(mx, id);
          }
        }
        mn = __reduce_min_sync(0xffffffffu, mn);
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 0u && mn <= mx) {
          atomicMin(&S->lo, mn);
          atomicMax(&S->hi, mx);
        }
        gsync();
        lo = S->lo;
        hi = S->hi;
        continue;
      }
      const uint32_t rb = 32u - (uint32_t)__clz(hi - lo);
      const uint32_t sh = rb > lb ? rb - lb : 0u;
#pragma unroll
      for (int k = 0; k < PP; ++k) {
        if (((vm >> k) & 1u) && (!idmode || kv[k] == v0)) {
          const uint32_t v = idmode ? I[tg + k * gt] : kv[k];
          if (v - lo <= hi - lo) atomicAdd(&H[(v - lo) >> sh], 1u);
        }
      }
      gsync();
      const uint2 h = *reinterpret_cast<const uint2*>(H + 2u * tg);
      *reinterpret_cast<uint2*>(H + 2u * tg) = make_uint2(0u, 0u);  // for the next pass
      const uint32_t mine = h.x + h.y;
      uint32_t incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
      }
      if (lane == 31u) wsum[warp] = incl;
      gsync();
      const uint32_t before = __reduce_add_sync(0xffffffffu, w0 + lane < warp ? wsum[w0 + lane] : 0u);
      const uint32_t cum = before + incl - mine;
      if (krem >= cum && krem - cum < mine) {
        const bool second = krem - cum >= h.x;
        const uint32_t nlo = lo + ((2u * tg + (second ? 1u : 0u)) << sh);
        S->lo = nlo;
        S->hi = hi - nlo < (1u << sh) ? hi : nlo + ((1u << sh) - 1u);
        S->krem = krem - cum - (second ? h.x : 0u);
        S->cnt = second ? h.y : h.x;
      }
      gsync();
      lo = S->lo;
      hi = S->hi;
      krem = S->krem;
      cnt = S->cnt;
    }
    arrive();
    // sides; the candidates are ranked by the full key
    uint32_t lm = 0u, cm = 0u;  // bit k: point k goes left / is a candidate
    if (!idmode) {
#pragma unroll
      for (int k = 0; k < PP; ++k) {
        if (kv[k] < lo) lm |= 1u << k;
        if (kv[k] - lo <= hi - lo) cm |= 1u << k;
      }
    } else {
#pragma unroll
      for (int k = 0; k < PP; ++k) {
        if (!((vm >> k) & 1u)) continue;
        const uint32_t id = kv[k] == v0 ? I[tg + k * gt] : 0u;
        if (kv[k] < v0 || (kv[k] == v0 && id < lo)) lm |= 1u << k;
        if (kv[k] == v0 && id - lo <= hi - lo) cm |= 1u << k;
      }
    }
    lm &= vm;
    cm &= vm;
    uint32_t rm = vm & ~(lm | cm);  // goes right
    if (cnt <= MCAND) {
      for (uint32_t left = cm; left; left &= left - 1u) {
        const uint32_t p = tg + ((uint32_t)__ffs((int)left) - 1u) * gt;
        const uint32_t at = atomicAdd(&S->ncand, 1u);
        if (at < MCAND)
          K[at] = order_key(X[p], I[p]);
        else
          atomicOr(err, ERRB_INTERNAL);
      }
    }
    gsync();
    for (uint32_t left = cm; left; left &= left - 1u) {
      const uint32_t k = (uint32_t)__ffs((int)left) - 1u, p = tg + k * gt;
      uint32_t less = 0u, eq = cnt;
      if (cnt <= MCAND) {
        const unsigned long long key = order_key(X[p], I[p]);
        eq = 0u;
        for (uint32_t o = 0; o < cnt; ++o) {
          const unsigned long long x = K[o];
          less += x < key ? 1u : 0u;
          eq += x == key ? 1u : 0u;
        }
      }
      // points with the pivot's very key (repeated keys only) take tickets
      uint32_t r = less;
      if (krem >= less && krem - less < eq) r += eq == 1u ? 0u : atomicAdd(&S->dup, 1u);
      if (r == krem) {
        uint32_t w[DIM + 1];
#pragma unroll
        for (int x = 0; x <= DIM; ++x) w[x] = rec[x * MIDN + ls + p];
        const uint32_t node = (1u << d) - 1u + t;
        tab.nodes[node] = make_uint4(w[0], DIM > 1 ? w[1 % (DIM + 1)] : 0u, DIM > 2 ? w[2 % (DIM + 1)] : 0u,
                                     DIM > 3 ? w[3 % (DIM + 1)] : w[DIM]);
        tab.ids[node] = w[DIM];
      } else if (r < krem) {
        lm |= 1u << k;
      } else {
        rm |= 1u << k;
      }
    }
    // destinations: one cursor step per warp
    uint32_t to[PP];
    {
      const uint32_t tot = __reduce_add_sync(0xffffffffu, __popc(lm) | (__popc(rm) << 16));
      uint32_t cur = 0u;
      if (lane == 0u) cur = atomicAdd(&S->cur, tot);
      cur = __shfl_sync(0xffffffffu, cur, 0);
      uint32_t nl = cur & 0xffffu, nr = cur >> 16;
      if (nl + (tot & 0xffffu) > rank || nr + (tot >> 16) > m - 1u - rank) {  // warp-uniform
        if (lane == 0u) atomicOr(err, ERRB_INTERNAL);
        lm = rm = 0u;
      }
      nr += rank + 1u;
      if (__all_sync(0xffffffffu, (lm | rm) == (1u << PP) - 1u)) {
        // every point of the warp moves: those that do not go left go right
        nr += lane;
#pragma unroll
        for (int k = 0; k < PP; ++k) {
          const bool l = (lm >> k) & 1u;
          const uint32_t bl = __ballot_sync(0xffffffffu, l), q = __popc(bl & lt), n = __popc(bl);
          to[k] = l ? nl + q : nr - q;
          nl += n;
          nr += 32u - n;
        }
      } else {
#pragma unroll
        for (int k = 0; k < PP; ++k) {
          const bool l = (lm >> k) & 1u;
          const uint32_t bl = __ballot_sync(0xffffffffu, l), br = __ballot_sync(0xffffffffu, (rm >> k) & 1u);
          to[k] = l ? nl + __popc(bl & lt) : nr + __popc(br & lt);
          nl += __popc(bl);
          nr += __popc(br);
        }
      }
    }
    const uint32_t mv = lm | rm;
    if (last) {
#pragma unroll
      for (int w = 0; w <= DIM; ++w) {
        uint32_t* out = (w < DIM ? dst.base + (uint64_t)w * dst.stride : dst.ids) + gb + ls;
#pragma unroll
        for (int k = 0; k < PP; ++k) {
          if ((mv >> k) & 1u) __stcs(out + to[k], rec[w * MIDN + ls + tg + k * gt]);
        }
      }
      break;
    }
    // two words at a time: all of a group's loads come before its stores
#pragma unroll
    for (int w = 0; w <= DIM; w += 2) {
      uint32_t a[PP], b[PP];
#pragma unroll
      for (int k = 0; k < PP; ++k) {
        if ((mv >> k) & 1u) {
          a[k] = rec[w * MIDN + ls + tg + k * gt];
          if (w < DIM) b[k] = rec[(w + 1) * MIDN + ls + tg + k * gt];
        }
      }
      gsync();
#pragma unroll
      for (int k = 0; k < PP; ++k) {
        if ((mv >> k) & 1u) {
          rec[w * MIDN + ls + to[k]] = a[k];
          if (w < DIM) rec[(w + 1) * MIDN + ls + to[k]] = b[k];
        }
      }
    }
    gsync();
    // the halves go on as groups of their own
    gt >>= 1;
    const uint32_t half = tg >= gt ? 1u : 0u;
    tg -= half * gt;
    gi = 2u * gi + half;
    t = 2u * t + half;
  }
}

uint32_t mid_capacity() { return (uint32_t)MIDN; }

template <int DIM>
static cudaError_t run_mid(const EvDesc* evs, const uint2* mids, uint32_t nmid, CSoA in, SoA b0, SoA b1, Table tab,
                           uint32_t* err, cudaStream_t stream) {
  constexpr size_t smem = mid_smem<DIM>();
  cudaError_t e = cudaFuncSetAttribute(k_mid<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  return chain_launch(k_mid<DIM>, dim3(nmid), dim3(MT), smem, stream, evs, mids, in, b0, b1, tab, err);
}

cudaError_t launch_mid(const EvDesc* evs, const uint2* mids, uint32_t nmid, CSoA in, SoA b0, SoA b1, Table tab,
                       uint32_t* err, int dim, cudaStream_t stream) {
  if (nmid == 0) return cudaSuccess;
  switch (dim) {
    case 1: return run_mid<1>(evs, mids, nmid, in, b0, b1, tab, err, stream);
    case 2: return run_mid<2>(evs, mids, nmid, in, b0, b1, tab, err, stream);
    case 3: return run_mid<3>(evs, mids, nmid, in, b0, b1, tab, err, stream);
    case 4: return run_mid<4>(evs, mids, nmid, in, b0, b1, tab, err, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fkd
