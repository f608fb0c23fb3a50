// fkd_tables.cu -- tables derived from a built tree for the searches
// (sm_100a), for one tree or every event of a batch:
//
//   dids          the ids in in-order position: node (d, t) owns the interval
//                 [start(d,t), start(d,t) + len(d,t)) of the build's working
//                 order (its left subtree, itself, its right subtree), so
//                 every subtree is one contiguous range
//   ipts          the nodes themselves in in-order position
//   sdig          the digest of every subtree (sum of mix64 over its ids)
//   bb            the bounding box of every subtree of height >= BB_HEIGHT:
//                 bb[2i], bb[2i+1] = (min), (max) of its points' coordinates.
//                 A subtree's cell (its ancestors' split values) also spans
//                 the empty space around its points; a box that lies in that
//                 space, or ends there, is decided by bb without a descent.
//
// k_tables takes a warp per bottom subtree ("bucket", height BB_HEIGHT, at
// most 31 points): lane k holds in-order position k of the bucket -- and one
// lane the node that follows the bucket, so that every position is written
// once and in order --, a warp scan gives the digests of all its subtrees
// and six warp reductions its bounding box.  It reads every node once and
// writes what was asked for (up to 48 B a point): bound by memory (0.40 ms for
// the 3-D events of a 33.6M-point batch with ipts, bb and sdig; the kernel it
// replaced wrote the in-order tables of 16M points in heap order, a 16-byte
// scatter, in 0.55 ms).
// k_tables_up combines the levels above, UP_LEVELS of them per launch.
#include "fkd_internal.h"

namespace fkd {
namespace {

constexpr int TT = 256;
constexpr uint32_t UP_LEVELS = 9;  // levels one CTA of k_tables_up combines (2^8 threads)

__device__ __forceinline__ float unmono(uint32_t m) {
  return __uint_as_float((m & 0x80000000u) ? (m & 0x7fffffffu) : ~m);
}

template <int DIM>
__global__ void __launch_bounds__(TT) k_tables(const EvDesc* __restrict__ evs, Table tab) {
  chain_wait();
  const EvDesc ev = evs[blockIdx.x];
  const Geom g = ev.g;
  if (g.n == 0u) return;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t bdep = g.H > BB_HEIGHT ? g.H - BB_HEIGHT : 0u;
  const uint4* nodes = tab.nodes + ev.base;
  float4* bb = tab.bb ? tab.bb + 2ull * bb_base(ev.base, blockIdx.x) : nullptr;
  const uint32_t wstep = gridDim.y * (TT / 32);
  for (uint32_t t = blockIdx.y * (TT / 32) + (threadIdx.x >> 5); t < (1u << bdep); t += wstep) {
    const uint32_t S = seg_start(g, bdep, t), len = seg_len(g, bdep, t);
    const uint32_t p = S + lane;
    const bool mine = lane < len;                    // a point of the bucket
    const bool have = lane <= len && p < g.n;        // ... or the node after it
    uint32_t d = 0u, u = 0u;
    const uint32_t i = have ? inorder_node(g, p, &d, &u) : 0u;
    uint4 nd = make_uint4(0u, 0u, 0u, 0u);
    if (have) nd = nodes[i];
    uint32_t id = nd.w;
    if (DIM > 3 && have && (tab.dids || tab.sdig)) id = tab.ids[ev.base + i];
    if (have) {
      if (tab.ipts) tab.ipts[ev.base + p] = nd;
      if (tab.dids) tab.dids[ev.base + p] = id;
    }
    if (bb) {
      const uint32_t w[4] = {nd.x, nd.y, nd.z, nd.w};
      float mn[4] = {0.f, 0.f, 0.f, 0.f}, mx[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < DIM; ++k) {
        const uint32_t m = mono_bits(w[k]);
        mn[k] = unmono(__reduce_min_sync(0xffffffffu, mine ? m : 0xffffffffu));
        mx[k] = unmono(__reduce_max_sync(0xffffffffu, mine ? m : 0u));
      }
      const uint32_t r = (1u << bdep) - 1u + t;
      if (lane == 0u) bb[2u * r] = make_float4(mn[0], mn[1], mn[2], mn[3]);
      if (lane == 1u) bb[2u * r + 1u] = make_float4(mx[0], mx[1], mx[2], mx[3]);
    }
    if (tab.sdig) {
      unsigned long long s = mine ? mix64(id) : 0ull;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= (uint32_t)o) s += y;
      }
      // the subtree of my node is the in-order range [a, a + n1) of the bucket
      const uint32_t a = mine ? seg_start(g, d, u) - S : 0u, n1 = mine ? seg_len(g, d, u) : 1u;
      const unsigned long long hi = __shfl_sync(0xffffffffu, s, (a + n1 - 1u) & 31u);
      const unsigned long long lo = __shfl_sync(0xffffffffu, s, (a - 1u) & 31u);
      if (mine) tab.sdig[ev.base + i] = hi - (a ? lo : 0ull);
    }
  }
}

// Levels [dr, dl) of every event: dl counts down from the bucket depth by
// UP_LEVELS per launch (`round`).  A CTA takes a node of depth dr and
// everything below it down to depth dl - 1, level by level.
template <int DIM>
__global__ void __launch_bounds__(1 << (UP_LEVELS - 1)) k_tables_up(const EvDesc* __restrict__ evs, Table tab,
                                                                   uint32_t round) {
  chain_wait();
  const EvDesc ev = evs[blockIdx.x];
  const Geom g = ev.g;
  if (g.n == 0u) return;
  const uint32_t bdep = g.H > BB_HEIGHT ? g.H - BB_HEIGHT : 0u;
  if (bdep <= round * UP_LEVELS) return;
  const uint32_t dl = bdep - round * UP_LEVELS;
  const uint32_t dr = dl > UP_LEVELS ? dl - UP_LEVELS : 0u;
  const uint4* nodes = tab.nodes + ev.base;
  float4* bb = tab.bb ? tab.bb + 2ull * bb_base(ev.base, blockIdx.x) : nullptr;
  unsigned long long* sd = tab.sdig ? tab.sdig + ev.base : nullptr;
  for (uint32_t r = blockIdx.y; r < (1u << dr); r += gridDim.y) {
    for (uint32_t d = dl; d-- > dr;) {
      const uint32_t k = threadIdx.x;
      if (k < (1u << (d - dr))) {
        const uint32_t i = (1u << d) - 1u + (r << (d - dr)) + k;
        const uint32_t l = 2u * i + 1u;  // both children exist: d < bdep <= H - 1 or H
        const uint4 nd = nodes[i];
        if (bb) {
          const float4 a0 = bb[2u * l], a1 = bb[2u * l + 1u], b0 = bb[2u * l + 2u], b1 = bb[2u * l + 3u];
          const float x = __uint_as_float(nd.x), y = __uint_as_float(nd.y), z = __uint_as_float(nd.z),
                      w = __uint_as_float(nd.w);
          float4 mn, mx;
          mn.x = fminf(fminf(a0.x, b0.x), x);
          mx.x = fmaxf(fmaxf(a1.x, b1.x), x);
          mn.y = DIM > 1 ? fminf(fminf(a0.y, b0.y), y) : 0.f;
          mx.y = DIM > 1 ? fmaxf(fmaxf(a1.y, b1.y), y) : 0.f;
          mn.z = DIM > 2 ? fminf(fminf(a0.z, b0.z), z) : 0.f;
          mx.z = DIM > 2 ? fmaxf(fmaxf(a1.z, b1.z), z) : 0.f;
          mn.w = DIM > 3 ? fminf(fminf(a0.w, b0.w), w) : 0.f;
          mx.w = DIM > 3 ? fmaxf(fmaxf(a1.w, b1.w), w) : 0.f;
          bb[2u * i] = mn;
          bb[2u * i + 1u] = mx;
        }
        if (sd) sd[i] = mix64(DIM <= 3 ? nd.w : tab.ids[ev.base + i]) + sd[l] + sd[l + 1u];
      }
      __syncthreads();
    }
  }
}

template <int DIM>
cudaError_t run_tables(const EvDesc* evs, uint32_t nev, uint32_t max_n, const Table& tab, cudaStream_t stream) {
  const Geom g = make_geom(max_n);
  const uint32_t bdep = g.H > BB_HEIGHT ? g.H - BB_HEIGHT : 0u;
  // about 8192 CTAs over all events
  const uint32_t cap = nev >= 1024u ? 8u : 8192u / nev;
  uint32_t gy = ((1u << bdep) + TT / 32 - 1u) / (TT / 32);
  if (gy > cap) gy = cap;
  FKD_CHAIN(k_tables<DIM>, dim3(dim3(nev, gy)), dim3(TT), 0, stream, evs, tab);
  if (tab.bb || tab.sdig) {
    for (uint32_t round = 0; round * UP_LEVELS < bdep; ++round) {
      const uint32_t dl = bdep - round * UP_LEVELS, dr = dl > UP_LEVELS ? dl - UP_LEVELS : 0u;
      uint32_t uy = 1u << dr;
      if (uy > cap) uy = cap;
      FKD_CHAIN(k_tables_up<DIM>, dim3(dim3(nev, uy)), dim3(1 << (UP_LEVELS - 1)), 0, stream, evs, tab, round);
    }
  }
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_tables(const EvDesc* evs, uint32_t nev, uint32_t max_n, const Table& tab, int dim,
                          cudaStream_t stream) {
  if (nev == 0 || max_n == 0) return cudaSuccess;
  switch (dim) {
    case 1: return run_tables<1>(evs, nev, max_n, tab, stream);
    case 2: return run_tables<2>(evs, nev, max_n, tab, stream);
    case 3: return run_tables<3>(evs, nev, max_n, tab, stream);
    case 4: return run_tables<4>(evs, nev, max_n, tab, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fkd
