// fkd_walk.cuh -- what the searches that use the subtrees' bounding boxes
// (fkd_tables.cu) share: box and ball tests against points and bounding boxes.
//
// Box tests by sign: a - lo < 0 exactly when a < lo, with gradual underflow
// and lo free of +0 (and hi - a with hi free of -0: a zero difference is then
// never -0); inf - inf is a NaN, whose sign is clear in the result of a
// subtraction.  The differences run in the FMA pipe and their signs are
// combined by three-input logic: half the work on the ALU pipe, which bounds
// these kernels, of comparisons.  Boxes with a NaN bound or lo > hi hold no
// point and are answered up front (ok below).
#pragma once
#include <math.h>

#include "fkd_internal.h"

namespace fkd {

__device__ __forceinline__ uint32_t diff(float a, float b) { return __float_as_uint(__fsub_rn(a, b)); }
__device__ __forceinline__ bool neg(uint32_t w) { return (int)w < 0; }
__device__ __forceinline__ float word(const float4& p, int c) {
  return c == 0 ? p.x : (c == 1 ? p.y : (c == 2 ? p.z : p.w));
}
__device__ __forceinline__ float4 as_float4(const uint4& p) {
  return make_float4(__uint_as_float(p.x), __uint_as_float(p.y), __uint_as_float(p.z), __uint_as_float(p.w));
}

// Batched search over a subset of the events (sc.evsel, in increasing
// order, with sc.evsel_q the exclusive prefix of their box counts): the
// qi-th box of the subset, and its event.
__device__ __forceinline__ uint32_t select_box(const SearchCtx& sc, uint32_t qi, uint32_t& ev) {
  uint32_t lo = 0u, hi = sc.nsel;  // evsel_q[lo] <= qi < evsel_q[hi]
  while (hi - lo > 1u) {
    const uint32_t mid = (lo + hi) >> 1;
    if (sc.evsel_q[mid] <= (uint64_t)qi)
      lo = mid;
    else
      hi = mid;
  }
  ev = sc.evsel[lo];
  return (uint32_t)(sc.evs[ev].qbase + ((uint64_t)qi - sc.evsel_q[lo]));
}

// The point at in-order position p (without the in-order copy, from its heap
// position: a bucket's points then are five contiguous pieces).
__device__ __forceinline__ uint4 inorder_point(const Table& tab, const Geom& g, uint32_t p) {
  if (tab.ipts) return __ldg(tab.ipts + p);
  uint32_t d, t;
  return __ldg(tab.nodes + inorder_node(g, p, &d, &t));
}

template <int DIM>
struct BoxShape {
  float lo[DIM], hi[DIM];
  // box j of SoA bounds; false when it can hold no point
  __device__ __forceinline__ bool load(const float* __restrict__ l, const float* __restrict__ h, uint64_t stride,
                                       uint64_t j) {
    bool ok = true;
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      lo[c] = l[(uint64_t)c * stride + j];
      hi[c] = h[(uint64_t)c * stride + j];
      ok = ok && lo[c] <= hi[c];
      if (lo[c] == 0.f) lo[c] = -0.f;
      if (hi[c] == 0.f) hi[c] = 0.f;
    }
    return ok;
  }
  // sign set: the point lies outside
  __device__ __forceinline__ uint32_t outside(const float4& p) const {
    uint32_t o = 0u;
#pragma unroll
    for (int c = 0; c < DIM; ++c) o |= diff(word(p, c), lo[c]) | diff(hi[c], word(p, c));
    return o;
  }
  // a subtree's bounding box: sign of `out`: no point of it is inside; sign of `cut`: not all are
  __device__ __forceinline__ void place(const float4& mn, const float4& mx, uint32_t& out, uint32_t& cut) const {
    out = cut = 0u;
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      out |= diff(word(mx, c), lo[c]) | diff(hi[c], word(mn, c));
      cut |= diff(word(mn, c), lo[c]) | diff(hi[c], word(mx, c));
    }
  }
};

// Ball of squared radius r2, the distances evaluated as fkd_nn.cu defines them
// (every operation rounded on its own).  Rounding is monotone, so the
// distances to the nearest and farthest corner, evaluated the same way, bound
// those of all points between: a subtree is dropped or taken whole only when
// every one of its points compares alike.
template <int DIM>
struct BallShape {
  float ctr[DIM], r2;
  // ball j: SoA centres and radii; false when it can hold no point
  __device__ __forceinline__ bool load(const float* __restrict__ c, const float* __restrict__ r, uint64_t stride,
                                       uint64_t j) {
    bool ok = r[j] >= 0.f;
    r2 = __fmul_rn(r[j], r[j]);
#pragma unroll
    for (int k = 0; k < DIM; ++k) {
      ctr[k] = c[(uint64_t)k * stride + j];
      ok = ok && ctr[k] == ctr[k];
    }
    return ok;
  }
  __device__ __forceinline__ uint32_t outside(const float4& p) const {
    float d2 = 0.f;
#pragma unroll
    for (int k = 0; k < DIM; ++k) {
      const float t = __fsub_rn(word(p, k), ctr[k]);
      d2 = __fadd_rn(d2, __fmul_rn(t, t));
    }
    return d2 <= r2 ? 0u : 0x80000000u;
  }
  __device__ __forceinline__ void place(const float4& mn, const float4& mx, uint32_t& out, uint32_t& cut) const {
    float near2 = 0.f, far2 = 0.f;
#pragma unroll
    for (int k = 0; k < DIM; ++k) {
      const float a = __fsub_rn(word(mn, k), ctr[k]), b = __fsub_rn(ctr[k], word(mx, k));
      const float t = fmaxf(fmaxf(a, b), 0.f);  // (infinite coordinates: a NaN counts as 0)
      near2 = __fadd_rn(near2, __fmul_rn(t, t));
      const float u = fmaxf(fabsf(a), fabsf(b));
      far2 = __fadd_rn(far2, __fmul_rn(u, u));
    }
    out = near2 > r2 ? 0x80000000u : 0u;
    // a point whose distance is not a number is not inside: then some difference here is infinite
    cut = (far2 <= r2 && far2 < INFINITY) ? 0u : 0x80000000u;
  }
};

}  // namespace fkd
