// Tree arithmetic shared by the hierarchy builders (lbvh.cu, ploc.cu).
#pragma once
#include "eos_internal.cuh"

namespace eos {

constexpr float kCostNode = 1.0f;  // SAH cost of visiting one node (two box tests)
constexpr float kCostTri = 1.0f;   // SAH cost of one triangle test

__device__ __forceinline__ float half_area(float4 l, float4 h) {
  float dx = h.x - l.x, dy = h.y - l.y, dz = h.z - l.z;
  return dx * dy + dy * dz + dz * dx;
}

// Box of a binary node from its children's boxes (l0, h0) and (l1, h1), whose .w of lo is the
// subtree's SAH cost; `size` triangles lie below it.  Returns the node's cost in lo.w and the
// leaf decision in hi.w: fixed layout -> a subtree of at most max_leaf triangles becomes one
// leaf; SAH layout -> additionally the leaf's cost kCostTri * size is not above kCostNode +
// (A_l cost_l + A_r cost_r) / A.
__device__ __forceinline__ void join_boxes(float4 l0, float4 h0, float4 l1, float4 h1, int size, int max_leaf, int sah,
                                           float4& lo, float4& hi) {
  lo = make_float4(fminf(l0.x, l1.x), fminf(l0.y, l1.y), fminf(l0.z, l1.z), 0.0f);
  hi = make_float4(fmaxf(h0.x, h1.x), fmaxf(h0.y, h1.y), fmaxf(h0.z, h1.z), 0.0f);
  const float a = half_area(lo, hi);
  const float inner = kCostNode + (a > 0.0f ? (half_area(l0, h0) * l0.w + half_area(l1, h1) * l1.w) / a : l0.w + l1.w);
  const float as_leaf = size <= max_leaf ? kCostTri * (float)size : kInf;
  const bool collapse = sah ? (as_leaf <= inner) : (size <= max_leaf);
  lo.w = collapse ? as_leaf : inner;
  hi.w = collapse ? 1.0f : 0.0f;
}

}  // namespace eos
