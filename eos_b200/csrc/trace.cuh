// BVH traversal and shading device functions (header-only; included by the kernel TUs).
//
// Nearest hit = the smallest t >= 0 over all triangles, exact ties resolved to the larger
// triangle id.  This is the reference's result (src/BVH.cpp:609-659 keeps t <= best
// through Triangle::hit, src/Triangle.cpp:37-38) without its dependence on one particular
// tree: the reference keeps the later of two equal hits in its own traversal order.
// Shadow rays = any triangle hit at t >= 0 (src/BVH.cpp:661-716 with the uninitialised
// distance at :703 read as FLT_MAX).
//
// Box tests are conservative so that culling never removes the exact answer:
//  * slab far distances are widened by 1 + 2*gamma(3) (rounding of (b - o) * (1/d));
//    the traversals use a one-instruction-per-plane form that accepts a superset of those
//    boxes (FmaSlabRay);
//  * a box is culled against the current best t only beyond best * (1 + 2^-12), a margin
//    for the rounding of the triangle test's own t;
//  * a direction component with |d| < 1e-30 is treated as parallel: its slab is the whole
//    line when the origin lies inside the closed slab and empty otherwise (the
//    reference's (b - o) * inf turns into NaN there, src/Box.cu:234-255).
#pragma once
#include "eos_internal.cuh"

namespace eos {

constexpr float kSlack = 1.0000004f;           // 1 + 2*gamma(3)
constexpr float kCull = 1.000244140625f;       // 1 + 2^-12
constexpr float kParallelEps = 1e-30f;
constexpr float kRayEps = 1e-3f;               // shadow / mirror ray offset, src/RayTracer.cpp:305

// Ray prepared for box tests.  sx / sy / sz are 16 x the near plane's chunk of each axis in a
// node record (chunks 0..2 = lo.xyz, 3..5 = hi.xyz): lo for a direction component >= 0 or a
// parallel axis, hi otherwise; the far plane is the other one.  The near and far
// distances are then (near - o) / d and (far - o) / d directly, the same values the
// min / max of the two plane distances would give.
struct SlabRay {
  float ox, oy, oz, ix, iy, iz;
  uint32_t sx, sy, sz;
  bool par;
};

__device__ __forceinline__ SlabRay make_slab(f3 o, f3 d) {
  SlabRay r;
  r.ox = o.x; r.oy = o.y; r.oz = o.z;
  bool px = fabsf(d.x) < kParallelEps, py = fabsf(d.y) < kParallelEps, pz = fabsf(d.z) < kParallelEps;
  r.ix = px ? 0.0f : 1.0f / d.x;
  r.iy = py ? 0.0f : 1.0f / d.y;
  r.iz = pz ? 0.0f : 1.0f / d.z;
  r.sx = (px || d.x >= 0.0f) ? 0u : 48u;
  r.sy = (py || d.y >= 0.0f) ? 16u : 64u;
  r.sz = (pz || d.z >= 0.0f) ? 32u : 80u;
  r.par = px || py || pz;
  return r;
}

// Three-input min / max (sm_100): exact, like two fminf / fmaxf.
__device__ __forceinline__ float min3f(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max3f(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Entry and exit distances of a box from its near planes (nx, ny, nz) and far planes
// (fx, fy, fz).  Rays with a (near-)zero direction component take the containment branch
// (near = lo, far = hi there); it is warp-uniform in practice (whole pixel columns share it).
__device__ __forceinline__ void slab_range(const SlabRay& r, float nx, float ny, float nz, float fx, float fy,
                                           float fz, float& tn, float& tf) {
  float tnx = (nx - r.ox) * r.ix, tfx = (fx - r.ox) * r.ix;
  float tny = (ny - r.oy) * r.iy, tfy = (fy - r.oy) * r.iy;
  float tnz = (nz - r.oz) * r.iz, tfz = (fz - r.oz) * r.iz;
  if (r.par) {
    if (r.ix == 0.0f) { tnx = -kInf; tfx = (r.ox >= nx && r.ox <= fx) ? kInf : -kInf; }
    if (r.iy == 0.0f) { tny = -kInf; tfy = (r.oy >= ny && r.oy <= fy) ? kInf : -kInf; }
    if (r.iz == 0.0f) { tnz = -kInf; tfz = (r.oz >= nz && r.oz <= fz) ? kInf : -kInf; }
  }
  tn = fmaxf(max3f(tnx, tny, tnz), 0.0f);
  tf = min3f(tfx, tfy, tfz) * kSlack;
}

// Box test in the form b = fma(p, i, c) per plane (i = 1/d), one instruction where
// (p - o) * i takes two; used by both traversals.  c is offset per axis: c_near = fl(c - eps),
// c_far = fl(c + eps), c = fl(-(o i)), eps = 2^-20 |c| + 2^-126.  With u = 2^-24 and
// x = (p - o) i: p i + c_near = x - o i d3 - eps' <= x - eps / 4 (the rounding of c is
// <= 1.0001u|c| <= eps / 16), so b_near <= x + u|x|, and likewise b_far >= x - u|x|;
// the (p - o) * i value a satisfies |a - x| <= 2.0001u|x|.  Hence max(b_near) <=
// max(a_near)(1 + 3.0002u) when that is >= 0 (both entries clamp to 0 otherwise) and
// min(b_far) >= min(a_far)(1 - 3.0002u) when min(a_far) >= 0, and the exit distance
// times 1 + 2^-19 (>= kSlack (1 + 8u) / (1 - u)) accepts every box that slab_hit accepts.
// The entry distance exceeds the exact form's by at most 3.0002u relative, so nearest-hit
// culling compares it with best * (kCull + 2^-19) (RayCull), which keeps every box and
// stack entry the exact form keeps.  Rays with a parallel axis or |o / d| above 1e30 keep
// the exact form (fma_slab_ok).
struct FmaSlabRay {
  float ix, iy, iz, nx, ny, nz, fx, fy, fz;
  uint32_t sx, sy, sz;
};

__device__ __forceinline__ bool fma_slab_ok(const SlabRay& r) {
  return !r.par && fabsf(r.ox * r.ix) <= 1e30f && fabsf(r.oy * r.iy) <= 1e30f && fabsf(r.oz * r.iz) <= 1e30f;
}

__device__ __forceinline__ void fma_axis(float o, float i, float& cn, float& cf) {
  const float c = -(o * i);
  const float eps = fabsf(c) * 0x1p-20f + 0x1p-126f;
  cn = c - eps;
  cf = c + eps;
}

__device__ __forceinline__ FmaSlabRay make_fma_slab(const SlabRay& r) {
  FmaSlabRay q;
  q.ix = r.ix; q.iy = r.iy; q.iz = r.iz;
  q.sx = r.sx; q.sy = r.sy; q.sz = r.sz;
  fma_axis(r.ox, r.ix, q.nx, q.fx);
  fma_axis(r.oy, r.iy, q.ny, q.fy);
  fma_axis(r.oz, r.iz, q.nz, q.fz);
  return q;
}

// Culling factor on the best hit distance per ray form: the fma form's entry distance can
// exceed the exact form's by 3.0002u relative, which 2^-19 more covers.
template <class Ray>
struct RayCull {
  static constexpr float k = kCull;
};
template <>
struct RayCull<FmaSlabRay> {
  static constexpr float k = 1.0f + 0x1p-12f + 0x1p-19f;
};

struct Hit {
  float t, u, v;
  int pos;  // sorted position, -1 on a miss
  int id;   // triangle id
  unsigned nodes, tests;  // interior nodes fetched, triangles tested
};

struct AnyResult {
  int hit;
  unsigned nodes, tests;
};

// Child references in a node record (written by the LBVH build):
//   >= 0          interior node index
//   leaf          0x80000000 | (count - 1) << 25 | first   (count <= 32, first < 2^25)
//   kDone (-1)    end of traversal (never stored in a node; bit 30 distinguishes it)
constexpr int kDone = -1;
__device__ __forceinline__ int leaf_first(int r) { return r & 0x01ffffff; }
__device__ __forceinline__ int leaf_count(int r) { return ((r >> 25) & 31) + 1; }

__device__ __forceinline__ void load_tri(const float4* __restrict__ tris, int p, f3& v1, f3& e1, f3& e2, int& id) {
  float4 a = __ldg(tris + 3 * (size_t)p);
  float4 b = __ldg(tris + 3 * (size_t)p + 1);
  float4 c = __ldg(tris + 3 * (size_t)p + 2);
  v1 = mk3(a.x, a.y, a.z);
  e1 = mk3(a.w, b.x, b.y);
  e2 = mk3(b.z, b.w, c.x);
  id = __float_as_int(c.y);
}

// ------------------------------------------------------------------ flat scenes
// Shared-memory accesses of the traversal stack by 32-bit address.  Each is one instruction
// under the predicate it depends on, so a node visit pushes its children without branches.
// What bounds a visit is instruction issue (and, once that fell, L1 wavefronts): with one
// branch per pushed child and a bound check per pop a visit's integer and control
// instructions outnumbered its box arithmetic.  Measured on the shadow rays of a 1080p view of
// 1.06M triangles (2.8M rays), branching form -> this one: 516 -> 411 M warp instructions,
// 662 -> 574 us; the same view's primary rays 231 -> 220 us.
__device__ __forceinline__ uint32_t shared_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void sts_ref(uint32_t a, int ref) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(ref));
}
__device__ __forceinline__ int lds_ref(uint32_t a) {
  int v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts_entry(uint32_t a, int ref, float t) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(a), "r"(ref), "f"(t));
}
__device__ __forceinline__ void lds_entry(uint32_t a, int& ref, float& t) {
  asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(ref), "=f"(t) : "r"(a));
}
// A visit's four children of a shadow ray (hit where tn <= tf), in slot order: `cur` takes
// the first hit one, the other hit ones are pushed, and with no hit the top entry is popped.
__device__ __forceinline__ void follow_hits(uint32_t& top, uint32_t stride, int& cur, const int4& ref,
                                            const float* tn, const float* tf) {
  asm volatile(
      "{\n.reg .pred p0, p1, p2, q1, q2, q3, a1, a2, a3;\n"
      "setp.le.f32 p0, %7, %11;\n"
      "setp.le.f32 p1, %8, %12;\n"
      "setp.le.f32 p2, %9, %13;\n"
      "and.pred q1, p1, p0;\n"
      "or.pred a1, p1, p0;\n"
      "and.pred q2, p2, a1;\n"
      "or.pred a2, p2, a1;\n"
      "setp.le.and.f32 q3, %10, %14, a2;\n"
      "setp.le.or.f32 a3, %10, %14, a2;\n"
      "@q1 add.u32 %0, %0, %2;\n@q1 st.shared.b32 [%0], %4;\n"
      "@q2 add.u32 %0, %0, %2;\n@q2 st.shared.b32 [%0], %5;\n"
      "@q3 add.u32 %0, %0, %2;\n@q3 st.shared.b32 [%0], %6;\n"
      "selp.b32 %1, %5, %6, p2;\n"
      "selp.b32 %1, %4, %1, p1;\n"
      "selp.b32 %1, %3, %1, p0;\n"
      "@!a3 ld.shared.b32 %1, [%0];\n@!a3 sub.u32 %0, %0, %2;\n}"
      : "+r"(top), "=&r"(cur)
      : "r"(stride), "r"(ref.x), "r"(ref.y), "r"(ref.z), "r"(ref.w), "f"(tn[0]), "f"(tn[1]), "f"(tn[2]), "f"(tn[3]),
        "f"(tf[0]), "f"(tf[1]), "f"(tf[2]), "f"(tf[3]));
}
// top += stride and store, where t < inf (nearest hit: a child box in reach).
__device__ __forceinline__ void push_if_near(uint32_t& top, uint32_t stride, int ref, float t) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.lt.f32 p, %3, 0f7F800000;\n@p add.u32 %0, %0, %1;\n"
      "@p st.shared.v2.b32 [%0], {%2, %3};\n}"
      : "+r"(top)
      : "r"(stride), "r"(ref), "f"(t));
}

// Traversal stack of a flat scene: a column of SH shared-memory entries (a child ref, and
// its entry distance with T), entry k at col + k * stride bytes.  Entry 0 is a sentinel --
// kDone, or kRefill when older entries lie in local memory -- so a pop needs no emptiness
// check.  When fewer than three entries are free, everything above the sentinel moves to
// local memory (at most CAP entries; CAP = SH is the small stack of the error-path test
// limit, eos_limits.small_stack: SH entries in all).  Shadow rays keep refs only, in 4-byte
// columns where their kernel traces nothing else: half the shared memory, and the rest of
// the SM's 256 KB is L1 (with 32 entries instead of 16 both stages lose about 10 %).  A
// kernel that traces both kinds keeps every thread inside its own 8-byte column, because
// lanes of one warp may be in different traversals.
constexpr int kRefill = (int)0xC0000002;
// Leaf refs as signed ints lie below kSpecial; kDone and kRefill in [kSpecial, 0).
constexpr int kSpecial = (int)0xC0000000;

template <int SH, int CAP, bool T>
struct ColumnStack {
  static_assert(SH >= 8, "a visit pushes up to three entries above the sentinel");
  static constexpr bool kSmall = CAP == SH;             // at most SH entries in all (test limit)
  static constexpr int kLocal = kSmall ? SH + 4 : CAP;  // entries of the local part
  uint32_t col, stride, top;
  int spilled;
  int ref_lo[kLocal];
  float t_lo[T ? kLocal : 1];
  __device__ __forceinline__ ColumnStack(uint32_t c, uint32_t s) : col(c), stride(s), top(c), spilled(0) {
    sentinel(kDone);
  }
  __device__ __forceinline__ void sentinel(int ref) {
    if (T) sts_entry(col, ref, -kInf);  // never beyond a limit
    else sts_ref(col, ref);
  }
  // Makes room for a visit's pushes; false when the local part is full too.
  __device__ __forceinline__ bool reserve() {
    if (top <= col + (SH - 4) * stride) return true;
#pragma unroll 1
    for (uint32_t a = col + stride; a <= top; a += stride) {
      if (spilled >= kLocal) return false;
      if (T) lds_entry(a, ref_lo[spilled], t_lo[spilled]);
      else ref_lo[spilled] = lds_ref(a);
      ++spilled;
    }
    top = col;
    sentinel(kRefill);
    return true;
  }
  // After a visit: false when the small stack's limit is passed.
  __device__ __forceinline__ bool within_limit() const {
    return !kSmall || (int)(top - col) <= (SH - spilled) * (int)stride;
  }
  // After a pop of kRefill: brings back the newest entries, half a column at most.
  __device__ __forceinline__ void refill() {
    const int n = min(spilled, (SH - 4) / 2);
    sentinel(spilled > n ? kRefill : kDone);
    top = col;
#pragma unroll 1
    for (int k = spilled - n; k < spilled; ++k) {
      top += stride;
      if (T) sts_entry(top, ref_lo[k], t_lo[k]);
      else sts_ref(top, ref_lo[k]);
    }
    spilled -= n;
  }
  __device__ __forceinline__ void push(int ref, float t) {
    top += stride;
    if (T) sts_entry(top, ref, t);
    else sts_ref(top, ref);
  }
  __device__ __forceinline__ int pop() {
    const int r = lds_ref(top);
    top -= stride;
    return r;
  }
  // The next entry whose box starts no later than `limit` (the sentinel's always does).
  __device__ __forceinline__ int pop_within(float limit) {
    int r;
    float t;
    do {
      lds_entry(top, r, t);
      top -= stride;
    } while (t > limit);
    return r;
  }
};

// Entry and exit distances of the four child boxes of a node record for a prepared ray.
// The fma form takes two children per instruction (fma.rn.f32x2: each half rounds as fmaf);
// 410 instead of 429 M warp instructions in the measurement above, at the same registers.
struct Box4 {
  float tn[4], tf[4];
};

// Address of node record `node`, whose chunk j lies at (address ^ 16 j): the record is
// 128-byte aligned and its chunks are stored swizzled by the low bits of its index (kNode
// record layout, eos_internal.cuh).
__device__ __forceinline__ size_t node_address(const float4* nodes, int node) {
  return (reinterpret_cast<size_t>(nodes) + (size_t)(uint32_t)node * 128u) ^ (((uint32_t)node & 7u) << 4);
}

__device__ __forceinline__ float4 ldg4(size_t a) { return __ldg(reinterpret_cast<const float4*>(a)); }

__device__ __forceinline__ Box4 child_boxes(size_t nd, const SlabRay& r) {
  const float4 lx = ldg4(nd ^ r.sx), ly = ldg4(nd ^ r.sy), lz = ldg4(nd ^ r.sz);  // near planes
  const float4 hx = ldg4(nd ^ r.sx ^ 48u), hy = ldg4(nd ^ r.sy ^ 80u), hz = ldg4(nd ^ r.sz ^ 112u);  // far planes
  Box4 b;
  slab_range(r, lx.x, ly.x, lz.x, hx.x, hy.x, hz.x, b.tn[0], b.tf[0]);
  slab_range(r, lx.y, ly.y, lz.y, hx.y, hy.y, hz.y, b.tn[1], b.tf[1]);
  slab_range(r, lx.z, ly.z, lz.z, hx.z, hy.z, hz.z, b.tn[2], b.tf[2]);
  slab_range(r, lx.w, ly.w, lz.w, hx.w, hy.w, hz.w, b.tn[3], b.tf[3]);
  return b;
}

typedef unsigned long long f2;  // two floats in a register pair
__device__ __forceinline__ f2 dup2(float v) {
  f2 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ f2 pack2(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ void axis4(float4 p, float i, float c, float* o) {
  unpack2(fma2(pack2(p.x, p.y), dup2(i), dup2(c)), o[0], o[1]);
  unpack2(fma2(pack2(p.z, p.w), dup2(i), dup2(c)), o[2], o[3]);
}

__device__ __forceinline__ Box4 child_boxes(size_t nd, const FmaSlabRay& r) {
  const float4 lx = ldg4(nd ^ r.sx), ly = ldg4(nd ^ r.sy), lz = ldg4(nd ^ r.sz);  // near planes
  const float4 hx = ldg4(nd ^ r.sx ^ 48u), hy = ldg4(nd ^ r.sy ^ 80u), hz = ldg4(nd ^ r.sz ^ 112u);  // far planes
  float x[4], y[4], z[4];
  Box4 b;
  axis4(lx, r.ix, r.nx, x);
  axis4(ly, r.iy, r.ny, y);
  axis4(lz, r.iz, r.nz, z);
#pragma unroll
  for (int i = 0; i < 4; ++i) b.tn[i] = fmaxf(max3f(x[i], y[i], z[i]), 0.0f);
  axis4(hx, r.ix, r.fx, x);
  axis4(hy, r.iy, r.fy, y);
  axis4(hz, r.iz, r.fz, z);
#pragma unroll
  for (int i = 0; i < 4; ++i) b.tf[i] = min3f(x[i], y[i], z[i]) * (1.0f + 0x1p-19f);
  return b;
}

// A visit's four children of a nearest-hit ray: those in reach (entry within the exit and
// the limit) sorted by entry distance (five compare-exchanges), the others but the nearest
// pushed farthest first; returns the nearest, or the next entry of the stack.
template <class Stack>
__device__ __forceinline__ int follow_nearest(Stack& st, const int4& ref, const Box4& b, float limit) {
  int c[4] = {ref.x, ref.y, ref.z, ref.w};
  float t[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) t[i] = b.tn[i] <= fminf(b.tf[i], limit) ? b.tn[i] : kInf;
#define EOS_CX(a, b)                 \
  if (t[b] < t[a]) {                 \
    float tt = t[a]; t[a] = t[b]; t[b] = tt; \
    int cc = c[a]; c[a] = c[b]; c[b] = cc;   \
  }
  EOS_CX(0, 1) EOS_CX(2, 3) EOS_CX(0, 2) EOS_CX(1, 3) EOS_CX(1, 2)
#undef EOS_CX
  push_if_near(st.top, st.stride, c[3], t[3]);
  push_if_near(st.top, st.stride, c[2], t[2]);
  push_if_near(st.top, st.stride, c[1], t[1]);
  return t[0] == kInf ? st.pop_within(limit) : c[0];
}

// Nearest hit.  Traversal in the two-loop form of Aila & Laine ("Understanding the
// efficiency of ray traversal on GPUs", HPG 2009): a lane that reaches a leaf parks it and
// keeps descending until every lane of the warp holds a leaf, then the lanes intersect
// their leaves together, so triangle tests run with full warps.
//
// A node visit tests the four child boxes of one 128-B record; an unused slot holds the box
// lo = +inf, hi = -inf: on every axis the near plane gives an entry of +inf and the far
// plane an exit of -inf, whatever the direction's sign (parallel axes fail the containment
// test), so both box tests reject it and no per-slot check is needed.  The hit children are
// sorted by entry distance (five compare-exchanges), pushed farthest first and the nearest
// popped again.
template <int SH, int CAP, class Ray>
__device__ __forceinline__ Hit closest_traverse(const DevScene& s, f3 o, f3 d, const Ray& r, uint32_t col,
                                               uint32_t stride, int* err) {
  constexpr float kCullR = RayCull<Ray>::k;
  Hit h;
  h.t = kInf; h.u = h.v = 0.0f; h.pos = -1; h.id = -1; h.nodes = 0; h.tests = 0;
  ColumnStack<SH, CAP, true> st(col, stride);
  int cur = 0;   // interior node, leaf ref, kRefill or kDone
  int leaf = 0;  // parked leaf (0 = none)
  for (;;) {
    while (cur >= 0) {
      size_t nd = node_address(s.nodes, cur);
      const int4 ref = __ldg(reinterpret_cast<const int4*>(nd ^ 96u));
      const Box4 b = child_boxes(nd, r);
      ++h.nodes;
      if (!st.reserve()) {
        atomicOr(err, kErrStack);
        return h;
      }
      cur = follow_nearest(st, ref, b, h.t * kCullR);
      if (!st.within_limit()) {
        atomicOr(err, kErrStack);
        return h;
      }
      if (cur < kSpecial && leaf == 0) {
        leaf = cur;
        cur = st.pop_within(h.t * kCullR);
      }
      if (!__any_sync(__activemask(), leaf == 0)) break;
    }
    if (cur < kSpecial && leaf == 0) {
      leaf = cur;
      cur = st.pop_within(h.t * kCullR);
    }
    while (leaf != 0) {
      const int cnt = leaf_count(leaf);
      int p = leaf_first(leaf);
      const int end = p + cnt;
      h.tests += cnt;
      do {
        f3 v1, e1, e2;
        int id;
        load_tri(s.tris, p, v1, e1, e2, id);
        float t, u, v;
        if (mt_intersect_fast(o, d, v1, e1, e2, t, u, v) && (t < h.t || (t == h.t && id > h.id))) {
          h.t = t; h.u = u; h.v = v; h.pos = p; h.id = id;
        }
      } while (++p < end);
      leaf = 0;
      if (cur < kSpecial) {
        leaf = cur;
        cur = st.pop_within(h.t * kCullR);
      }
    }
    if (cur == kDone) return h;
    if (cur == kRefill) {
      st.refill();
      cur = st.pop_within(h.t * kCullR);
    }
  }
}

template <int SH, int CAP = kStackMax>
__device__ __forceinline__ Hit closest_hit_body(const DevScene& s, f3 o, f3 d, uint32_t col, uint32_t stride,
                                                int* err) {
  const SlabRay r = make_slab(o, d);
  if (fma_slab_ok(r)) return closest_traverse<SH, CAP>(s, o, d, make_fma_slab(r), col, stride, err);
  return closest_traverse<SH, CAP>(s, o, d, r, col, stride, err);
}

// Any hit at t >= 0 (shadow rays), same two-loop form; returns at the first hit.  Children
// in slot order: nearest first measured slower for shadow rays.
template <int SH, int CAP, class Ray>
__device__ __forceinline__ AnyResult any_traverse(const DevScene& s, f3 o, f3 d, const Ray& r, uint32_t col,
                                                  uint32_t stride, int* err) {
  AnyResult res{0, 0u, 0u};
  ColumnStack<SH, CAP, false> st(col, stride);
  int cur = 0;
  int leaf = 0;
  for (;;) {
    while (cur >= 0) {
      size_t nd = node_address(s.nodes, cur);
      const int4 ref = __ldg(reinterpret_cast<const int4*>(nd ^ 96u));
      const Box4 b = child_boxes(nd, r);
      ++res.nodes;
      if (!st.reserve()) {
        atomicOr(err, kErrStack);
        return res;
      }
      follow_hits(st.top, stride, cur, ref, b.tn, b.tf);
      if (!st.within_limit()) {
        atomicOr(err, kErrStack);
        return res;
      }
      if (cur < kSpecial && leaf == 0) {
        leaf = cur;
        cur = st.pop();
      }
      if (!__any_sync(__activemask(), leaf == 0)) break;
    }
    if (cur < kSpecial && leaf == 0) {
      leaf = cur;
      cur = st.pop();
    }
    while (leaf != 0) {
      int p = leaf_first(leaf);
      const int end = p + leaf_count(leaf);
      do {
        f3 v1, e1, e2;
        int id;
        load_tri(s.tris, p, v1, e1, e2, id);
        float t, u, v;
        ++res.tests;
        if (mt_intersect_fast(o, d, v1, e1, e2, t, u, v)) {
          res.hit = 1;
          return res;
        }
      } while (++p < end);
      leaf = 0;
      if (cur < kSpecial) {
        leaf = cur;
        cur = st.pop();
      }
    }
    if (cur == kDone) return res;
    if (cur == kRefill) {
      st.refill();
      cur = st.pop();
    }
  }
}

template <int SH, int CAP = kStackMax>
__device__ __forceinline__ AnyResult any_hit_body(const DevScene& s, f3 o, f3 d, uint32_t col, uint32_t stride,
                                                  int* err) {
  const SlabRay r = make_slab(o, d);
  if (fma_slab_ok(r)) return any_traverse<SH, CAP>(s, o, d, make_fma_slab(r), col, stride, err);
  return any_traverse<SH, CAP>(s, o, d, r, col, stride, err);
}

// Out-of-line copies for kernels whose registers are set for two-level scenes.
template <int SH>
__device__ __noinline__ Hit closest_hit_call(const DevScene& s, f3 o, f3 d, uint32_t col, uint32_t stride, int* err) {
  return closest_hit_body<SH>(s, o, d, col, stride, err);
}
template <int SH>
__device__ __noinline__ AnyResult any_hit_call(const DevScene& s, f3 o, f3 d, uint32_t col, uint32_t stride, int* err) {
  return any_hit_body<SH>(s, o, d, col, stride, err);
}

// ------------------------------------------------------------------ two-level scenes
// A scene of instances (eos_scene_create_instanced): s.nodes is a tree over the instances'
// world boxes whose leaves each hold one instance; reaching one moves the ray into the
// instance's object space and continues in its mesh's tree.  A marker entry below the
// mesh's entries on the stack (t = -inf, so no limit drops it) brings the ray back.  t is
// the same parameter in both spaces (the direction is not renormalised), so one limit
// culls both levels.  Nearest-hit semantics as for a flat scene, with global ids.
constexpr int kExitMesh = (int)0xC0000001;

// o' = Minv [o, 1], d' = Minv [d, 0]; row r: ((m_r0 x + m_r1 y) + m_r2 z) (+ m_r3).
__device__ __forceinline__ void to_object(const DevInstance* I, f3 o, f3 d, f3& oo, f3& od) {
  const float4* m = reinterpret_cast<const float4*>(I->minv);
  const float4 a = __ldg(m), b = __ldg(m + 1), c = __ldg(m + 2);
  oo = mk3(((a.x * o.x + a.y * o.y) + a.z * o.z) + a.w, ((b.x * o.x + b.y * o.y) + b.z * o.z) + b.w,
           ((c.x * o.x + c.y * o.y) + c.z * o.z) + c.w);
  od = mk3((a.x * d.x + a.y * d.y) + a.z * d.z, (b.x * d.x + b.y * d.y) + b.z * d.z,
           (c.x * d.x + c.y * d.y) + c.z * d.z);
}

__device__ __forceinline__ bool prepare_ray(f3 o, f3 d, SlabRay& r) {
  r = make_slab(o, d);
  return true;
}
__device__ __forceinline__ bool prepare_ray(f3 o, f3 d, FmaSlabRay& r) {
  const SlabRay e = make_slab(o, d);
  r = make_fma_slab(e);
  return fma_slab_ok(e);
}

// ANY: returns at the first hit (h.pos >= 0 then); otherwise the nearest hit.  *ok: false when
// the ray, in world or some object space, needs the exact box test (Ray = FmaSlabRay only);
// the result is then unusable.  The world-space ray is prepared again on the way out of an
// instance rather than kept: its twelve registers would spill.
template <int SH, bool ANY, class Ray>
__device__ __forceinline__ Hit walk_instanced(const DevScene& s, f3 o, f3 d, uint32_t col, uint32_t stride, int* err,
                                              bool* ok) {
  constexpr float kCullR = RayCull<Ray>::k;
  Hit h;
  h.t = kInf; h.u = h.v = 0.0f; h.pos = -1; h.id = -1; h.nodes = 0; h.tests = 0;
  Ray r;
  *ok = prepare_ray(o, d, r);
  if (!*ok) return h;
  f3 oo = o, od = d;
  const float4* nodes = s.nodes;
  const float4* tris = nullptr;
  int id_off = 0;
  bool in_mesh = false;
  ColumnStack<SH, kStackMax, !ANY> st(col, stride);
  int cur = 0;
  for (;;) {
    if (cur >= 0) {
      size_t nd = node_address(nodes, cur);
      const int4 ref = __ldg(reinterpret_cast<const int4*>(nd ^ 96u));
      const Box4 b = child_boxes(nd, r);
      ++h.nodes;
      if (!st.reserve()) {
        atomicOr(err, kErrStack);
        return h;
      }
      if (ANY) follow_hits(st.top, stride, cur, ref, b.tn, b.tf);
      else cur = follow_nearest(st, ref, b, h.t * kCullR);
      continue;
    }
    if (cur == kDone) return h;
    if (cur == kExitMesh) {  // back to the instance tree
      prepare_ray(o, d, r);
      nodes = s.nodes;
      in_mesh = false;
    } else if (cur == kRefill) {
      st.refill();
    } else if (!in_mesh) {  // an instance: continue in its mesh, in object space
      const DevInstance* I = s.inst + leaf_first(cur);
      to_object(I, o, d, oo, od);
      *ok = prepare_ray(oo, od, r);
      if (!*ok) return h;
      nodes = I->nodes;
      tris = I->tris;
      id_off = I->id_offset;
      if (!st.reserve()) {
        atomicOr(err, kErrStack);
        return h;
      }
      st.push(kExitMesh, -kInf);
      in_mesh = true;
      cur = 0;
      continue;
    } else {  // a leaf of the mesh
      const int first = leaf_first(cur), cnt = leaf_count(cur);
      for (int p = first; p < first + cnt; ++p) {
        f3 v1, e1, e2;
        int id;
        load_tri(tris, p, v1, e1, e2, id);
        float t, u, v;
        ++h.tests;
        if (!mt_intersect_fast(oo, od, v1, e1, e2, t, u, v)) continue;
        const int gid = id_off + id;
        if (ANY) {
          h.t = t; h.u = u; h.v = v; h.pos = p; h.id = gid;
          return h;
        }
        if (t < h.t || (t == h.t && gid > h.id)) {
          h.t = t; h.u = u; h.v = v; h.pos = p; h.id = gid;
        }
      }
    }
    cur = ANY ? st.pop() : st.pop_within(h.t * kCullR);
  }
}

template <int SH, bool ANY>
__device__ __noinline__ Hit walk_instanced_exact(const DevScene& s, f3 o, f3 d, uint32_t col, uint32_t stride,
                                                 int* err) {
  bool ok;
  return walk_instanced<SH, ANY, SlabRay>(s, o, d, col, stride, err, &ok);
}

// In the fma box test's form; the rare ray that needs the exact one starts again in that.
// (Carrying both forms with a branch per visit cost 13 %; the exact form alone 10 % more than
// this: 1080p view of 801 instances 12.1 -> 10.9 ms with the traversal inline.  Letting lanes
// descend until all hold a leaf is slower, 10.1 -> 11.7: lanes change space at each instance.)
template <int SH, bool ANY>
__device__ __forceinline__ Hit traverse_instanced(const DevScene& s, f3 o, f3 d, uint32_t col, uint32_t stride,
                                               int* err) {
  bool ok;
  const Hit h = walk_instanced<SH, ANY, FmaSlabRay>(s, o, d, col, stride, err, &ok);
  return ok ? h : walk_instanced_exact<SH, ANY>(s, o, d, col, stride, err);
}

// Instance holding global triangle id `gid` (instances in id order).
__device__ __forceinline__ const DevInstance* instance_of(const DevScene& s, int gid) {
  int lo = 0, hi = s.n_inst - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(&s.inst[mid].id_offset) <= gid) lo = mid;
    else hi = mid - 1;
  }
  return s.inst + lo;
}

// How a kernel holds the traversals: kFlat the flat one inline and none for two-level scenes,
// kTwoLevel the two-level one inline and the flat one out of line (a pass may hold both kinds
// of scenes).  CAP (inline traversals of flat scenes): total stack entries, see ColumnStack.
enum TraversalForm { kFlat, kTwoLevel };

template <int SH, TraversalForm F, int CAP = kStackMax>
__device__ __forceinline__ Hit closest_hit(const DevScene& s, f3 o, f3 d, uint32_t col, uint32_t stride, int* err) {
  if constexpr (F == kTwoLevel)
    if (s.inst) return traverse_instanced<SH, false>(s, o, d, col, stride, err);
  if constexpr (F == kFlat || CAP == SH) return closest_hit_body<SH, CAP>(s, o, d, col, stride, err);
  else return closest_hit_call<SH>(s, o, d, col, stride, err);
}

template <int SH, TraversalForm F, int CAP = kStackMax>
__device__ __forceinline__ AnyResult any_hit(const DevScene& s, f3 o, f3 d, uint32_t col, uint32_t stride, int* err) {
  if constexpr (F == kTwoLevel)
    if (s.inst) {
      const Hit h = traverse_instanced<SH, true>(s, o, d, col, stride, err);
      return AnyResult{h.pos >= 0 ? 1 : 0, h.nodes, h.tests};
    }
  if constexpr (F == kFlat || CAP == SH) return any_hit_body<SH, CAP>(s, o, d, col, stride, err);
  else return any_hit_call<SH>(s, o, d, col, stride, err);
}

// Traversal work counters, reduced per warp into the context's counter block:
// [3] interior nodes fetched by nearest-hit rays, [4] their triangle tests,
// [5] nodes fetched by shadow rays, [6] their triangle tests, [7] shaded hits.
enum { kCntPrimary = 0, kCntShadow = 1, kCntSecondary = 2, kCntNodesC = 3, kCntTestsC = 4, kCntNodesA = 5,
       kCntTestsA = 6, kCntHits = 7, kNumCounts = 8 };

__device__ __forceinline__ void warp_add_count(unsigned long long* dst, unsigned long long v) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(dst, v);
}

// ------------------------------------------------------------------ shading
// Hit point o + t*d and the shading normal normalize(n1(1-u-v) + n2 u + n3 v), normalised
// once more as the reference does after its (identity) world transform
// (src/Triangle.cpp:41-46, src/BVH.cpp:373-380).
__device__ __forceinline__ void hit_geometry(const DevScene& s, f3 o, f3 d, const Hit& h, f3& P, f3& N, int& obj) {
  P = add3(o, scale3(h.t, d));
  const DevInstance* I = s.inst ? instance_of(s, h.id) : nullptr;
  const float4* sr = (I ? I->shade : s.shade) + 3 * (size_t)h.pos;
  float4 a = __ldg(sr), b = __ldg(sr + 1), c = __ldg(sr + 2);
  f3 n1 = mk3(a.x, a.y, a.z), n2 = mk3(a.w, b.x, b.y), n3 = mk3(b.z, b.w, c.x);
  obj = __float_as_int(c.y);
  float w = (1.0f - h.u) - h.v;
  f3 n = norm3(add3(add3(scale3(w, n1), scale3(h.u, n2)), scale3(h.v, n3)));
  if (I) {  // normal to world space: Minv^T n, column c of Minv: ((m_0c n.x + m_1c n.y) + m_2c n.z)
    const float* m = I->minv;
    n = mk3((__ldg(m + 0) * n.x + __ldg(m + 4) * n.y) + __ldg(m + 8) * n.z,
            (__ldg(m + 1) * n.x + __ldg(m + 5) * n.y) + __ldg(m + 9) * n.z,
            (__ldg(m + 2) * n.x + __ldg(m + 6) * n.y) + __ldg(m + 10) * n.z);
    obj += I->mat_base;
  }
  N = norm3(n);
}

// Replay of a recorded hit (the adjoint): the hit of global triangle `id` for ray (o, d),
// through the same exact-order test as the traversal (in the instance's object space for a
// two-level scene), so t, u, v and the sorted position equal the forward pass's.  False if
// the triangle does not take the ray (a record from another scene or camera).
__device__ __forceinline__ bool hit_of_id(const DevScene& s, f3 o, f3 d, int id, Hit& h) {
  const float4* tris = s.tris;
  const int32_t* pos = s.pos_of_id;
  int local = id;
  f3 oo = o, od = d;
  if (s.inst) {
    const DevInstance* I = instance_of(s, id);
    to_object(I, o, d, oo, od);
    tris = I->tris;
    pos = I->pos_of_id;
    local = id - I->id_offset;
  }
  h.id = id;
  h.pos = pos[local];
  f3 v1, e1, e2;
  int rid;
  load_tri(tris, h.pos, v1, e1, e2, rid);
  return mt_intersect(oo, od, v1, e1, e2, h.t, h.u, h.v);
}

// RayTracer::calcPhong + findDiffuseColor for one light (src/RayTracer.cpp:418-458):
// diffuse max(0, L.N) kd Lc, specular [V.R > 0] pow(V.R, shininess) Lc ks with
// R = normalize(2 (N.L) N - L) and V towards the camera position.
__device__ __forceinline__ f3 phong_light(const float* m, const float* l, f3 P, f3 N, f3 cam) {
  f3 L = norm3(sub3(mk3(l[0], l[1], l[2]), P));
  f3 V = norm3(sub3(cam, P));
  float ndl = dot3(N, L);
  float two = 2.0f * ndl;
  f3 R = norm3(sub3(scale3(two, N), L));
  float dd = dot3(L, N);
  dd = dd > 0.0f ? dd : 0.0f;
  f3 diff = mk3((dd * m[0]) * l[3], (dd * m[1]) * l[4], (dd * m[2]) * l[5]);
  float vr = dot3(V, R);
  if (vr > 0.0f) {
    float st = powf(vr, m[6]);
    return add3(diff, mk3((st * l[3]) * m[3], (st * l[4]) * m[4], (st * l[5]) * m[5]));
  }
  return diff;
}

// RayTracer::fresnel (src/RayTracer.cpp:52-64, after Bram de Greve 2006), in its float
// order: reflectance of an interface n1 -> n2 for a unit incident direction and the normal
// on the incident side; 1 under total internal reflection.
__device__ __forceinline__ float fresnel(f3 incident, f3 normal, float n1, float n2) {
  const float n = n1 / n2;
  const float cos_i = -dot3(normal, incident);
  const float sin_t2 = (n * n) * (1.0f - cos_i * cos_i);
  if (sin_t2 > 1.0f) return 1.0f;
  const float cos_t = sqrtf(1.0f - sin_t2);
  const float r_orth = (n1 * cos_i - n2 * cos_t) / (n1 * cos_i + n2 * cos_t);
  const float r_par = (n2 * cos_i - n1 * cos_t) / (n2 * cos_i + n1 * cos_t);
  return (r_orth * r_orth + r_par * r_par) / 2.0f;
}

// Secondary ray of a hit with material m (RayTracer::shadeIntersection,
// src/RayTracer.cpp:329-407).  Reflective: the mirror ray from P + 1e-3 R, weight =
// reflectivity.  Transparent: the reference computes the Fresnel weight K and traces the
// mirror ray about the incident-side normal from P + 1e-3 n -- twice, as "reflected" and,
// by a slip at :403, again as "refracted" -- and mixes K c + (1 - K) c; the refracted ray
// itself is never traced.  That ray once, with w = -K: the sign bit marks the mix.
// Returns false when the material spawns no ray.
// The mirror ray of a reflective hit: normalize(reflect(d, N)) from P + 1e-3 of it (:339-351).
__device__ __forceinline__ void mirror_ray(f3 d, f3 P, f3 N, f3& ro, f3& rd) {
  rd = norm3(reflect3(d, N));
  ro = add3(P, scale3(kRayEps, rd));
}

// The ray of a transparent hit (:353-407) and its Fresnel weight K.
__device__ __forceinline__ float transparent_ray(const float* m, float ambient, f3 d, f3 P, f3 N, f3& ro, f3& rd) {
  const f3 inc = norm3(d);
  f3 n = N;
  float n1 = ambient, n2 = m[9];
  if (!(dot3(inc, N) < 0.0f)) {  // leaving the material: normal flipped as 0 - N
    n1 = m[9];
    n2 = ambient;
    n = sub3(mk3(0.0f, 0.0f, 0.0f), N);
  }
  const float K = fresnel(inc, n, n1, n2);
  rd = norm3(reflect3(d, n));
  ro = add3(P, scale3(kRayEps, n));
  return K;
}

__device__ __forceinline__ bool secondary_ray(const float* m, float ambient, f3 d, f3 P, f3 N, f3& ro, f3& rd,
                                              float& w) {
  if (m[7] > 0.0f) {
    mirror_ray(d, P, N, ro, rd);
    w = m[7];
    return true;
  }
  if (m[8] > 0.0f) {
    w = -transparent_ray(m, ambient, d, P, N, ro, rd);
    return true;
  }
  w = 0.0f;
  return false;
}

// Colour of a ray-tree node (a material that is both reflective and transparent traces
// both rays, src/RayTracer.cpp:339-407) as :410 sums it: (phong + wR c_mirror) +
// (K c_t + (1 - K) c_t); a term the material lacks is 0 (wR = 0, has_t false), a child not
// traced (beyond the trace depth, or a miss) has colour 0.  For a node with one secondary
// ray this equals fold_colour bit for bit (x + 0 = x for the non-negative sums here).
__device__ __forceinline__ f3 tree_colour(f3 phong, float wR, f3 cR, bool has_t, float K, f3 cT) {
  const f3 refr = has_t ? add3(scale3(K, cT), scale3(1.0f - K, cT)) : mk3(0.0f, 0.0f, 0.0f);
  return add3(add3(phong, scale3(wR, cR)), refr);
}

// Colour fold of one bounce: phong + w c for a mirror (or no) bounce; for a transparent
// one (sign bit of w set, K = -w) (phong + 0) + (K c + (1 - K) c) as the reference sums it.
__device__ __forceinline__ f3 fold_colour(f3 phong, float w, f3 c) {
  if (signbit(w)) {
    const float K = -w, L = 1.0f - K;
    return add3(phong, add3(scale3(K, c), scale3(L, c)));
  }
  return add3(phong, scale3(w, c));
}

// Weight of the next bounce's colour in the adjoint: d(fold)/dc.
__device__ __forceinline__ float fold_weight(float w) { return signbit(w) ? (-w) + (1.0f - (-w)) : w; }

// 8-bit quantisation of src/RayTracer.cpp:150-153: floor(c == 1 ? 255 : min(256 c, 255)).
// 256*c, the min and the floor are exact in float, so the float form matches the
// reference's double arithmetic bit for bit.
__device__ __forceinline__ uint8_t quantize(float c) {
  float q = c == 1.0f ? 255.0f : fminf(c * 256.0f, 255.0f);
  q = floorf(q);
  return (uint8_t)(q > 0.0f ? q : 0.0f);
}

}  // namespace eos
