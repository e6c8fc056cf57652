// GPU BVH build: Morton codes -> stable radix sort -> hierarchy (Karras radix tree, or
// PLOC clustering in ploc.cu) -> refit (LBVH; PLOC makes its boxes as it merges) -> 128-byte
// node records (4-wide, or 2 children per record) / 48-byte triangle records.
//
// Replaces the reference's CPU top-down median/SAH build (src/BVH.cpp:97-111,549-606) and
// its SoA upload (src/cudaStructures.cu:36-174,274-405).  The Morton encoder is the
// reference's 30-bit EncodeMorton3 (src/morton.h:45-48); the centroid is the reference
// triangle centroid ((v1 + v2) + v3) / 3 (src/Triangle.h:37), quantised per axis over the
// centroid bounds as q = min(1023, (uint)((1024 * (c - lo)) / (hi - lo))).
// Primitive order = stable sort by (code, triangle id).
#include <algorithm>

#include "eos_internal.cuh"
#include "ring.cuh"
#include "scan.cuh"
#include "tree.cuh"

namespace eos {
namespace {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;  // keys per block
constexpr int kRadixBits = 10;  // the 30-bit codes in three passes
constexpr int kRadix = 1 << kRadixBits;

__device__ __forceinline__ uint32_t float_to_ordered(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ordered_to_float(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__device__ __forceinline__ f3 load_vert(const float* v, uint32_t i) {
  return mk3(v[3 * (size_t)i], v[3 * (size_t)i + 1], v[3 * (size_t)i + 2]);
}

// Centroids and their bounds.  bounds: [6] ordered uints (min xyz, max xyz).
__global__ void k_centroids(const float* __restrict__ verts, uint32_t n_verts,
                            const uint32_t* __restrict__ tris, int n, float4* __restrict__ cent,
                            uint32_t* __restrict__ bounds, int* err) {
  float lo[3] = {kInf, kInf, kInf}, hi[3] = {-kInf, -kInf, -kInf};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t a = tris[3 * (size_t)i], b = tris[3 * (size_t)i + 1], c = tris[3 * (size_t)i + 2];
    if (a >= n_verts || b >= n_verts || c >= n_verts) {
      atomicOr(err, kErrIndex);
      a = b = c = 0;
    }
    f3 s = add3(add3(load_vert(verts, a), load_vert(verts, b)), load_vert(verts, c));
    f3 m = mk3(s.x / 3.0f, s.y / 3.0f, s.z / 3.0f);
    cent[i] = make_float4(m.x, m.y, m.z, 0.0f);
    lo[0] = fminf(lo[0], m.x); lo[1] = fminf(lo[1], m.y); lo[2] = fminf(lo[2], m.z);
    hi[0] = fmaxf(hi[0], m.x); hi[1] = fmaxf(hi[1], m.y); hi[2] = fmaxf(hi[2], m.z);
  }
  for (int k = 0; k < 3; ++k) {
    for (int off = 16; off > 0; off >>= 1) {
      lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], off));
      hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], off));
    }
  }
  // one atomic per block and bound: a warp's six atomics on the same six words were most of
  // the kernel's time (1.06M triangles: 43 us)
  __shared__ uint32_t s[6];
  if (threadIdx.x < 6) s[threadIdx.x] = threadIdx.x < 3 ? 0xffffffffu : 0u;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    for (int k = 0; k < 3; ++k) {
      if (lo[k] <= hi[k]) {
        atomicMin(&s[k], float_to_ordered(lo[k]));
        atomicMax(&s[3 + k], float_to_ordered(hi[k]));
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < 3) atomicMin(&bounds[threadIdx.x], s[threadIdx.x]);
  else if (threadIdx.x < 6) atomicMax(&bounds[threadIdx.x], s[threadIdx.x]);
}

// Morton codes of one tile and, as k_sort_hist, the tile's counts of the first pass's digit.
__global__ void __launch_bounds__(kSortThreads) k_morton(const float4* __restrict__ cent, int n,
                                                         const uint32_t* __restrict__ bounds,
                                                         uint32_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                                         uint32_t* __restrict__ counts, int n_tiles) {
  __shared__ uint32_t h[kRadix];
  for (int i = threadIdx.x; i < kRadix; i += kSortThreads) h[i] = 0;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const int i = blockIdx.x * kSortTile + r * kSortThreads + threadIdx.x;
    if (i >= n) break;
    float4 c = cent[i];
    float cc[3] = {c.x, c.y, c.z};
    uint32_t q[3];
    for (int k = 0; k < 3; ++k) {
      float lo = ordered_to_float(bounds[k]);
      float hi = ordered_to_float(bounds[3 + k]);
      float ext = hi - lo;
      if (ext > 0.0f) {
        float f = (1024.0f * (cc[k] - lo)) / ext;
        uint32_t u = (uint32_t)f;
        q[k] = u > 1023u ? 1023u : u;
      } else {
        q[k] = 0u;
      }
    }
    const uint32_t key = morton3(q[0], q[1], q[2]);
    keys[i] = key;
    vals[i] = (uint32_t)i;
    atomicAdd(&h[key & (kRadix - 1)], 1u);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < kRadix; d += kSortThreads) counts[(size_t)d * n_tiles + blockIdx.x] = h[d];
}

// ------------------------------------------------------------------ stable LSD radix sort
// Three passes of ten bits: per-tile digit counts (of the first pass: k_morton) -> per-digit
// exclusive scan over the tiles -> stable scatter, which scans the digit totals itself.
// Inside a tile, warp w owns keys [w*256, w*256+256) in 8 rounds of 32; peers with the same
// digit are found with __match_any_sync and ranked with popc, so the scatter keeps the input
// order (stability gives the (code, id) order).  Small sorts are bound by launches: nine
// with the codes, where four passes of eight bits with a scan of their own took seventeen.
__global__ void __launch_bounds__(kSortThreads) k_sort_hist(const uint32_t* __restrict__ keys, int n, int shift,
                                                            uint32_t* __restrict__ counts, int n_tiles) {
  __shared__ uint32_t h[kRadix];
  uint32_t key[kSortItems];
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const int i = blockIdx.x * kSortTile + r * kSortThreads + threadIdx.x;
    key[r] = i < n ? keys[i] : 0u;
  }
  for (int i = threadIdx.x; i < kRadix; i += kSortThreads) h[i] = 0;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortItems; ++r)
    if (blockIdx.x * kSortTile + r * kSortThreads + threadIdx.x < n) atomicAdd(&h[(key[r] >> shift) & (kRadix - 1)], 1u);
  __syncthreads();
  for (int d = threadIdx.x; d < kRadix; d += kSortThreads) counts[(size_t)d * n_tiles + blockIdx.x] = h[d];
}

// One warp per digit: exclusive scan of that digit's per-tile counts (in place), and its total.
__global__ void __launch_bounds__(kSortThreads) k_sort_scan_rows(uint32_t* __restrict__ counts, int n_tiles,
                                                                 uint32_t* __restrict__ totals) {
  const int lane = threadIdx.x & 31, digit = (blockIdx.x * kSortThreads + threadIdx.x) >> 5;
  uint32_t* row = counts + (size_t)digit * n_tiles;
  uint32_t carry = 0;
  for (int b = 0; b < n_tiles; b += 128) {  // four loads in flight
    uint32_t v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = b + 32 * k + lane;
      v[k] = i < n_tiles ? row[i] : 0u;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = b + 32 * k + lane;
      const uint32_t incl = warp_inclusive_scan(v[k]);
      if (i < n_tiles) row[i] = carry + incl - v[k];
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
  if (lane == 0) totals[digit] = carry;
}

__global__ void __launch_bounds__(kSortThreads) k_sort_scatter(
    const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin, uint32_t* __restrict__ kout,
    uint32_t* __restrict__ vout, int n, int shift, const uint32_t* __restrict__ counts, int n_tiles,
    const uint32_t* __restrict__ totals) {
  constexpr int kWarps = kSortThreads / 32, kPer = kRadix / kSortThreads;
  __shared__ uint32_t wh[kWarps][kRadix];
  __shared__ uint32_t tile_base[kRadix];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t lt_mask = (1u << lane) - 1u;
  uint32_t key[kSortItems], val[kSortItems], local[kSortItems];
  const int base = blockIdx.x * kSortTile + w * 32 * kSortItems;
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const int idx = base + r * 32 + lane;
    key[r] = idx < n ? kin[idx] : 0u;
    val[r] = idx < n ? vin[idx] : 0u;
  }
  // each thread's kPer consecutive digits: scan of the totals + this tile's place in each
  uint32_t sum = 0, mine[kPer];
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    mine[k] = totals[kPer * threadIdx.x + k];
    sum += mine[k];
  }
  for (int i = threadIdx.x; i < kWarps * kRadix; i += kSortThreads) (&wh[0][0])[i] = 0;
  uint32_t all;
  uint32_t before = block_exclusive_scan(sum, all);
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int d = kPer * threadIdx.x + k;
    tile_base[d] = before + counts[(size_t)d * n_tiles + blockIdx.x];
    before += mine[k];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const bool valid = base + r * 32 + lane < n;
    const uint32_t digit = valid ? ((key[r] >> shift) & (kRadix - 1)) : (uint32_t)kRadix + lane;
    const uint32_t peers = __match_any_sync(0xffffffffu, digit);
    const uint32_t rank = __popc(peers & lt_mask);
    const uint32_t pre = valid ? wh[w][digit] : 0u;
    __syncwarp();
    if (valid && rank == 0) wh[w][digit] = pre + __popc(peers);
    __syncwarp();
    local[r] = pre + rank;
  }
  __syncthreads();
  for (int d = threadIdx.x; d < kRadix; d += kSortThreads) {
    uint32_t s = tile_base[d];
#pragma unroll
    for (int ww = 0; ww < kWarps; ++ww) {
      const uint32_t t = wh[ww][d];
      wh[ww][d] = s;
      s += t;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    if (base + r * 32 + lane < n) {
      const uint32_t pos = wh[w][(key[r] >> shift) & (kRadix - 1)] + local[r];
      kout[pos] = key[r];
      vout[pos] = val[r];
    }
  }
}

// ------------------------------------------------------------------ Karras hierarchy
__device__ __forceinline__ int common_prefix(const uint32_t* __restrict__ k, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  uint32_t a = k[i], b = k[j];
  if (a == b) return 32 + __clz((uint32_t)(i ^ j));
  return __clz(a ^ b);
}

// Internal node i of n-1 (Karras 2012, "Maximizing parallelism in the construction of
// BVHs, octrees and k-d trees").  Node numbering: interior 0..n-2, leaf p -> n-1+p.
__global__ void k_karras(const uint32_t* __restrict__ k, int n, int2* __restrict__ child,
                         int* __restrict__ first_of, int* __restrict__ count, int* __restrict__ parent) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  int d = (common_prefix(k, n, i, i + 1) - common_prefix(k, n, i, i - 1)) >= 0 ? 1 : -1;
  int dmin = common_prefix(k, n, i, i - d);
  int lmax = 2;
  while (common_prefix(k, n, i, i + lmax * d) > dmin) lmax <<= 1;
  int l = 0;
  for (int t = lmax >> 1; t >= 1; t >>= 1)
    if (common_prefix(k, n, i, i + (l + t) * d) > dmin) l += t;
  int j = i + l * d;
  int dnode = common_prefix(k, n, i, j);
  int s = 0;
  int t = l;
  do {
    t = (t + 1) >> 1;
    if (common_prefix(k, n, i, i + (s + t) * d) > dnode) s += t;
  } while (t > 1);
  int gamma = i + s * d + min(d, 0);
  int first = min(i, j), last = max(i, j);
  int left = (first == gamma) ? (n - 1 + gamma) : gamma;
  int right = (last == gamma + 1) ? (n - 1 + gamma + 1) : gamma + 1;
  child[i] = make_int2(left, right);
  first_of[i] = first;
  count[i] = last - first + 1;
  parent[left] = i;
  parent[right] = i;
}

// Box of a triangle; .w: SAH cost of one triangle, leaf flag.
__device__ __forceinline__ void triangle_box(f3 v1, f3 v2, f3 v3, float4& lo, float4& hi) {
  lo = make_float4(fminf(fminf(v1.x, v2.x), v3.x), fminf(fminf(v1.y, v2.y), v3.y), fminf(fminf(v1.z, v2.z), v3.z),
                   1.0f);
  hi = make_float4(fmaxf(fmaxf(v1.x, v2.x), v3.x), fmaxf(fmaxf(v1.y, v2.y), v3.y), fmaxf(fmaxf(v1.z, v2.z), v3.z),
                   1.0f);
}

// Leaf boxes in Morton order (the PLOC builder's input; its records come after the tree,
// in the tree's leaf order).
__global__ void k_leaf_boxes(const float* __restrict__ verts, uint32_t n_verts, const uint32_t* __restrict__ tris,
                             const uint32_t* __restrict__ order, int n, float4* __restrict__ blo,
                             float4* __restrict__ bhi) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n) return;
  const uint32_t id = order[m];
  uint32_t a = tris[3 * (size_t)id], b = tris[3 * (size_t)id + 1], c = tris[3 * (size_t)id + 2];
  if (a >= n_verts || b >= n_verts || c >= n_verts) a = b = c = 0;  // flagged in k_centroids
  triangle_box(load_vert(verts, a), load_vert(verts, b), load_vert(verts, c), blo[n - 1 + m], bhi[n - 1 + m]);
}

// Triangle records, id -> position map and (blo not NULL) leaf boxes.  The triangle at Morton
// position m goes to record position p = perm[m] (perm NULL: p = m).
__global__ void k_records(const float* __restrict__ verts, const float* __restrict__ normals, uint32_t n_verts,
                          const uint32_t* __restrict__ tris, const uint32_t* __restrict__ obj,
                          const uint32_t* __restrict__ order, const uint32_t* __restrict__ perm, int n, uint32_t n_obj,
                          float4* __restrict__ trec, float4* __restrict__ srec, int32_t* __restrict__ pos_of_id,
                          float4* __restrict__ blo, float4* __restrict__ bhi, int* err) {
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n) return;
  uint32_t id = order[m];
  const int p = perm ? (int)perm[m] : m;
  uint32_t a = tris[3 * (size_t)id], b = tris[3 * (size_t)id + 1], c = tris[3 * (size_t)id + 2];
  if (a >= n_verts || b >= n_verts || c >= n_verts) a = b = c = 0;  // flagged in k_centroids
  f3 v1 = load_vert(verts, a), v2 = load_vert(verts, b), v3 = load_vert(verts, c);
  f3 e1 = sub3(v2, v1), e2 = sub3(v3, v1);
  trec[3 * (size_t)p] = make_float4(v1.x, v1.y, v1.z, e1.x);
  trec[3 * (size_t)p + 1] = make_float4(e1.y, e1.z, e2.x, e2.y);
  trec[3 * (size_t)p + 2] = make_float4(e2.z, __int_as_float((int)id), 0.0f, 0.0f);
  f3 n1 = load_vert(normals, a), n2 = load_vert(normals, b), n3 = load_vert(normals, c);
  srec[3 * (size_t)p] = make_float4(n1.x, n1.y, n1.z, n2.x);
  srec[3 * (size_t)p + 1] = make_float4(n2.y, n2.z, n3.x, n3.y);
  uint32_t ob = obj[id];
  if (ob >= n_obj) {
    atomicOr(err, kErrIndex);
    ob = 0;
  }
  srec[3 * (size_t)p + 2] = make_float4(n3.z, __int_as_float((int)ob), 0.0f, 0.0f);
  pos_of_id[id] = p;
  if (blo) triangle_box(v1, v2, v3, blo[n - 1 + p], bhi[n - 1 + p]);
}

// Leaf reference: 0x80000000 | (count - 1) << 25 | first  (count <= 32, first < 2^25).
__host__ __device__ __forceinline__ int pack_leaf(int first, int count) {
  return (int)(0x80000000u | ((uint32_t)(count - 1) << 25) | (uint32_t)first);
}

// Bottom-up refit: one thread per leaf walks to the root; the second thread to reach an
// interior node merges the two child boxes and decides whether the subtree becomes one
// leaf (join_boxes; node records are written afterwards by the wide conversion).  Bounded
// walk: the tree depth is at most kStackMax.
__global__ void k_refit(int n, const int2* __restrict__ child, const int* __restrict__ count,
                        const int* __restrict__ parent, float4* blo, float4* bhi, int* __restrict__ arrive,
                        int max_leaf, int sah, int* err) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  int node = parent[n - 1 + p];
  for (int step = 0; node >= 0; ++step) {
    if (step > kStackMax) {
      atomicOr(err, kErrDepth);
      return;
    }
    __threadfence();
    if (atomicAdd(&arrive[node], 1) == 0) return;
    __threadfence();
    int2 c = child[node];
    float4 lo, hi;
    join_boxes(__ldcg(&blo[c.x]), __ldcg(&bhi[c.x]), __ldcg(&blo[c.y]), __ldcg(&bhi[c.y]), count[node], max_leaf, sah,
               lo, hi);
    blo[node] = lo;
    bhi[node] = hi;
    node = parent[node];
  }
}

// ------------------------------------------------------------------ node records
// Every node record has four child slots.  A node is made from one binary node by
// replacing its interior child of largest surface area by that child's two children until
// it has `max_children` children (4 for the 4-wide layout, 2 for the binary one) or only
// leaves (one-triangle leaves and collapsed subtrees stay leaves).  Top-down, one launch
// per level (k_wide_level).
//
// Record, 128 B = 8 x float4 (structure of arrays over the four slots; node_chunk order):
//   [0] lo.x[4] [1] lo.y[4] [2] lo.z[4] [3] hi.x[4] [4] hi.y[4] [5] hi.z[4]
//   [6] ref[4]: interior record index, packed leaf, or kEmptyRef for an unused slot
//       (whose box is lo = +inf, hi = -inf: every slab test misses it, so the traversal
//       needs no per-slot check)
//   [7] count[4]: triangles of a leaf, 0 for an interior child, -1 for an unused slot
constexpr int kEmptyRef = (int)0xC0000000;

__device__ __forceinline__ void write_record(float4* nodes, int n, const float (&v)[6][4], const int (&ref)[4],
                                             const int (&cnt)[4]) {
  float4* o = nodes + 8 * (size_t)n;
#pragma unroll
  for (int a = 0; a < 6; ++a) o[node_chunk(n, a)] = make_float4(v[a][0], v[a][1], v[a][2], v[a][3]);
  o[node_chunk(n, 6)] = make_float4(__int_as_float(ref[0]), __int_as_float(ref[1]), __int_as_float(ref[2]), __int_as_float(ref[3]));
  o[node_chunk(n, 7)] = make_float4(__int_as_float(cnt[0]), __int_as_float(cnt[1]), __int_as_float(cnt[2]), __int_as_float(cnt[3]));
}

// Greedy opening of one binary node: its children, then the children of the largest-area
// interior child until max_children are reached; returns how many of them get records of
// their own.
__device__ __forceinline__ int wide_select_one(int n, const int2* __restrict__ child, const float4* __restrict__ blo,
                                               const float4* __restrict__ bhi, int node, int max_children, int* c,
                                               float4* lo, float4* hi) {
  // a child's own children are read along with its box, before it is known whether it is
  // opened: one dependent read per opening instead of two
  int2 sub[4];
  auto take = [&](int i, int ci) {
    c[i] = ci;
    lo[i] = blo[ci];
    hi[i] = bhi[ci];
    sub[i] = ci < n - 1 ? child[ci] : make_int2(-1, -1);
  };
  const int2 ch = child[node];
  take(0, ch.x);
  take(1, ch.y);
  c[2] = c[3] = -1;
#pragma unroll
  for (int k = 2; k < 4; ++k) {
    if (k >= max_children) break;
    int best = -1;
    float best_area = -1.0f;
#pragma unroll
    for (int i = 0; i < k; ++i) {
      if (c[i] >= n - 1 || hi[i].w != 0.0f) continue;  // triangle or collapsed subtree: a leaf
      const float a = half_area(lo[i], hi[i]);
      if (a > best_area) {
        best_area = a;
        best = i;
      }
    }
    if (best < 0) break;
    int2 g = make_int2(0, 0);
#pragma unroll
    for (int i = 0; i < k; ++i)
      if (i == best) g = sub[i];
#pragma unroll
    for (int i = 0; i < k; ++i)
      if (i == best) take(i, g.x);
    take(k, g.y);
  }
  int m = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) m += c[i] >= 0 && c[i] < n - 1 && hi[i].w == 0.0f;
  return m;
}

// The binary tree as the wide conversion reads it: interior 0..n-2, leaf n-1+p; blo / bhi
// (hi.w: leaf decision); record position of a leaf (perm, NULL: p) and of a collapsed
// subtree's first triangle, and its triangle count.
struct BinaryTree {
  int n;
  const int2* child;
  const float4* blo;
  const float4* bhi;
  const int* first;
  const int* count;
  const uint32_t* perm;
};

// Level state: [0] nodes of the level, [1] their first record, [3] tickets taken.
__global__ void k_wide_init(int* __restrict__ state, int root, int* __restrict__ frontier) {
  for (int k = 0; k < 8; ++k) state[k] = k == 0;  // the other state: no nodes until a level writes it
  frontier[0] = root;
}

// One level of the wide records: each frontier node's children are opened greedily, those
// that get a record of their own are numbered by a scan over the level (tiles by ticket, the
// offsets by look-back), and the record is written.  Records come out level by level, each
// node's children in consecutive records, the same on every run.  Bound by the latency of
// the child -> box chain and by launches (a tree has 10 to 20 levels): one launch per level,
// with the level's size read from the state the previous one wrote, where a select / scan /
// write sequence took three and a read-back of the size.
__global__ void __launch_bounds__(kScanBlock) k_wide_level(BinaryTree T, int* __restrict__ state,
                                                           int* __restrict__ state_out, int* __restrict__ slot,
                                                           int number, int level, int polls,
                                                           unsigned long long* __restrict__ words,
                                                           const int* __restrict__ frontier,
                                                           int* __restrict__ frontier_out, int max_children,
                                                           float4* __restrict__ wnodes, int max_nodes, int* err) {
  __shared__ int s_tile;
  __shared__ unsigned long long s_before;
  ring_wait();
  const int n_in = state[0], base = state[1], n = T.n;
  const int n_tiles = (n_in + kScanBlock - 1) / kScanBlock;
  const int next_base = base + n_in;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    state_out[3] = 0;
    if (n_in == 0 && !(*(volatile int*)err & kErrTimeout)) {  // past the last level
      state_out[0] = 0;
      state_out[1] = next_base;
      ring_publish(slot, 0, next_base, 0, number);
    }
  }
  for (;;) {
    if (threadIdx.x == 0) s_tile = take_tile(&state[3], err);
    __syncthreads();
    const int tile = s_tile;
    if (tile >= n_tiles) return;
    const int t = tile * kScanBlock + threadIdx.x;
    int c[4];
    float4 lo[4], hi[4];
    int m = 0;
    if (t < n_in) m = wide_select_one(n, T.child, T.blo, T.bhi, frontier[t], max_children, c, lo, hi);
    int total;
    const int ex = block_exclusive_scan(m, total);
    if (threadIdx.x < 32) {
      const unsigned long long before = tiles_before(words, tile, (unsigned long long)total,
                                                     (unsigned)(level % 4095 + 1), polls);
      if (threadIdx.x == 0) {
        s_before = before;
        if (tile == n_tiles - 1 && before <= kTileValue) {
          state_out[0] = (int)before + total;
          state_out[1] = next_base;
          ring_publish(slot, (int)before + total, next_base, 0, number);
        }
      }
    }
    __syncthreads();
    if (s_before > kTileValue) {  // an earlier tile did not publish its sum
      if (threadIdx.x == 0) atomicOr(err, kErrTimeout);
      return;
    }
    if (t < n_in) {
      int next = (int)s_before + ex;
      float v[6][4];
      int ref[4], cnt[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int ci = c[i];
        ref[i] = kEmptyRef;
        cnt[i] = -1;
        bool used = ci >= 0;
        if (used) {
          if (ci >= n - 1) {
            cnt[i] = 1;
            ref[i] = pack_leaf(T.perm ? (int)T.perm[ci - (n - 1)] : ci - (n - 1), 1);
          } else if (hi[i].w != 0.0f) {
            cnt[i] = T.count[ci];
            ref[i] = pack_leaf(T.first[ci], cnt[i]);
          } else if (next_base + next < max_nodes) {
            frontier_out[next] = ci;
            ref[i] = next_base + next++;
            cnt[i] = 0;
          } else {  // cannot happen: the tree has at most n - 1 records (the host stops)
            atomicOr(err, kErrQueue);
            used = false;
            ++next;
          }
        }
        v[0][i] = used ? lo[i].x : kInf;  // unused: a box no ray enters
        v[1][i] = used ? lo[i].y : kInf;
        v[2][i] = used ? lo[i].z : kInf;
        v[3][i] = used ? hi[i].x : -kInf;
        v[4][i] = used ? hi[i].y : -kInf;
        v[5][i] = used ? hi[i].z : -kInf;
      }
      write_record(wnodes, base + t, v, ref, cnt);
    }
    __syncthreads();  // s_tile and s_before are reused
  }
}

// Root record of a scene with 0 or 1 triangle (no binary interior node exists).
__global__ void k_small_root(int n, const float4* __restrict__ blo, const float4* __restrict__ bhi,
                             float4* __restrict__ nodes) {
  float v[6][4];
  for (int a = 0; a < 6; ++a)
    for (int i = 0; i < 4; ++i) v[a][i] = a < 3 ? kInf : -kInf;
  int ref[4] = {kEmptyRef, kEmptyRef, kEmptyRef, kEmptyRef};
  int cnt[4] = {-1, -1, -1, -1};
  if (n == 1) {
    const float4 l = blo[0], h = bhi[0];
    v[0][0] = l.x; v[1][0] = l.y; v[2][0] = l.z;
    v[3][0] = h.x; v[4][0] = h.y; v[5][0] = h.z;
    ref[0] = pack_leaf(0, 1);
    cnt[0] = 1;
  }
  write_record(nodes, 0, v, ref, cnt);
}

inline int grid_for(size_t n, int block) { return (int)std::max<size_t>(1, (n + block - 1) / block); }

// Writes the node records of the binary tree in the given width (top-down, one launch per
// level; the launches run ahead of the host as the PLOC rounds do, and a launch past the last
// level writes nothing).  Returns the number of levels through *levels (kStackMax * 4 + 1
// when the walk did not end, which cannot happen for a tree of depth <= kStackMax).
eos_status write_records(eos_ctx* ctx, const BinaryTree& T, int root, int width, float4* out, int max_nodes,
                         int* levels, int* n_records) {
  cudaStream_t st = ctx->stream;
  eos_status es = EOS_OK;
  const size_t nn = (size_t)T.n;
  int* frontier[2] = {(int*)scratch(ctx, "lbvh.wide.fa", 4 * nn, &es), (int*)scratch(ctx, "lbvh.wide.fb", 4 * nn, &es)};
  const size_t words_bytes = 8 * (size_t)scan_blocks(T.n);
  unsigned long long* words = (unsigned long long*)scratch(ctx, "lbvh.wide.words", words_bytes, &es);
  int* state = (int*)scratch(ctx, "lbvh.wide.state", 32, &es);
  if (es != EOS_OK) return es;
  RoundRing ring(ctx);
  if ((es = ring.init()) != EOS_OK) return es;
  EOS_CUDA(cudaMemsetAsync(words, 0, words_bytes, st));
  k_wide_init<<<1, 1, 0, st>>>(state, root, frontier[0]);
  long long most = 1;  // nodes of the level at most
  int s[3] = {1, 0, 0}, lv = 0;
  for (;;) {
    if (ring.full()) {
      if ((es = ring.read(s)) != EOS_OK) return es;
      ++lv;
      if ((long long)s[1] + s[0] > max_nodes) return EOS_ERR_QUEUE_OVERFLOW;  // cannot happen, as above
      if (s[0] == 0 || lv > 4 * kStackMax) break;
    }
    const int k = (int)(ring.issued & 1);
    const int grid = (int)std::min<long long>(scan_blocks(most), ctx->num_sms * 4);
    es = ring.launch(k_wide_level, grid, kScanBlock, T, state + 4 * k, state + 4 * (k ^ 1), ring.next_slot(),
                     ring.next_number(), (int)ring.issued, ctx->build_polls, words, frontier[k], frontier[k ^ 1], width, out, max_nodes,
                     ctx->d_err);
    if (es != EOS_OK) return es;
    most = std::min<long long>(most * width, T.n);
  }
  *n_records = std::min(s[1] + s[0], max_nodes);
  *levels = s[0] > 0 ? 4 * kStackMax + 1 : lv;
  return EOS_OK;
}

// Node records of the scene.  The traversal stack holds at most width - 1 entries per
// level, so a 4-wide tree deeper than kStackMax / 3 levels (degenerate geometry) is written
// with two children per record instead; a binary tree's depth is at most 62 <= kStackMax.
eos_status build_records(eos_ctx* ctx, eos_scene* sc, const BinaryTree& T, int root) {
  const int max_nodes = T.n - 1;
  EOS_CUDA(pool_alloc(ctx, &sc->d_nodes, 128 * (size_t)max_nodes));
  sc->device_bytes += 128 * (size_t)max_nodes;
  int levels = 0, records = 0;
  eos_status es = write_records(ctx, T, root, sc->width, (float4*)sc->d_nodes, max_nodes, &levels, &records);
  if (es != EOS_OK) return es;
  if (sc->width == 4 && 3 * levels > kStackMax) {
    sc->width = 2;
    es = write_records(ctx, T, root, 2, (float4*)sc->d_nodes, max_nodes, &levels, &records);
    if (es != EOS_OK) return es;
  }
  if ((sc->width - 1) * levels > kStackMax) return EOS_ERR_STACK_OVERFLOW;
  sc->n_nodes = (uint32_t)records;
  sc->levels = levels;
  return EOS_OK;
}

}  // namespace

eos_status build_scene(eos_ctx* ctx, eos_scene* sc, const float* d_verts, const float* d_normals,
                       uint32_t n_verts, const uint32_t* d_tris, const uint32_t* d_obj, uint32_t n_tris) {
  cudaStream_t st = ctx->stream;
  const int n = (int)n_tris;
  const size_t nn = std::max<size_t>(1, n);
  eos_status es = EOS_OK;
  const size_t n_nodes = std::max<size_t>(1, nn - 1);
  // persistent scene buffers (node records: build_records, or one root record below)
  EOS_CUDA(pool_alloc(ctx, &sc->d_tris, 48 * nn));
  EOS_CUDA(pool_alloc(ctx, &sc->d_shade, 48 * nn));
  EOS_CUDA(pool_alloc(ctx, &sc->d_pos_of_id, 4 * nn));
  EOS_CUDA(pool_alloc(ctx, &sc->d_codes, 4 * nn));
  EOS_CUDA(pool_alloc(ctx, &sc->d_order, 4 * nn));
  sc->device_bytes += 48 * nn * 2 + 4 * nn * 3;
  // temporaries
  float4* cent = (float4*)scratch(ctx, "lbvh.cent", 16 * nn, &es);
  uint32_t* bounds = (uint32_t*)scratch(ctx, "lbvh.bounds", 64, &es);
  uint32_t* k2 = (uint32_t*)scratch(ctx, "lbvh.k2", 4 * nn, &es);
  uint32_t* v2 = (uint32_t*)scratch(ctx, "lbvh.v2", 4 * nn, &es);
  const int n_tiles = (int)((nn + kSortTile - 1) / kSortTile);
  uint32_t* counts = (uint32_t*)scratch(ctx, "lbvh.counts", 4 * (size_t)kRadix * n_tiles, &es);
  uint32_t* totals = (uint32_t*)scratch(ctx, "lbvh.totals", 4 * kRadix, &es);
  int2* child = (int2*)scratch(ctx, "lbvh.child", 8 * n_nodes, &es);
  int* count = (int*)scratch(ctx, "lbvh.count", 4 * n_nodes, &es);
  int* first = (int*)scratch(ctx, "lbvh.first", 4 * n_nodes, &es);
  float4* blo = (float4*)scratch(ctx, "lbvh.blo", 16 * (2 * nn), &es);
  float4* bhi = (float4*)scratch(ctx, "lbvh.bhi", 16 * (2 * nn), &es);
  if (es != EOS_OK) return es;

  uint32_t* keys = (uint32_t*)sc->d_codes;
  uint32_t* vals = (uint32_t*)sc->d_order;
  EOS_CUDA(cudaEventRecord(ctx->ev0, st));
  if (n > 0) {
    uint32_t init[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
    EOS_CUDA(cudaMemcpyAsync(bounds, init, sizeof init, cudaMemcpyHostToDevice, st));
    int g = std::min(grid_for(nn, 256), ctx->num_sms * 8);
    k_centroids<<<g, 256, 0, st>>>(d_verts, n_verts, d_tris, n, cent, bounds, ctx->d_err);
    uint32_t *ki = k2, *vi = v2, *ko = keys, *vo = vals;  // three passes end in (keys, vals)
    k_morton<<<n_tiles, kSortThreads, 0, st>>>(cent, n, bounds, ki, vi, counts, n_tiles);
    for (int shift = 0; shift < 30; shift += kRadixBits) {
      if (shift > 0) k_sort_hist<<<n_tiles, kSortThreads, 0, st>>>(ki, n, shift, counts, n_tiles);
      k_sort_scan_rows<<<kRadix * 32 / kSortThreads, kSortThreads, 0, st>>>(counts, n_tiles, totals);
      k_sort_scatter<<<n_tiles, kSortThreads, 0, st>>>(ki, vi, ko, vo, n, shift, counts, n_tiles, totals);
      std::swap(ki, ko);
      std::swap(vi, vo);
    }
  }
  auto records = [&](const uint32_t* perm, float4* lo, float4* hi) {
    k_records<<<grid_for(nn, 256), 256, 0, st>>>(d_verts, d_normals, n_verts, d_tris, d_obj, vals, perm, n,
                                                 (uint32_t)sc->dev.n_obj, (float4*)sc->d_tris, (float4*)sc->d_shade,
                                                 (int32_t*)sc->d_pos_of_id, lo, hi, ctx->d_err);
  };
  if (n >= 2) {
    uint32_t* perm = nullptr;
    int root = 0;
    if (sc->builder == EOS_BUILDER_PLOC) {
      // PLOC over the leaf boxes in Morton order; the records in the tree's depth-first leaf
      // order (every subtree a contiguous range)
      perm = (uint32_t*)scratch(ctx, "lbvh.perm", 4 * nn, &es);
      if (es != EOS_OK) return es;
      k_leaf_boxes<<<grid_for(nn, 256), 256, 0, st>>>(d_verts, n_verts, d_tris, vals, n, blo, bhi);
      int depth = 0;
      es = build_ploc(ctx, n, sc->leaf_size, sc->layout == EOS_LAYOUT_SAH, blo, bhi, child, count, first, perm, &depth);
      if (es != EOS_OK) return es;
      if (depth + 2 <= kStackMax) {
        root = n - 2;
        records(perm, nullptr, nullptr);
      } else {  // deeper than the refit walks: the LBVH instead
        sc->builder = EOS_BUILDER_LBVH;
      }
    }
    if (sc->builder == EOS_BUILDER_LBVH) {
      perm = nullptr;
      int* parent = (int*)scratch(ctx, "lbvh.parent", 4 * (2 * nn), &es);
      int* arrive = (int*)scratch(ctx, "lbvh.arrive", 4 * n_nodes, &es);
      if (es != EOS_OK) return es;
      records(nullptr, blo, bhi);
      EOS_CUDA(cudaMemsetAsync(arrive, 0, 4 * n_nodes, st));
      EOS_CUDA(cudaMemsetAsync(parent, 0xff, 4 * (2 * nn), st));
      k_karras<<<grid_for(n - 1, 256), 256, 0, st>>>(keys, n, child, first, count, parent);
      k_refit<<<grid_for(nn, 256), 256, 0, st>>>(n, child, count, parent, blo, bhi, arrive, sc->leaf_size,
                                                sc->layout == EOS_LAYOUT_SAH, ctx->d_err);
    }
    // SAH cost of the tree (subtree cost of the root, in triangle-test units)
    EOS_CUDA(cudaMemcpyAsync(&sc->sah_cost, &blo[root].w, sizeof(float), cudaMemcpyDeviceToHost, st));
    const BinaryTree T{n, child, blo, bhi, first, count, perm};
    eos_status ws = build_records(ctx, sc, T, root);
    if (ws != EOS_OK) return ws;
  } else {
    if (n == 1) records(nullptr, blo, bhi);
    EOS_CUDA(pool_alloc(ctx, &sc->d_nodes, 128));
    sc->device_bytes += 128;
    k_small_root<<<1, 1, 0, st>>>(n, blo, bhi, (float4*)sc->d_nodes);
    sc->n_nodes = 1;
    sc->levels = 1;
  }
  EOS_CUDA(cudaGetLastError());
  EOS_CUDA(cudaEventRecord(ctx->ev1, st));
  EOS_CUDA(cudaEventSynchronize(ctx->ev1));
  EOS_CUDA(cudaEventElapsedTime(&sc->build_ms, ctx->ev0, ctx->ev1));
  return EOS_OK;
}

}  // namespace eos
