// Plain renderer: one launch per frame, a lane per pixel (all its samples), the whole
// Whitted path of that pixel in the lane: nearest hit, one shadow ray per light, Phong,
// mirror bounce up to trace_depth (src/RayTracer.cpp:99-174,268-458).  This is the
// B200 replacement of the reference's primary-only __rayTrace_MegaKernel
// (src/kernelInvocations.cu:172-310) with the CPU renderer's full semantics.
//
// Also the ray-query kernels behind eos_trace_closest / eos_trace_any.
#include <algorithm>
#include <climits>
#include <type_traits>

#include "trace.cuh"

namespace eos {
namespace {

struct PlainParams {
  DevScene s;
  float cam[12];
  int width, height, trace_depth, spp;
  int y0, rows;  // image rows [y0, y0 + rows) are rendered; outputs hold those rows
  float pixel_offset;
  uint32_t jitter_seed;
  int grid;  // side of the reference's AA grid (EOS_FLAG_AA_GRID), 0 = jitter
  float* rgb;
  uint8_t* rgba8;
  int32_t* hit;
  eos_path_record* paths;
  eos_tree_node* tree;         // tree-form records (TREE kernel): EOS_TREE_NODES(trace_depth) per path
  int* err;
  unsigned long long* counts;  // kNumCounts traversal counters
  uint32_t* work;     // pixels taken (zero at the call's start)
  uint32_t n_work;    // pixels of the band's 8x4 tiles
  int lanes;          // lanes of a warp that trace (lanes_of)
};

// A shaded hit: its point, normal and material, the Phong sum over its unblocked lights and
// the mask of the blocked ones.
struct ShadedHit {
  f3 P, N, phong;
  const float* m;
  uint32_t mask;
};

template <int SH, TraversalForm F>
__device__ __forceinline__ ShadedHit shade_hit(const PlainParams& P, f3 o, f3 d, const Hit& h, unsigned* cnt,
                                               uint32_t col, uint32_t stride) {
  const DevScene& s = P.s;
  const f3 campos = mk3(P.cam[0], P.cam[1], P.cam[2]);
  ShadedHit r;
  int obj;
  hit_geometry(s, o, d, h, r.P, r.N, obj);
  r.m = s.mats + kMatStride * obj;
  r.phong = mk3(0.0f, 0.0f, 0.0f);
  r.mask = 0;
  for (int li = 0; li < s.n_lights; ++li) {
    const float* l = s.lights + 6 * li;
    f3 sd = norm3(sub3(mk3(l[0], l[1], l[2]), r.P));
    f3 so = add3(r.P, scale3(kRayEps, sd));
    cnt[kCntShadow]++;
    AnyResult ar = any_hit<SH, F>(s, so, sd, col, stride, P.err);
    cnt[kCntNodesA] += ar.nodes;
    cnt[kCntTestsA] += ar.tests;
    if (ar.hit) r.mask |= 1u << li;
    else r.phong = add3(r.phong, phong_light(r.m, l, r.P, r.N, campos));
  }
  return r;
}

// A path of one secondary ray per hit, traced a ray at a time: begin, then step until it
// returns true; colour with the reference's fold c_k = phong_k + w_k c_{k+1} (fold_colour).
template <int SH, TraversalForm F>
struct ChainPath {
  f3 o, d;
  int k;  // bounce of the ray
  f3 phong[kMaxBounces];
  float weight[kMaxBounces];
  int32_t hits[kMaxBounces];
  uint32_t masks[kMaxBounces];

  __device__ __forceinline__ void begin(const PlainParams& P, size_t path) {
    k = 0;
#pragma unroll
    for (int i = 0; i < kMaxBounces; ++i) {
      hits[i] = EOS_HIT_UNTRACED;
      masks[i] = 0;
    }
  }
  __device__ __forceinline__ bool step(const PlainParams& P, size_t path, f3& c, unsigned* cnt, uint32_t col,
                                       uint32_t stride) {
    const DevScene& s = P.s;
    cnt[k == 0 ? kCntPrimary : kCntSecondary]++;
    Hit h = closest_hit<SH, F>(s, o, d, col, stride, P.err);
    cnt[kCntNodesC] += h.nodes;
    cnt[kCntTestsC] += h.tests;
    int nb = k;
    hits[k] = h.pos < 0 ? EOS_HIT_NONE : h.id;
    if (h.pos >= 0) {
      cnt[kCntHits]++;
      const ShadedHit r = shade_hit<SH, F>(P, o, d, h, cnt, col, stride);
      masks[k] = r.mask;
      phong[k] = r.phong;
      nb = k + 1;
      f3 ro, rd;
      if (secondary_ray(r.m, s.ambient_index, d, r.P, r.N, ro, rd, weight[k]) && k < P.trace_depth) {
        o = ro;
        d = rd;
        ++k;
        return false;
      }
    }
    c = mk3(0.0f, 0.0f, 0.0f);
    for (int i = nb - 1; i >= 0; --i) c = fold_colour(phong[i], weight[i], c);
    if (P.hit) P.hit[path] = hits[0];
    if (P.paths) {
      eos_path_record rec;
#pragma unroll
      for (int i = 0; i < kMaxBounces; ++i) {
        rec.hit[i] = hits[i];
        rec.shadow[i] = masks[i];
      }
      P.paths[path] = rec;
    }
    return true;
  }
};

// One shaded node of a ray tree waiting for its children (TreePath).
struct TreeFrame {
  f3 phong, cR;   // the node's Phong sum; its mirror child's colour once known
  f3 to, td;      // its transparent child's ray; to: that child's colour once another lane has it
  float wR, K;    // reflectivity (0: no mirror ray), Fresnel weight of the transparent ray
  int node, depth;
  bool has_t;     // transparent ray present
  bool in_t;      // the child being traced (or waited for) is the transparent one
};

// A path as a ray tree (materials both reflective and transparent trace both secondary
// rays, src/RayTracer.cpp:339-407), traced a ray at a time: a post-order walk with an
// explicit stack of shaded nodes (at most one per bounce), mirror child first as the
// reference recurses; node colours by tree_colour.  Tree records in heap order.
//
// What bounds a frame of ray trees is the serial walk of its deepest trees (31 nodes at trace
// depth 4, each with its shadow rays), while most lanes' trees end after a ray or two.  So a
// lane without a tree takes the transparent child of a waiting node from another lane of
// its warp (share): the subtree nearest the root first, whose colour goes back to the
// owner's frame, which sums it in its place, with the same operations.
template <int SH, TraversalForm F>
struct TreePath {
  f3 o, d;
  int sp, node, depth;
  uint32_t open;   // frames whose transparent child is still to be traced, by bit
  uint32_t lent;   // frames whose transparent child another lane traces
  int owner;       // lane and frame that this subtree's colour goes to, (lane | frame << 8); -1: a pixel
  bool waiting;    // for the lent child of the top frame: nothing to trace
  TreeFrame st[kMaxBounces];

  __device__ __forceinline__ void begin(const PlainParams& P, size_t path) {
    sp = node = depth = 0;
    open = lent = 0;
    owner = -1;
    waiting = false;
    if (P.tree) {
      const int nn = EOS_TREE_NODES(P.trace_depth);
      eos_tree_node* rec = P.tree + path * nn;
      for (int k = 0; k < nn; ++k) rec[k] = eos_tree_node{EOS_HIT_UNTRACED, 0u};
    }
  }
  // The colour waited for is there: hand_up goes on.
  __device__ __forceinline__ bool resumes() const { return waiting && !(lent >> (sp - 1) & 1u); }

  __device__ __forceinline__ bool step(const PlainParams& P, size_t path, f3& c, unsigned* cnt, uint32_t col,
                                       uint32_t stride) {
    const DevScene& s = P.s;
    const f3 zero = mk3(0.0f, 0.0f, 0.0f);
    c = zero;
    cnt[depth == 0 ? kCntPrimary : kCntSecondary]++;
    Hit h = closest_hit<SH, F>(s, o, d, col, stride, P.err);
    cnt[kCntNodesC] += h.nodes;
    cnt[kCntTestsC] += h.tests;
    const int id = h.pos < 0 ? EOS_HIT_NONE : h.id;
    if (node == 0 && P.hit) P.hit[path] = id;
    eos_tree_node* rec = P.tree ? P.tree + path * EOS_TREE_NODES(P.trace_depth) + node : nullptr;
    if (rec) rec->hit = id;
    if (h.pos >= 0) {
      cnt[kCntHits]++;
      const ShadedHit r = shade_hit<SH, F>(P, o, d, h, cnt, col, stride);
      if (rec) rec->shadow = r.mask;
      TreeFrame f;
      f.phong = r.phong;
      f3 ro = zero, rd = zero;
      const bool has_r = r.m[7] > 0.0f;
      f.wR = has_r ? r.m[7] : 0.0f;
      if (has_r) mirror_ray(d, r.P, r.N, ro, rd);
      f.has_t = r.m[8] > 0.0f;
      f.K = f.has_t ? transparent_ray(r.m, s.ambient_index, d, r.P, r.N, f.to, f.td) : 0.0f;
      f.cR = zero;
      f.node = node;
      f.depth = depth;
      if (depth < P.trace_depth && (has_r || f.has_t)) {
        f.in_t = !has_r;
        if (has_r && f.has_t) open |= 1u << sp;
        st[sp++] = f;
        if (has_r) {
          o = ro;
          d = rd;
          node = 2 * node + 1;
        } else {
          o = f.to;
          d = f.td;
          node = 2 * node + 2;
        }
        ++depth;
        return false;
      }
      c = tree_colour(f.phong, f.wR, zero, f.has_t, f.K, zero);  // children beyond the trace depth
    }
    return hand_up(c);
  }
  // Hands a finished child's colour up until a node still has its transparent child to
  // trace or to wait for; true: c is the whole tree's.
  __device__ __forceinline__ bool hand_up(f3& c) {
    const f3 zero = mk3(0.0f, 0.0f, 0.0f);
    if (waiting) {
      const TreeFrame& f = st[--sp];
      waiting = false;
      c = tree_colour(f.phong, f.wR, f.cR, true, f.K, f.to);
    }
    while (sp > 0) {
      TreeFrame& f = st[sp - 1];
      const uint32_t bit = 1u << (sp - 1);
      if (!f.in_t) {
        f.cR = c;
        if (f.has_t) {
          f.in_t = true;
          if (open & bit) {
            open &= ~bit;
            o = f.to;
            d = f.td;
            node = 2 * f.node + 2;
            depth = f.depth + 1;
            return false;
          }
          if (lent & bit) {
            waiting = true;
            return false;
          }
          c = tree_colour(f.phong, f.wR, f.cR, true, f.K, f.to);  // another lane traced it
        } else {
          c = tree_colour(f.phong, f.wR, f.cR, false, 0.0f, zero);
        }
      } else {
        c = tree_colour(f.phong, f.wR, f.cR, true, f.K, c);
      }
      --sp;
    }
    return true;
  }
};

// The `idle` lanes take open subtrees of the warp's other lanes, with the owner's pixel (x, ly,
// smp).  Warp-uniform.
template <class Path>
__device__ __forceinline__ void share_trees(Path& t, uint32_t idle, bool& active, bool& fresh, int& x, int& ly,
                                            int& smp) {
  const int lane = threadIdx.x & 31;
  __syncwarp();  // the owner's clearing of its tree record comes before the taker's writes to it
  uint32_t open = __ballot_sync(0xffffffffu, active && t.open != 0);
  while (open && idle) {
    const int from = __ffs(open) - 1, to = __ffs(idle) - 1;
    open &= open - 1;
    idle &= idle - 1;
    f3 o = mk3(0, 0, 0), d = o;
    int node = 0, depth = 0, frame = 0;
    if (lane == from) {
      frame = __ffs(t.open) - 1;
      t.open &= t.open - 1;
      t.lent |= 1u << frame;
      const TreeFrame& f = t.st[frame];
      o = f.to;
      d = f.td;
      node = 2 * f.node + 2;
      depth = f.depth + 1;
    }
    o = mk3(__shfl_sync(~0u, o.x, from), __shfl_sync(~0u, o.y, from), __shfl_sync(~0u, o.z, from));
    d = mk3(__shfl_sync(~0u, d.x, from), __shfl_sync(~0u, d.y, from), __shfl_sync(~0u, d.z, from));
    node = __shfl_sync(~0u, node, from);
    depth = __shfl_sync(~0u, depth, from);
    frame = __shfl_sync(~0u, frame, from);
    const int fx = __shfl_sync(~0u, x, from), fly = __shfl_sync(~0u, ly, from), fsmp = __shfl_sync(~0u, smp, from);
    if (lane == to) {
      t.o = o;
      t.d = d;
      t.node = node;
      t.depth = depth;
      t.sp = 0;
      t.open = t.lent = 0;
      t.owner = from | (frame << 8);
      t.waiting = false;
      x = fx;
      ly = fly;
      smp = fsmp;
      active = true;
      fresh = false;
    }
  }
}

// Colours of the subtrees that lanes of `done` have finished go to their owners.  Warp-uniform.
template <class Path>
__device__ __forceinline__ void return_trees(Path& t, uint32_t done, f3 c) {
  const int lane = threadIdx.x & 31;
  while (done) {
    const int from = __ffs(done) - 1;
    done &= done - 1;
    const int owner = __shfl_sync(~0u, t.owner, from);
    const f3 v = mk3(__shfl_sync(~0u, c.x, from), __shfl_sync(~0u, c.y, from), __shfl_sync(~0u, c.z, from));
    if (lane == (owner & 255)) {
      t.st[owner >> 8].to = v;
      t.lent &= ~(1u << (owner >> 8));
    }
  }
}

// The traversals are inline, for flat scenes without the two-level one (TraversalForm), and the
// registers capped where resident warps and spills balance.  Measured, us for a 1080p frame of
// 200k triangles and a 961x541 frame of ray trees: out of line at 64 registers 867 and 2,050;
// inline at 56 854 and 1,917, 64 816 and 1,896, 72 807 and 1,769, 80 817 and 1,765, 88 842 and
// 1,753.  1080p of 801 instances: out of line at 64 13.2 ms; inline at 64 12.1, 80 11.6, 96 12.0.
template <int SH, bool TREE, TraversalForm F>
__global__ void __maxnreg__(F == kTwoLevel ? 80 : TREE ? 88 : 72) k_render_plain(PlainParams P) {
  extern __shared__ uint2 shstack[];
  const uint32_t col = shared_address(shstack + threadIdx.x), stride = 8 * blockDim.x;
  unsigned cnt[kNumCounts] = {0, 0, 0, 0, 0, 0, 0, 0};
  const int lane = threadIdx.x & 31;
  const int tiles_x = (P.width + 7) >> 3;
  typename std::conditional<TREE, TreePath<SH, F>, ChainPath<SH, F>>::type path;
  bool active = false, fresh = false;  // a pixel in hand; its next sample not begun
  bool more = lane < P.lanes;          // may take another pixel
  int x = 0, ly = 0, smp = 0;
  f3 sum = mk3(0.0f, 0.0f, 0.0f);
  for (;;) {
    if constexpr (TREE) {
      const uint32_t spare = __ballot_sync(0xffffffffu, lane < P.lanes && !active);
      if (spare) share_trees(path, spare, active, fresh, x, ly, smp);
    }
    const uint32_t idle = __ballot_sync(0xffffffffu, more && !active);
    const uint32_t busy = __ballot_sync(0xffffffffu, active);
    // the next pixels once all lanes are done: taking them as single lanes end, or 16 of them,
    // mixes bounces in a warp, 813 -> 841 and 830 us for a 1080p frame of 200k triangles
    if (idle && !busy) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(P.work, __popc(idle));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (more && !active) {
        const uint32_t g = base + __popc(idle & ((1u << lane) - 1u));
        more = g < P.n_work;
        // 32 consecutive pixels = one 8x4 tile (coherent primary rays)
        const int tile = (int)(g >> 5), q = (int)(g & 31u);
        x = (tile % tiles_x) * 8 + (q & 7);
        ly = (tile / tiles_x) * 4 + (q >> 3);  // row within the rendered band
        active = fresh = more && x < P.width && ly < P.rows;
        smp = 0;
        sum = mk3(0.0f, 0.0f, 0.0f);
      }
    } else if (!busy) {
      break;
    }
    if (active && fresh) {
      float ox, oy;  // the sample hash takes the pixel of the whole image
      const int y = P.y0 + ly;
      sample_offset((uint32_t)(y * P.width + x), smp, P.spp, P.jitter_seed, P.pixel_offset, ox, oy, P.grid);
      path.d = primary_direction(P.cam, P.width, P.height, x, y, ox, oy);
      path.o = mk3(P.cam[0], P.cam[1], P.cam[2]);
      path.begin(P, ((size_t)ly * P.width + x) * P.spp + smp);
      fresh = false;
    }
    // a ray of the path in hand (its index in the outputs); true when the path ends with colour c
    auto trace = [&](f3& c) {
      return path.step(P, ((size_t)ly * P.width + x) * P.spp + smp, c, cnt, col, stride);
    };
    auto end_sample = [&](f3 c) {
      sum = add3(sum, c);
      fresh = true;
      if (++smp < P.spp) return;
      active = false;
      const size_t pix = (size_t)ly * P.width + x;  // pixel of the outputs
      if (P.spp > 1 || P.grid > 0) sum = scale3(sample_weight(P.spp, P.grid), sum);
      if (P.rgb) {
        P.rgb[3 * pix] = sum.x;
        P.rgb[3 * pix + 1] = sum.y;
        P.rgb[3 * pix + 2] = sum.z;
      }
      if (P.rgba8)
        reinterpret_cast<uchar4*>(P.rgba8)[pix] = make_uchar4(quantize(sum.x), quantize(sum.y), quantize(sum.z), 255);
    };
    if constexpr (!TREE) {
      f3 c;
      if (active && trace(c)) end_sample(c);
      __syncwarp();
    } else {
      const bool traces = active && !path.waiting;
      f3 c = mk3(0.0f, 0.0f, 0.0f);
      bool ends = traces && trace(c);  // the tree, or the subtree in hand
      // cannot happen: who waits has lent a subtree to a lane that traces or waits in turn
      if (!__any_sync(0xffffffffu, traces) && __any_sync(0xffffffffu, active)) {
        if (lane == 0) atomicOr(P.err, kErrTimeout);
        break;
      }
      // subtree colours to their owners; owners that waited for one go on
      uint32_t done = __ballot_sync(0xffffffffu, ends && path.owner >= 0);
      while (done) {
        return_trees(path, done, c);
        if (done >> lane & 1u) active = ends = false;
        if (active && !ends && path.resumes()) ends = path.hand_up(c);
        done = __ballot_sync(0xffffffffu, ends && path.owner >= 0);
      }
      if (ends) end_sample(c);
    }
  }
#pragma unroll
  for (int c = 0; c < kNumCounts; ++c) warp_add_count(&P.counts[c], cnt[c]);
}

// Ray of this thread: `lanes` of each warp take one (lanes_of).
__device__ __forceinline__ int query_ray(int lanes) {
  const int lane = threadIdx.x & 31, warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  return lane < lanes ? warp * lanes + lane : INT_MAX;
}

// Ray queries, one warp a block: the caller's rays are as incoherent as it likes, so a warp
// walks the union of its lanes' nodes and what helps is warps in flight and blocks that end
// early.  The traversal is inline (62 and 55 registers; two-level scenes 80 and 88).  Measured
// on 60k triangles against the traversal out of line at 90 registers in blocks of 128: 300k
// rays nearest 182 -> 159 us and any 147 -> 131, 1M rays 477 -> 370 and 365 -> 291, 1,000 rays
// (4 lanes a warp) 59 -> 50 and 47 -> 45; at 48 registers 194 and 144 for 300k.
template <int SH, TraversalForm F>
__global__ void __maxnreg__(80) k_trace_closest(DevScene s, const float* __restrict__ rays,
                                                                      int n, int lanes, int32_t* ids, float* ts,
                                                                      int* err) {
  extern __shared__ uint2 shstack[];
  const int i = query_ray(lanes);
  if (i >= n) return;
  const float* r = rays + 6 * (size_t)i;
  Hit h = closest_hit<SH, F>(s, mk3(r[0], r[1], r[2]), mk3(r[3], r[4], r[5]), shared_address(shstack + threadIdx.x),
                             8 * blockDim.x, err);
  ids[i] = h.pos < 0 ? EOS_HIT_NONE : h.id;
  if (ts) ts[i] = h.t;
}

template <int SH, TraversalForm F>
__global__ void __maxnreg__(F == kTwoLevel ? 96 : 56) k_trace_any(DevScene s, const float* __restrict__ rays, int n,
                                                                  int lanes, uint8_t* occ, int* err) {
  extern __shared__ int shrefs[];
  const int i = query_ray(lanes);
  if (i >= n) return;
  const float* r = rays + 6 * (size_t)i;
  occ[i] = any_hit<SH, F>(s, mk3(r[0], r[1], r[2]), mk3(r[3], r[4], r[5]), shared_address(shrefs + threadIdx.x),
                          4 * blockDim.x, err).hit ? 1 : 0;
}

inline int clamp_block(int b) { return b <= 0 ? 128 : std::min(512, std::max(32, (b / 32) * 32)); }
inline int pick_stack(int d) { return d <= 0 ? 16 : (d <= 8 ? 8 : (d <= 16 ? 16 : 32)); }

}  // namespace

namespace {

// Lanes of a warp that trace.  A frame of few pixels is bound by the time of its slowest
// warp, which walks the union of its lanes' nodes, while most of the chip idles: with fewer
// lanes a warp the same pixels spread over more warps.  Chains: the fewest lanes that leave
// every warp resident in the kernel for flat scenes (28 warps of 72 registers per SM; the
// two-level one holds 25, the queries 32 and 21, and their steps are taken at the same
// place).  Measured, us at 32 / 16 / 8 / 4 lanes: 64x64 of 200k triangles 207 / 188 / 181 / 147,
// 128x128 238 / 226 / 189 / 174, 256x256 247 / 244 / 249 / 287, 512x512 355 / 396 / 518 / 763;
// 801 instances 64x64 1,294 / 969 / 777 / 629, 256x256 2,045 / 1,797 / 1,636 / 1,870, 512x512
// 2,893 / 3,391; nearest hits of 1,000 rays 61 / 61 / 59 / 58, 33,000 71 / 70 / 71 / 83, 300,000
// 157 / 194.  Ray trees have longer tails (a pixel's tree is walked by a warp): 8 lanes up to
// four such fillings, 16 up to eight.  At 32 / 16 / 8 lanes: 400x300 1,449 / 1,565 / 1,300,
// 640x360 1,644 / 1,429 / 1,287, 800x450 1,651 / 1,545 / 1,626, 961x541 1,886 / 1,721 / 1,998,
// 1200x675 2,210 / 2,143 / 2,361, 1440x810 2,394 / 2,483; between the steps the rule is up to
// 10 % from the best count.
int lanes_of(uint32_t n_work, int num_sms, bool tree) {
  const uint32_t full = 28u * (uint32_t)num_sms;  // warps that fill the chip
  if (tree) return n_work / 8 <= 4 * full ? 8 : n_work / 16 <= 8 * full ? 16 : 32;
  for (int lanes = 4; lanes < 32; lanes *= 2)
    if (n_work / lanes <= full) return lanes;
  return 32;
}

template <int SH, bool TREE, TraversalForm F>
eos_status launch_plain(eos_ctx* ctx, const PlainParams& P, int block) {
  auto* kernel = k_render_plain<SH, TREE, F>;
  const size_t smem = (size_t)SH * block * sizeof(uint2);
  if (smem > 48 * 1024)  // opt in to more than the default 48 KB of dynamic shared memory
    EOS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int resident = 0;
  EOS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kernel, block, smem));
  const long long per_block = (long long)P.lanes * (block / 32);
  const long long blocks = ((long long)P.n_work + per_block - 1) / per_block;
  const int grid = (int)std::max<long long>(1, std::min<long long>(blocks, (long long)ctx->num_sms * std::max(1, resident)));
  kernel<<<grid, block, smem, ctx->stream>>>(P);
  EOS_CUDA(cudaGetLastError());
  return EOS_OK;
}

template <bool TREE, TraversalForm F>
eos_status launch_plain(eos_ctx* ctx, const PlainParams& P, int sh, int block) {
  if (sh == 8) return launch_plain<8, TREE, F>(ctx, P, block);
  if (sh == 16) return launch_plain<16, TREE, F>(ctx, P, block);
  return launch_plain<32, TREE, F>(ctx, P, block);
}

}  // namespace

// tree: ray-tree kernel (scenes with materials both reflective and transparent, or tree
// records asked for); paths then points at tree-form records.
eos_status render_plain(eos_ctx* ctx, const eos_scene* sc, const eos_camera& cam, const eos_render_params& p,
                        float* rgb, uint8_t* rgba8, int32_t* hit, void* paths, bool tree) {
  PlainParams P;
  P.s = sc->dev;
  for (int k = 0; k < 3; ++k) {
    P.cam[k] = cam.position[k];
    P.cam[3 + k] = cam.view[k];
    P.cam[6 + k] = cam.right[k];
    P.cam[9 + k] = cam.up[k];
  }
  P.width = cam.width;
  P.height = cam.height;
  P.y0 = p.row_end > 0 ? p.row_begin : 0;
  P.rows = p.row_end > 0 ? p.row_end - p.row_begin : cam.height;
  P.trace_depth = p.trace_depth;
  P.spp = p.spp;
  P.pixel_offset = p.pixel_offset;
  P.jitter_seed = p.jitter_seed;
  P.grid = (p.flags & EOS_FLAG_AA_GRID) ? aa_grid_side(p.spp) : 0;
  P.rgb = rgb;
  P.rgba8 = rgba8;
  P.hit = hit;
  P.paths = tree ? nullptr : (eos_path_record*)paths;
  P.tree = tree ? (eos_tree_node*)paths : nullptr;
  P.err = ctx->d_err;
  P.counts = ctx->d_counts;
  P.work = (uint32_t*)ctx->d_work;
  P.n_work = (uint32_t)((long long)((cam.width + 7) / 8) * ((P.rows + 3) / 4) * 32);
  P.lanes = lanes_of(P.n_work, ctx->num_sms, tree);
  const int block = clamp_block(p.block_size);
  const int sh = pick_stack(p.stack_depth);
  const eos_status st = sc->instanced ? (tree ? launch_plain<true, kTwoLevel>(ctx, P, sh, block)
                                              : launch_plain<false, kTwoLevel>(ctx, P, sh, block))
                                      : (tree ? launch_plain<true, kFlat>(ctx, P, sh, block)
                                              : launch_plain<false, kFlat>(ctx, P, sh, block));
  if (st != EOS_OK) return st;
  ctx->launches += 1;
  return EOS_OK;
}

eos_status trace_closest(eos_ctx* ctx, const eos_scene* sc, const float* d_rays, uint32_t n, int32_t* d_ids,
                         float* d_t) {
  if (n == 0) return EOS_OK;
  const int block = 32, lanes = lanes_of(n, ctx->num_sms, false), per_block = lanes * (block / 32);
  const int grid = (int)((n + per_block - 1) / per_block);
  (sc->instanced ? k_trace_closest<16, kTwoLevel> : k_trace_closest<16, kFlat>)
      <<<grid, block, 16 * block * sizeof(uint2), ctx->stream>>>(sc->dev, d_rays, (int)n, lanes, d_ids, d_t, ctx->d_err);
  EOS_CUDA(cudaGetLastError());
  return EOS_OK;
}

eos_status trace_any(eos_ctx* ctx, const eos_scene* sc, const float* d_rays, uint32_t n, uint8_t* d_occ) {
  if (n == 0) return EOS_OK;
  const int block = 32, lanes = lanes_of(n, ctx->num_sms, false), per_block = lanes * (block / 32);
  const int grid = (int)((n + per_block - 1) / per_block);
  (sc->instanced ? k_trace_any<16, kTwoLevel> : k_trace_any<16, kFlat>)
      <<<grid, block, 16 * block * sizeof(int), ctx->stream>>>(sc->dev, d_rays, (int)n, lanes, d_occ, ctx->d_err);
  EOS_CUDA(cudaGetLastError());
  return EOS_OK;
}

}  // namespace eos
