// Adjoint of the shading (no reference counterpart): gradients of an image loss L with
// respect to per-object kd, ks, log(shininess) and per-light colour and position, with
// visibility frozen from the forward pass's path records (hit triangle per bounce and
// blocked-light masks).  Nothing else of the forward pass is stored: each bounce's hit is
// re-derived from its triangle id with the same exact-order Moller-Trumbore, hit point,
// normal and secondary ray as the forward kernels (in the instance's object space for a
// two-level scene), so the geometry matches the forward pass bit for bit.
//
// Forward model per path (src/RayTracer.cpp:302-458): c = sum_k T_k phong_k with
// T_k = prod_{j<k} w_j, w = reflectivity for a mirror bounce and K + (1 - K) for a
// transparent one (its Fresnel mix of one colour); for a ray tree the sum runs over its
// nodes, T the product of the edge weights from the primary ray.  Per unblocked light l,
//   phong = max(0, N.L) kd*C_l + [V.R > 0] (V.R)^s C_l*ks,  L = (p_l - P)/|p_l - P|,
//   R = w/|w|, w = 2 (N.L) N - L,  V = normalize(camera - P),  s = shininess.
// Gradients with g = dL/dc * T_k:
//   dkd_c += g_c max(0,N.L) C_c          dks_c += g_c (V.R)^s C_c
//   dlog s += sum_c g_c ks_c C_c (V.R)^s ln(V.R) s
//   dC_c  += g_c (max(0,N.L) kd_c + (V.R)^s ks_c)
//   dp_l  += a (N - (N.L) L)/|u|  [N.L > 0]
//          + b s (V.R)^(s-1) (I - L L^T)/|u| (2 N N^T - I) (V - (V.R) R)/|w|  [V.R > 0]
//   with a = sum_c g_c C_c kd_c, b = sum_c g_c C_c ks_c.
// Both sums are reduced over the warp first (every lane takes part, with zeros for blocked
// lights and finished paths; per-object sums for one object of the warp at a time), eight
// components in nine shuffles (warp_sum8), then one shared-memory atomic whose lanes hold
// the components, and at the end of a block one global atomic per component.  The blocks
// are a few per SM and take many paths each: bound by instruction issue and the latency of
// the replay's gathers (record -> position -> triangle -> normals), so what helps is fewer
// instructions per path and resident warps.  Measured (eight 256x256 views, 3 lights, 524k
// paths): 100 us with a warp sum per component, 64-bit index divisions, two powf per light,
// unshared object sums and a block per 128 paths; 42 us now (31.6 -> 24.4 M warp
// instructions, 34 -> 69 % of the issue slots; 64 registers with 56 B of spills are 2 us
// faster than 80).
#include <algorithm>

#include "trace.cuh"

namespace eos {
namespace {

struct BwArgs {
  DevScene s;
  const float* cams;  // n_views x 12
  int w, h, n_views, trace_depth, spp;
  int y0, rows;   // image rows [y0, y0 + rows) of the forward records (a row band, or all)
  float off;
  uint32_t seed;  // sample jitter (spp > 1), as in the forward pass
  int grid;       // side of the reference's AA grid (EOS_FLAG_AA_GRID), 0 = jitter
  const eos_path_record* paths;  // chain records, or
  const eos_tree_node* tree;     // tree records, nn nodes per path
  int nn;
  const float* drgb;
  float* gmat;    // n_obj x 7
  float* glight;  // n_lights x 6
  int* err;
  long long total;  // paths
  int obj_shared;   // per-object sums fit the block's shared memory
};

// Sums of eight values over the warp: each step halves the values a lane carries, so it takes
// 4 + 2 + 1 + 1 + 1 shuffles, not 40.  Lane L gets the sum of component sum8_component(L).
__device__ __forceinline__ int sum8_component(int lane) {
  return ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
}
__device__ __forceinline__ float warp_sum8(const float* v) {
  const int lane = threadIdx.x & 31;
  float a[4], b[2], c;
  const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
#pragma unroll
  for (int k = 0; k < 4; ++k) a[k] = (h4 ? v[4 + k] : v[k]) + __shfl_xor_sync(0xffffffffu, h4 ? v[k] : v[4 + k], 16);
#pragma unroll
  for (int k = 0; k < 2; ++k) b[k] = (h3 ? a[2 + k] : a[k]) + __shfl_xor_sync(0xffffffffu, h3 ? a[k] : a[2 + k], 8);
  c = (h2 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, h2 ? b[0] : b[1], 4);
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  return c + __shfl_xor_sync(0xffffffffu, c, 1);
}

// Primary ray and weighted dL/dc of path i (pixel-major, samples consecutive).  I: an
// unsigned type that holds every path index (32 bits where they fit: the divisions).
template <class I>
__device__ __forceinline__ void path_start(const BwArgs& A, I i, f3& o, f3& d, f3& campos, float* g) {
  const I npx = (I)A.w * (I)A.rows;
  I px = i;  // view * npx + pixel
  int smp = 0;
  if (A.spp > 1) {
    px = i / (unsigned)A.spp;
    smp = (int)(i - px * (unsigned)A.spp);
  }
  const int view = (int)(px / npx);
  const unsigned pix = (unsigned)(px - (I)view * npx);
  const float* cam = A.cams + 12 * view;
  const int row = (int)(pix / (unsigned)A.w);
  const int x = (int)(pix - (unsigned)row * (unsigned)A.w), y = A.y0 + row;  // image row
  float ox, oy;
  sample_offset((uint32_t)(y * A.w + x), smp, A.spp, A.seed, A.off, ox, oy, A.grid);
  d = primary_direction(cam, A.w, A.h, x, y, ox, oy);
  campos = mk3(cam[0], cam[1], cam[2]);
  o = campos;
  // the pixel is the weighted sum of its samples (the mean, or the reference grid's (1/n)^2)
  const float ws = (A.spp > 1 || A.grid > 0) ? sample_weight(A.spp, A.grid) : 1.0f;
  const float* dr = A.drgb + 3 * (size_t)px;
  g[0] = dr[0] * ws;
  g[1] = dr[1] * ws;
  g[2] = dr[2] * ws;
}

// Re-derives the recorded hit `id` of ray (o, d): false (and *alive cleared) when the
// record does not match this scene / camera or holds no hit.
__device__ __forceinline__ bool replay_hit(const BwArgs& A, int id, f3 o, f3 d, f3& P, f3& N, int& obj,
                                           const float*& m) {
  const DevScene& s = A.s;
  if (id < 0 || id >= s.n_tris) return false;
  Hit h;
  if (!hit_of_id(s, o, d, id, h)) {
    atomicOr(A.err, kErrIndex);  // record does not match this scene / camera
    return false;
  }
  hit_geometry(s, o, d, h, P, N, obj);
  m = s.mats + kMatStride * obj;
  return true;
}

// The block's sums: per light [n_lights][6], then, where they fit, per object [n_obj][7].
extern __shared__ float s_sums[];

__device__ __forceinline__ void clear_sums(const BwArgs& A) {
  const int n = 6 * A.s.n_lights + (A.obj_shared ? 7 * A.s.n_obj : 0);
  for (int i = threadIdx.x; i < n; i += blockDim.x) s_sums[i] = 0.0f;
  __syncthreads();
}

__device__ __forceinline__ void flush_sums(const BwArgs& A) {
  __syncthreads();
  const int nl = 6 * A.s.n_lights, n = nl + (A.obj_shared ? 7 * A.s.n_obj : 0);
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    if (s_sums[i] != 0.0f) atomicAdd(i < nl ? &A.glight[i] : &A.gmat[i - nl], s_sums[i]);
}

// Adjoint of one shaded hit per lane (alive lanes; the others take part with zeros):
// per-light terms reduced over the warp into the block's sums, per-object terms by a warp
// segmented reduction.  gT = dL/dc times the hit's throughput.  Warp-uniform.
__device__ __forceinline__ void hit_adjoint(const BwArgs& A, bool alive, f3 P, f3 N, int obj, const float* m,
                                            uint32_t mask, f3 campos, const float* gT) {
  const DevScene& s = A.s;
  const int lane = threadIdx.x & 31, comp = sum8_component(lane);
  const bool adds = (lane & 3) == 0;
  float gm[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  float kd[3] = {0, 0, 0}, ks[3] = {0, 0, 0}, shin = 0.0f;
  f3 V = mk3(0, 0, 1);
  if (alive) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      kd[c] = __ldg(m + c);
      ks[c] = __ldg(m + 3 + c);
    }
    shin = __ldg(m + 6);
    V = norm3(sub3(campos, P));
  } else {
    mask = 0xffffffffu;
  }
  for (int l = 0; l < s.n_lights; ++l) {
    const bool lit = !(mask & (1u << l));
    if (!__any_sync(0xffffffffu, lit)) continue;
    float gl[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (lit) {
      const float* lp = s.lights + 6 * l;
      const float C[3] = {__ldg(lp + 3), __ldg(lp + 4), __ldg(lp + 5)};
      f3 u = sub3(mk3(__ldg(lp), __ldg(lp + 1), __ldg(lp + 2)), P);
      const float ul = sqrtf(dot3(u, u)), iul = 1.0f / ul;
      f3 L = scale3(iul, u);
      float ndl = dot3(N, L);
      f3 wv = sub3(scale3(2.0f * ndl, N), L);
      const float iwl = 1.0f / sqrtf(dot3(wv, wv));
      f3 R = scale3(iwl, wv);
      float fd = ndl > 0.0f ? ndl : 0.0f;
      float vr = dot3(V, R);
      float fs = vr > 0.0f ? powf(vr, shin) : 0.0f;
      float a = 0.0f, b = 0.0f;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        gm[c] += gT[c] * fd * C[c];
        gm[3 + c] += gT[c] * fs * C[c];
        gl[c] = gT[c] * (fd * kd[c] + fs * ks[c]);
        a += gT[c] * C[c] * kd[c];
        b += gT[c] * C[c] * ks[c];
      }
      f3 gp = mk3(0, 0, 0);
      if (ndl > 0.0f) gp = add3(gp, scale3(a / ul, sub3(N, scale3(ndl, L))));
      if (vr > 0.0f) {
        gm[6] += b * fs * logf(vr) * shin;
        f3 q = scale3(iwl, sub3(V, scale3(vr, R)));
        f3 q2 = sub3(scale3(2.0f * dot3(N, q), N), q);
        f3 gs = scale3(iul, sub3(q2, scale3(dot3(L, q2), L)));
        // s (V.R)^(s-1): by a second power where (V.R)^s has lost bits or all of them
        const float p1 = fs >= 0x1p-126f ? fs / vr : powf(vr, shin - 1.0f);
        gp = add3(gp, scale3(b * (shin * p1), gs));
      }
      gl[3] = gp.x;
      gl[4] = gp.y;
      gl[5] = gp.z;
    }
    const float v = warp_sum8(gl);
    if (adds && comp < 6 && v != 0.0f) atomicAdd(&s_sums[6 * l + comp], v);
  }
  // one object of the warp after another
  float* gobj = A.obj_shared ? s_sums + 6 * s.n_lights : A.gmat;
  int key = alive ? obj : -1;
  uint32_t pending = __ballot_sync(0xffffffffu, key >= 0);
  while (pending) {
    const int lk = __shfl_sync(0xffffffffu, key, __ffs(pending) - 1);
    const bool mine = key == lk;
    float t[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) t[c] = mine ? gm[c] : 0.0f;
    const float v = warp_sum8(t);
    if (adds && comp < 7 && v != 0.0f) atomicAdd(&gobj[7 * lk + comp], v);
    pending &= ~__ballot_sync(0xffffffffu, mine);
  }
}

// Chain records: one secondary ray per hit, T_k+1 = T_k fold_weight(w_k).
template <class I>
__global__ void __launch_bounds__(256, 4) k_backward(BwArgs A) {
  clear_sums(A);
  const DevScene& s = A.s;
  const I total = (I)A.total, step = (I)gridDim.x * blockDim.x;
  // warps stay whole: `first` is the warp's first path
  for (I first = (I)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); first < total; first += step) {
    const I i = first + (threadIdx.x & 31);
    bool alive = i < total;
    const eos_path_record* rec = A.paths + (alive ? i : first);
    f3 o = mk3(0, 0, 0), d = mk3(0, 0, 1), campos = o;
    float g[3] = {0, 0, 0};
    if (alive) path_start<I>(A, i, o, d, campos, g);
    float T = 1.0f;
    for (int k = 0; k <= A.trace_depth; ++k) {
      int obj = -1;
      f3 P = o, N = o;
      const float* m = nullptr;
      uint32_t mask = 0;
      if (alive) {
        alive = replay_hit(A, __ldg(&rec->hit[k]), o, d, P, N, obj, m);
        mask = __ldg(&rec->shadow[k]);
      }
      if (!__any_sync(0xffffffffu, alive)) break;
      const float gT[3] = {g[0] * T, g[1] * T, g[2] * T};
      hit_adjoint(A, alive, P, N, obj, m, mask, campos, gT);
      if (alive) {
        f3 ro, rd;
        float w;
        if (k + 1 > A.trace_depth || !secondary_ray(m, s.ambient_index, d, P, N, ro, rd, w)) {
          alive = false;
        } else {
          T *= fold_weight(w);
          o = ro;
          d = rd;
        }
      }
    }
  }
  flush_sums(A);
}

// Tree records: a walk over each path's ray tree with a stack of pending rays (mirror
// child 2j + 1 with weight reflectivity, transparent child 2j + 2 with K + (1 - K)); one
// node per lane per step, so the warp reductions stay warp-uniform.
template <class I>
__global__ void __launch_bounds__(256, 4) k_backward_tree(BwArgs A) {
  clear_sums(A);
  struct Pending {
    f3 o, d;
    float T;
    int node, k;
  };
  const DevScene& s = A.s;
  const I total = (I)A.total, step = (I)gridDim.x * blockDim.x;
  for (I first = (I)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); first < total; first += step) {
    const I i = first + (threadIdx.x & 31);
    Pending st[kMaxBounces + 1];  // depth-first: at most one waiting sibling per bounce, plus the current
    int sp = 0;
    f3 campos = mk3(0, 0, 0);
    float g[3] = {0, 0, 0};
    const eos_tree_node* rec = nullptr;
    if (i < total) {
      f3 o, d;
      path_start<I>(A, i, o, d, campos, g);
      rec = A.tree + (size_t)i * A.nn;
      st[sp++] = Pending{o, d, 1.0f, 0, 0};
    }
    while (__any_sync(0xffffffffu, sp > 0)) {
      bool alive = sp > 0;
      Pending q;
      if (alive) q = st[--sp];
      int obj = -1;
      f3 P = q.o, N = q.o;
      const float* m = nullptr;
      if (alive) alive = replay_hit(A, rec[q.node].hit, q.o, q.d, P, N, obj, m);
      const float gT[3] = {g[0] * q.T, g[1] * q.T, g[2] * q.T};
      hit_adjoint(A, alive, P, N, obj, m, alive ? rec[q.node].shadow : 0u, campos, gT);
      if (alive && q.k + 1 <= A.trace_depth) {
        if (m[8] > 0.0f) {
          Pending c;
          const float K = transparent_ray(m, s.ambient_index, q.d, P, N, c.o, c.d);
          c.T = q.T * fold_weight(-K);
          c.node = 2 * q.node + 2;
          c.k = q.k + 1;
          st[sp++] = c;
        }
        if (m[7] > 0.0f) {
          Pending c;
          mirror_ray(q.d, P, N, c.o, c.d);
          c.T = q.T * m[7];
          c.node = 2 * q.node + 1;
          c.k = q.k + 1;
          st[sp++] = c;
        }
      }
    }
  }
  flush_sums(A);
}

}  // namespace

eos_status render_backward(eos_ctx* ctx, const eos_scene* sc, const eos_camera* cams, uint32_t n_views,
                           const eos_render_params& p, const void* d_paths, const float* d_rgb,
                           float* d_gmat, float* d_glight) {
  eos_status es = EOS_OK;
  float* d_cams = (float*)scratch(ctx, "bw.cams", 48ull * n_views, &es);
  if (es != EOS_OK) return es;
  std::vector<float>& hc = ctx->bw_cams;  // outlives the copy: the entry point waits for the call
  hc.resize(12 * (size_t)n_views);
  for (uint32_t v = 0; v < n_views; ++v)
    for (int k = 0; k < 3; ++k) {
      hc[12 * v + k] = cams[v].position[k];
      hc[12 * v + 3 + k] = cams[v].view[k];
      hc[12 * v + 6 + k] = cams[v].right[k];
      hc[12 * v + 9 + k] = cams[v].up[k];
    }
  EOS_CUDA(cudaMemcpyAsync(d_cams, hc.data(), hc.size() * 4, cudaMemcpyHostToDevice, ctx->stream));
  EOS_CUDA(cudaMemsetAsync(d_gmat, 0, 28ull * sc->dev.n_obj, ctx->stream));
  EOS_CUDA(cudaMemsetAsync(d_glight, 0, 24ull * std::max(1, sc->dev.n_lights), ctx->stream));
  BwArgs A;
  A.s = sc->dev;
  A.cams = d_cams;
  A.w = cams[0].width;
  A.h = cams[0].height;
  A.n_views = (int)n_views;
  A.trace_depth = p.trace_depth;
  A.y0 = p.row_end > 0 ? p.row_begin : 0;
  A.rows = p.row_end > 0 ? p.row_end - p.row_begin : A.h;
  A.spp = p.spp;
  A.seed = p.jitter_seed;
  A.grid = (p.flags & EOS_FLAG_AA_GRID) ? aa_grid_side(p.spp) : 0;
  A.off = p.pixel_offset;
  const bool tree = (p.flags & EOS_FLAG_TREE_RECORDS) != 0;
  A.paths = tree ? nullptr : (const eos_path_record*)d_paths;
  A.tree = tree ? (const eos_tree_node*)d_paths : nullptr;
  A.nn = EOS_TREE_NODES(p.trace_depth);
  A.drgb = d_rgb;
  A.gmat = d_gmat;
  A.glight = d_glight;
  A.err = ctx->d_err;
  A.total = (long long)A.w * A.rows * p.spp * n_views;
  // per-object sums in shared memory up to 32 KB a block (1,170 objects); beyond that each
  // warp's sums go to global memory
  const size_t light_bytes = 24ull * sc->dev.n_lights, obj_bytes = 28ull * sc->dev.n_obj;
  A.obj_shared = light_bytes + obj_bytes <= 32 * 1024;
  const size_t smem = light_bytes + (A.obj_shared ? obj_bytes : 0);
  const int block = 256;
  const long long blocks = (A.total + block - 1) / block;
  const bool narrow = A.total + (long long)ctx->num_sms * 8 * block < (1ll << 32);  // indices plus one step fit
  auto run = [&](auto* kernel) -> eos_status {
    int resident = 0;
    EOS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kernel, block, smem));
    const int grid = (int)std::min<long long>(blocks, (long long)ctx->num_sms * std::min(8, std::max(1, resident)));
    kernel<<<grid, block, smem, ctx->stream>>>(A);
    return EOS_OK;
  };
  const eos_status launched = tree ? (narrow ? run(k_backward_tree<uint32_t>) : run(k_backward_tree<unsigned long long>))
                                   : (narrow ? run(k_backward<uint32_t>) : run(k_backward<unsigned long long>));
  if (launched != EOS_OK) return launched;
  EOS_CUDA(cudaGetLastError());
  return EOS_OK;
}

}  // namespace eos
