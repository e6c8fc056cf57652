// PLOC hierarchy: parallel locally-ordered clustering (Meister & Bittner, "Parallel Locally-
// Ordered Clustering for Bounding Volume Hierarchy Construction", IEEE TVCG 2018), a second
// builder beside the Karras LBVH.  No reference counterpart (the reference builds a CPU
// SAH tree, src/BVH.cpp:97-111); it is a tree-quality choice only -- the traversal's
// results do not depend on the tree.
//
// Input: the leaf boxes in Morton order.  Clusters start as the leaves; each iteration
//   1. every cluster finds its nearest neighbour among the clusters within kRadius places
//      of it (distance = surface area of the merged box; ties to the lower index);
//   2. mutual nearest neighbours merge into a new interior node at the lower position;
//   3. the surviving clusters are compacted in order.
// One launch per iteration does all three (the blocks' tiles overlap by the search radius,
// and the compaction's offsets come from a look-back over the earlier tiles), and writes each
// new node whole: children, box, SAH cost and leaf decision, what the refit computes for the
// LBVH.  Interior nodes are numbered in creation order (deterministic: a scan of the kept
// clusters and made nodes, no atomics), the root last.  Afterwards the first leaf position
// in depth-first order (left subtree first) of every leaf and collapsed subtree is found by
// a walk to the root, so that every subtree covers a contiguous range of triangle records.
#include <algorithm>

#include "eos_internal.cuh"
#include "ring.cuh"
#include "scan.cuh"
#include "tree.cuh"

namespace eos {
namespace {

constexpr int kRadius = 16;        // neighbours searched on each side
// Clusters of one block's tile: one per thread over the tile and kRadius more on each side,
// whose nearest neighbours decide which pairs at the tile's ends are mutual.
constexpr int round_tile(int threads) { return threads - 2 * kRadius; }
constexpr int kTail = 1024;  // clusters at or below which one block runs the remaining rounds
constexpr int kMaxWalk = 4 * kStackMax;  // bound of the walks to the root

__device__ __forceinline__ float merged_area(float4 al, float4 ah, float4 bl, float4 bh) {
  const float dx = fmaxf(ah.x, bh.x) - fminf(al.x, bl.x);
  const float dy = fmaxf(ah.y, bh.y) - fminf(al.y, bl.y);
  const float dz = fmaxf(ah.z, bh.z) - fminf(al.z, bl.z);
  return dx * dy + dy * dz + dz * dx;
}

// Round state on the device: [0] clusters, [1] interior nodes made so far, [2] nodes made
// by the last round, [3] tickets taken by this round's blocks.  Rounds are launched ahead of
// the host, which reads the state back a few rounds later (build_ploc).
__global__ void k_ploc_state_init(int* __restrict__ state, int n, int* __restrict__ depth_max) {
  state[0] = n;
  state[1] = 0;
  state[2] = 1;
  for (int k = 3; k < 8; ++k) state[k] = 0;  // the other state: no clusters until a round writes it
  *depth_max = 0;
}

// The tree being built: creation-order ids (interior 0..n-2, root n-2; leaf at Morton
// position p: n-1+p).  up[v] = (parent, triangles of the left siblings below it); blo / bhi
// with the cost and leaf decision of join_boxes; count of interior nodes.
struct PlocTree {
  int n, max_leaf, sah;
  int2* child;
  int2* up;
  int* count;
  float4* blo;
  float4* bhi;
};

// Triangles below a cluster: in its hi.w; the first round's clusters (cid NULL) are the leaves.
__device__ __forceinline__ int cluster_count(const int* cid, float4 hi) { return cid ? __float_as_int(hi.w) : 1; }

// Writes node k = (a, b) and returns its box (lo.w its cost).
__device__ __forceinline__ void make_node(const PlocTree& T, int k, int a, int b, int ca, int cb, float4 al, float4 ah,
                                          float4 bl, float4 bh, float4& lo, float4& hi) {
  join_boxes(al, ah, bl, bh, ca + cb, T.max_leaf, T.sah, lo, hi);
  T.child[k] = make_int2(a, b);
  T.count[k] = ca + cb;
  T.up[a] = make_int2(k, 0);
  T.up[b] = make_int2(k, ca);
  T.blo[k] = lo;
  T.bhi[k] = hi;
}

// Partner of cluster i, -1 for none.  With `force` (an iteration that merged nothing) the
// pairs (2k, 2k + 1) merge instead of the mutual nearest neighbours, which bounds the number
// of iterations.
__device__ __forceinline__ int forced_partner(int i, int nc) { return (i & 1) ? i - 1 : (i + 1 < nc ? i + 1 : -1); }

// One iteration.  Bound by its serial chain and launches for most rounds (their cluster
// counts fall by about a fifth each), by the neighbour search for the first: threads 2u and
// 2u + 1 search for clusters 2u and 2u + 1 together, one over the boxes of even index, the other
// over the odd ones, so a box read from shared memory serves both clusters and the search is
// half as long (even and odd boxes lie apart, 64 bytes off in the banks: no conflicts).
// Places outside the clusters hold an infinite box, whose merged area is never below the
// best.  Measured against four launches an iteration (search, flags, scan of the block sums,
// merge) and a refit of the finished tree: builds of 20k and 1.06M triangles 1,240 -> 580 and
// 2,200 -> 1,210 us, node records included, with one thread searching for two clusters.
template <int kRoundThreads>
__global__ void __launch_bounds__(kRoundThreads) k_ploc_round(
    PlocTree T, int* __restrict__ state, int* __restrict__ state_out, int* __restrict__ slot, int number, int round,
    int force, int polls, unsigned long long* __restrict__ words, const int* __restrict__ cid, const float4* __restrict__ lo,
    const float4* __restrict__ hi, int* __restrict__ cid_out, float4* __restrict__ lo_out, float4* __restrict__ hi_out,
    int* err) {
  constexpr int kBoxes = kRoundThreads + 2 * kRadius, kRoundTile = round_tile(kRoundThreads);
  __shared__ float4 slo[2][kBoxes / 2 + 4], shi[2][kBoxes / 2 + 4];
  __shared__ int sid[kBoxes], snn[kRoundThreads];
  __shared__ int s_tile;
  __shared__ unsigned long long s_before;
  const int t = threadIdx.x;
  ring_wait();
  if (t == 0) s_tile = take_tile(&state[3], err);
  const int nc = state[0], node_base = state[1];
  __syncthreads();
  const int tile = s_tile;
  const int n_tiles = (nc + kRoundTile - 1) / kRoundTile;
  if (tile >= n_tiles) return;
  const int base = tile * kRoundTile;  // first cluster of the tile
  for (int e = t; e < kBoxes; e += kRoundThreads) {
    const int g = base - 2 * kRadius + e;
    const bool in = g >= 0 && g < nc;
    slo[e & 1][e >> 1] = in ? lo[g] : make_float4(-kInf, -kInf, -kInf, 0.0f);
    shi[e & 1][e >> 1] = in ? hi[g] : make_float4(kInf, kInf, kInf, 0.0f);
    sid[e] = !in ? 0 : cid ? cid[g] : T.n - 1 + g;
  }
  __syncthreads();
  const int i = base - kRadius + t;  // this thread's cluster
  const bool own = t >= kRadius && t < kRoundThreads - kRadius && i < nc;
  int p = -1;  // its partner
  if (!force) {
    constexpr int kMid = kRadius / 2;
    const int u = t >> 1, h = t & 1;
    const int i0 = base - kRadius + 2 * u;  // the pair's even cluster; box m is i0 - kRadius + 2 m + h
    const float4 al = slo[0][u + kMid], ah = shi[0][u + kMid], bl = slo[1][u + kMid], bh = shi[1][u + kMid];
    float best0 = kInf, best1 = kInf;
    int m0 = 0, m1 = 0;
    const int skip0 = h ? kRadius : kMid, skip1 = h ? kMid : 0;  // beyond kRadius, or the cluster itself
#pragma unroll 1
    for (int m = 0; m <= kRadius; ++m) {
      const float4 cl = slo[h][u + m], ch = shi[h][u + m];
      const float a0 = merged_area(al, ah, cl, ch), a1 = merged_area(bl, bh, cl, ch);
      if (m != skip0 && a0 < best0) { best0 = a0; m0 = m; }
      if (m != skip1 && a1 < best1) { best1 = a1; m1 = m; }
    }
    // the least (area, index) of the two threads
    int j0 = i0 - kRadius + 2 * m0 + h, j1 = i0 - kRadius + 2 * m1 + h;
    const float o0 = __shfl_xor_sync(0xffffffffu, best0, 1), o1 = __shfl_xor_sync(0xffffffffu, best1, 1);
    const int k0 = __shfl_xor_sync(0xffffffffu, j0, 1), k1 = __shfl_xor_sync(0xffffffffu, j1, 1);
    if (o0 < best0 || (o0 == best0 && k0 < j0)) { best0 = o0; j0 = k0; }
    if (o1 < best1 || (o1 == best1 && k1 < j1)) { best1 = o1; j1 = k1; }
    int j = h ? j1 : j0;
    if (!((h ? best1 : best0) < kInf)) j = i == 0 ? 1 : i - 1;
    snn[t] = j;
    __syncthreads();
    // mutual?  (a neighbour of a cluster of the tile lies within the searched ones)
    if (own && j < nc && snn[j - (base - kRadius)] == i) p = j;
  } else if (own) {
    p = forced_partner(i, nc);
  }
  const bool keep = own && (p < 0 || i < p), make = keep && p >= 0;
  int total;  // kept clusters (low half) and made nodes (high half)
  const int ex = block_exclusive_scan((int)keep | ((int)make << 16), total);
  if (t < 32) {
    const unsigned long long sum = (unsigned)(total & 0xffff) | ((unsigned long long)(total >> 16) << 25);
    const unsigned long long before = tiles_before(words, tile, sum, (unsigned)(round % 4095 + 1), polls);
    if (t == 0) s_before = before;
    if (t == 0 && tile == 0) state_out[3] = 0;
    if (t == 0 && tile == n_tiles - 1 && before <= kTileValue) {
      const unsigned long long all = before + sum;
      const int kept = (int)(all & 0x1ffffffu), made = (int)(all >> 25);
      state_out[0] = kept;
      state_out[1] = node_base + made;
      state_out[2] = made;
      ring_publish(slot, kept, node_base + made, made, number);
    }
  }
  __syncthreads();
  if (s_before > kTileValue) {  // an earlier tile did not publish its sum
    if (t == 0) atomicOr(err, kErrTimeout);
    return;
  }
  if (!keep) return;
  const int pos = (int)(s_before & 0x1ffffffu) + (ex & 0xffff);
  const int k = node_base + (int)(s_before >> 25) + (ex >> 16);
  const int e = t + kRadius;
  const float4 al = slo[e & 1][e >> 1], ah = shi[e & 1][e >> 1];
  int id = sid[e], cnt = cluster_count(cid, ah);
  float4 ol = al, oh = ah;
  if (make) {
    const int f = p - base + 2 * kRadius;
    const float4 bl = slo[f & 1][f >> 1], bh = shi[f & 1][f >> 1];
    const int cb = cluster_count(cid, bh);
    if (k < T.n - 1)  // always: n leaves make n - 1 nodes
      make_node(T, k, id, sid[f], cnt, cb, al, ah, bl, bh, ol, oh);
    id = k;
    cnt += cb;
  }
  cid_out[pos] = id;
  lo_out[pos] = ol;
  hi_out[pos] = make_float4(oh.x, oh.y, oh.z, __int_as_float(cnt));
}

// The rounds left once at most kTail clusters remain, in one block with the clusters in
// shared memory: the same neighbour search, pair rule, forced round after a round that
// merged nothing, and creation-order numbering as the per-round kernel, so the tree is
// the same; what it saves is the launches of the last ~30 rounds.  The rounds are a serial
// chain, so as clusters get fewer more threads (up to 32) share one cluster's search.
__global__ void __launch_bounds__(kTail) k_ploc_tail(PlocTree T, int* __restrict__ state, const int* __restrict__ cid_in,
                                                     const float4* __restrict__ lo_in, const float4* __restrict__ hi_in,
                                                     int* __restrict__ err) {
  // boxes with kRadius places on each side, which hold an infinite box (as those past the
  // last cluster): its merged area is never below the best, so the search checks no range
  __shared__ float4 slo_[kTail + 2 * kRadius], shi_[kTail + 2 * kRadius];
  __shared__ int scid[kTail], scount[kTail], snn[kTail];
  __shared__ int wsum[kTail / 32];
  float4 *const slo = slo_ + kRadius, *const shi = shi_ + kRadius;
  const float4 out_lo = make_float4(-kInf, -kInf, -kInf, 0.0f), out_hi = make_float4(kInf, kInf, kInf, 0.0f);
  const int i = threadIdx.x, lane = i & 31, warp = i >> 5;
  if (*err & kErrTimeout) return;  // a round gave up: its clusters are not complete
  int nc = state[0], node_base = state[1];
  int force = state[2] == 0 && nc > 1;  // the last round merged nothing: the forced round is next
  if (nc > kTail) {  // the host launches this only at or below kTail
    if (i == 0) atomicOr(err, kErrIndex);
    return;
  }
  if (i < nc) {
    slo[i] = lo_in[i];
    shi[i] = hi_in[i];
    scid[i] = cid_in ? cid_in[i] : T.n - 1 + i;
    scount[i] = cluster_count(cid_in, shi[i]);
  } else {
    slo[i] = out_lo;
    shi[i] = out_hi;
  }
  if (i < kRadius) {
    slo_[i] = slo[kTail + i] = out_lo;
    shi_[i] = shi[kTail + i] = out_hi;
  }
  __syncthreads();
  int iters = 0;
  while (nc > 1) {
    if (++iters > 4 * kTail + 8) {  // cannot happen: every round or its forced repeat merges
      if (i == 0) atomicOr(err, kErrTimeout);
      break;
    }
    if (!force) {
      // 2^lg threads per cluster, each every 2^lg-th of its 32 neighbours (the threads of a warp
      // read neighbouring boxes: no bank conflicts); the least (area, index)
      const int lg = nc > 512 ? 0 : nc > 256 ? 1 : nc > 128 ? 2 : nc > 48 ? 3 : nc > 16 ? 4 : 5;
      const int c = i >> lg, g = i & ((1 << lg) - 1);
      if ((i & ~31) >> lg < nc) {  // warps without a cluster wait
        float best = kInf;
        int bj = kTail;
        const float4 al = slo[c], ah = shi[c];  // c past nc in the last warp: an infinite box
#pragma unroll 4
        for (int w = g; w < 2 * kRadius; w += 1 << lg) {
          const int j = c - kRadius + w + (w >= kRadius);  // all places but c
          const float a = merged_area(al, ah, slo[j], shi[j]);
          if (a < best) {
            best = a;
            bj = j;
          }
        }
        for (int off = 1; off < (1 << lg); off <<= 1) {
          const float o = __shfl_xor_sync(0xffffffffu, best, off);
          const int oj = __shfl_xor_sync(0xffffffffu, bj, off);
          if (o < best || (o == best && oj < bj)) {
            best = o;
            bj = oj;
          }
        }
        if (c < nc && g == 0) snn[c] = best < kInf ? bj : (c == 0 ? 1 : c - 1);
      }
    }
    __syncthreads();
    const bool works = warp * 32 < nc;  // warps with clusters: the others only wait
    const int n_warps = (nc + 31) >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    int partner = -1;
    bool keep = false, make = false;
    uint32_t kb = 0, mb = 0;
    if (works) {
      if (i < nc) {
        if (force) {
          partner = forced_partner(i, nc);
        } else {
          const int j = snn[i];
          partner = j < nc && snn[j] == i ? j : -1;
        }
      }
      keep = i < nc && (partner < 0 || i < partner);
      make = keep && partner >= 0;
      kb = __ballot_sync(0xffffffffu, keep);
      mb = __ballot_sync(0xffffffffu, make);
      if (lane == 0) wsum[warp] = __popc(kb) | (__popc(mb) << 16);
    }
    __syncthreads();
    unsigned total = 0;
    for (int w = lane; w < n_warps; w += 32) total = wsum[w];
    int pos = 0, id = 0, cnt = 0;
    float4 ol = out_lo, oh = out_hi;
    if (works) {
      const unsigned before = __reduce_add_sync(0xffffffffu, lane < warp ? total : 0u);
      pos = (int)(before & 0xffff) + __popc(kb & lt);
      if (keep) {
        id = scid[i];
        cnt = scount[i];
        ol = slo[i];
        oh = shi[i];
        if (make) {
          const int k = node_base + (int)(before >> 16) + __popc(mb & lt);
          const float4 al = ol, ah = oh;
          const int cb = scount[partner];
          if (k < T.n - 1)  // always: n leaves make n - 1 nodes
            make_node(T, k, id, scid[partner], cnt, cb, al, ah, slo[partner], shi[partner], ol, oh);
          id = k;
          cnt += cb;
        }
      }
    }
    total = __reduce_add_sync(0xffffffffu, total);
    __syncthreads();  // every read of this round's clusters is done
    if (keep) {
      scid[pos] = id;
      scount[pos] = cnt;
      slo[pos] = ol;
      shi[pos] = oh;
    }
    const int made = (int)(total >> 16), kept = (int)(total & 0xffff);
    if (i >= kept && i < nc) {
      slo[i] = out_lo;
      shi[i] = out_hi;
    }
    node_base += made;
    nc = kept;
    force = made == 0 && !force;
    __syncthreads();
  }
  if (i == 0) {
    state[0] = nc;
    state[1] = node_base;
  }
}

// Depth-first position of the first triangle of every leaf (perm[p], by Morton position) and
// of every collapsed subtree (first[v]): the sum of the left siblings' counts on the way to
// the root.  A too deep tree is reported as deeper than kMaxWalk, an unfinished one (a round
// gave up) as kUnfinished.
constexpr int kUnfinished = kMaxWalk + 2;
__global__ void k_ploc_positions(PlocTree T, const int* __restrict__ state, int* __restrict__ first,
                                 uint32_t* __restrict__ perm, int* __restrict__ depth_max,
                                 const int* __restrict__ err) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = T.n;
  int steps = 0;
  if (state[1] != n - 1 || (*err & kErrTimeout)) {
    steps = kUnfinished;
  } else if (v >= n - 1 ? v < 2 * n - 1 : T.bhi[v].w != 0.0f) {
    int pos = 0, node = v;
    while (node != n - 2 && steps <= kMaxWalk) {
      const int2 u = T.up[node];
      pos += u.y;
      node = u.x;
      ++steps;
    }
    if (v < n - 1) first[v] = pos;
    else perm[v - (n - 1)] = (uint32_t)pos;
  }
  const int deepest = __reduce_max_sync(0xffffffffu, steps);
  if ((threadIdx.x & 31) == 0 && deepest > *(volatile int*)depth_max) atomicMax(depth_max, deepest);
}

inline int grid_of(long long n, int block) { return (int)std::max<long long>(1, (n + block - 1) / block); }

}  // namespace

// Builds the hierarchy over n >= 2 leaves whose boxes lie at blo / bhi[n-1+p] (Morton
// position p; .w of lo and hi 1), in creation-order ids: child, count, box, cost and leaf
// decision of every interior node, perm[p] = the record position of Morton position p and
// first[v] = that of a collapsed subtree's first triangle.  *depth = the deepest node's
// depth; above 4 * kStackMax first and perm are not complete and the caller must use another
// builder.  EOS_ERR_TIMEOUT when a round gave up: nothing may be read then.
eos_status build_ploc(eos_ctx* ctx, int n, int max_leaf, int sah, float4* blo, float4* bhi, int2* child, int* count,
                      int* first, uint32_t* perm, int* depth) {
  cudaStream_t st = ctx->stream;
  eos_status es = EOS_OK;
  const size_t nn = (size_t)n;
  int* cid[2] = {(int*)scratch(ctx, "ploc.cid0", 4 * nn, &es), (int*)scratch(ctx, "ploc.cid1", 4 * nn, &es)};
  float4* clo[2] = {(float4*)scratch(ctx, "ploc.lo0", 16 * nn, &es), (float4*)scratch(ctx, "ploc.lo1", 16 * nn, &es)};
  float4* chi[2] = {(float4*)scratch(ctx, "ploc.hi0", 16 * nn, &es), (float4*)scratch(ctx, "ploc.hi1", 16 * nn, &es)};
  // Blocks of 512 threads, and of 256 once those are fewer than the SMs: the search is then a
  // shorter part of the round on more of them.
  const int small_max = round_tile(256) * ctx->num_sms;
  const size_t words_bytes = 8 * (size_t)std::max(grid_of(n, round_tile(512)), ctx->num_sms);
  unsigned long long* words = (unsigned long long*)scratch(ctx, "ploc.words", words_bytes, &es);
  int2* up = (int2*)scratch(ctx, "ploc.up", 8 * (2 * nn), &es);
  int* state = (int*)scratch(ctx, "ploc.state", 64, &es);  // two states, by round parity, and the depth
  if (es != EOS_OK) return es;
  int* dmax = state + 8;
  const PlocTree T{n, max_leaf, sah, child, up, count, blo, bhi};
  // Rounds run ahead of the host until at most kTail clusters are left (k_ploc_tail does the
  // rest): grids are sized by an upper bound of the cluster count
  // (the last one read back; it only falls), and the host reads each round's state
  // RoundRing::kAhead rounds later instead of waiting after every round.  A round that merges nothing
  // changes nothing, so the rounds queued behind one repeat it harmlessly; when the host
  // sees it, it waits for the queue and runs the forced round (as a synchronous loop
  // would right away), so the tree is the same.
  RoundRing ring(ctx);
  if ((es = ring.init()) != EOS_OK) return es;
  EOS_CUDA(cudaMemsetAsync(words, 0, words_bytes, st));
  k_ploc_state_init<<<1, 1, 0, st>>>(state, n, dmax);
  int nc_ub = n, cur = 0;
  bool small = nc_ub <= small_max;
  auto enqueue = [&](int force) {
    const int r = (int)ring.issued;
    if (!small && nc_ub <= small_max) {  // other tiles from here on
      small = true;
      EOS_CUDA(cudaMemsetAsync(words, 0, words_bytes, st));
    }
    const int threads = small ? 256 : 512;
    // the first round's clusters are the leaf boxes themselves
    const eos_status st_l = ring.launch(
        small ? k_ploc_round<256> : k_ploc_round<512>, grid_of(nc_ub, round_tile(threads)), threads, T,
        state + 4 * cur, state + 4 * (cur ^ 1), ring.next_slot(), ring.next_number(), r, force, ctx->build_polls, words,
        r ? cid[cur] : nullptr, r ? clo[cur] : blo + (n - 1), r ? chi[cur] : bhi + (n - 1), cid[cur ^ 1],
        clo[cur ^ 1], chi[cur ^ 1], ctx->d_err);
    cur ^= 1;
    return st_l;
  };
  for (;;) {
    if (nc_ub > kTail && ring.full()) {  // read the oldest round in flight
      int s[3];
      if ((es = ring.read(s)) != EOS_OK) return es;
      nc_ub = std::min(nc_ub, s[0]);
      if (nc_ub <= 1) break;
      if (s[2] == 0) {  // stalled: drain, then the forced round
        EOS_CUDA(cudaStreamSynchronize(st));
        if ((es = enqueue(1)) != EOS_OK) return es;
        while (!ring.empty())
          if ((es = ring.read(s)) != EOS_OK) return es;
        nc_ub = std::min(nc_ub, s[0]);
        if (nc_ub <= 1) break;
      }
    }
    if (nc_ub <= kTail) {  // the rest in one block, behind the rounds in flight
      const bool any = ring.issued > 0;
      k_ploc_tail<<<1, kTail, 0, st>>>(T, state + 4 * cur, any ? cid[cur] : nullptr, any ? clo[cur] : blo + (n - 1),
                                       any ? chi[cur] : bhi + (n - 1), ctx->d_err);
      break;
    }
    if (ring.issued > 4ll * n + 8) return EOS_ERR_TIMEOUT;  // cannot happen: every round or its forced repeat merges
    if ((es = enqueue(0)) != EOS_OK) return es;
  }
  k_ploc_positions<<<grid_of(2 * (long long)n - 1, 256), 256, 0, st>>>(T, state + 4 * cur, first, perm, dmax,
                                                                       ctx->d_err);
  EOS_CUDA(cudaMemcpyAsync(depth, dmax, 4, cudaMemcpyDeviceToHost, st));
  EOS_CUDA(cudaStreamSynchronize(st));
  return *depth == kUnfinished ? EOS_ERR_TIMEOUT : EOS_OK;
}

}  // namespace eos
