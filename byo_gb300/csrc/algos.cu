// algos.cu -- connectivity and PageRank over the shared graph view (d_off /
// d_slots with kSentinel gaps / d_deg).
//
// Connectivity (SimpleUnionAsync semantics, Connectivity.h:32-136): union-find
// that always hooks the larger root under the smaller, so every root is the
// minimum id of its component.  Edges are processed Afforest-style
// (Sutton, Ben-Nun & Barak, IPDPS 2018): join every vertex to its first
// kSample neighbours, compress, pick the most frequent root among sampled vertices,
// then link the remaining edges of vertices outside that component only.  The
// final labels do not depend on the order of links.
//
// PageRank (PageRank.h:125-193): Jacobi pull over warp-sized work units,
// FP32 state with compensated (TwoSum) per-vertex sums, FP64 L1 residual.
// Bytes per iteration: 4 B per slot (ids) + 4 B per slot (p_div gather) +
// 16 B offsets/degrees + 12 B state per vertex.
#include <algorithm>
#include <cmath>
#include <vector>

#include "device.cuh"
#include "engine.h"
#include "gridsync.cuh"
#include "internal.h"
#include "scan.cuh"

namespace byo {

// ================================================================ connectivity

constexpr int kSample = 2;  // cc_run's two rounds

__device__ __forceinline__ uint32_t ld_parent(const uint32_t *p, uint32_t v) { return __ldcg(p + v); }

// Root of v, whose parent is `cur`; parents only ever point to smaller ids.  With
// kShorten the entries read on the way are pointed at ancestors: v's own at the
// root, and the others by path halving from the kPlainHops-th step on, which a
// chain needs.  Halving at every step, all vertices of a large tree store into the
// few entries below its root, and stores and loads of one word take turns at the L2,
// about one a ns (second round of a uniform graph of 1 M vertices, average degree 1.6:
// 0.4 to 1.6 ms halving at every step, the whole labelling 0.4 ms now).  kFar: where
// the parents are far larger than the L2 a step waits for memory instead, and
// halving at every step, with no other store, is the faster (see cc_run).
constexpr int kPlainHops = 16;
template <bool kShorten = true, bool kFar = false>
__device__ __forceinline__ uint32_t cc_find(uint32_t *p, uint32_t v, uint32_t cur) {
  if (cur == v) return v;
  uint32_t prev = v, next;
  int hops = 0;
  while (cur > (next = ld_parent(p, cur))) {
    if (kShorten && (++hops > kPlainHops || kFar)) p[prev] = next;
    prev = cur;
    cur = next;
  }
  if (kShorten && !kFar && hops) p[v] = cur;
  return cur;
}

// Hook the larger root under the smaller until both share a root.  Equal parents
// end it before the roots, which are the words all threads read, are touched
// (`equal`: worth looking).
template <bool kFar = false>
__device__ __forceinline__ void cc_link(uint32_t *p, uint32_t u, uint32_t v, bool equal = true) {
  const uint32_t pu = ld_parent(p, u), pv = ld_parent(p, v);
  if (equal && pu == pv) return;
  uint32_t ru = cc_find<true, kFar>(p, u, pu), rv = cc_find<true, kFar>(p, v, pv);
  while (ru != rv) {
    uint32_t hi = ru > rv ? ru : rv, lo = ru > rv ? rv : ru;
    uint32_t old = atomicCAS(p + hi, hi, lo);
    if (old == hi) return;
    // hi got a parent meanwhile: continue from the new roots
    ru = cc_find<true, kFar>(p, old, ld_parent(p, old));
    rv = cc_find<true, kFar>(p, lo, ld_parent(p, lo));
  }
}

// The round-th neighbour of v (kSentinel: it has fewer).
__device__ __forceinline__ uint32_t cc_sampled(const uint64_t *__restrict__ off, const uint32_t *__restrict__ slots,
                                               uint64_t v, int round) {
  const uint64_t b = off[v], e = off[v + 1];
  if (b + round >= e) return kSentinel;  // fewer than round + 1 slots
  // slots b .. b + round: the sampled neighbour is the last when none is a
  // gap (always, on a compact CSR)
  uint32_t x = kSentinel;
  bool gap = false;
  for (int r = 0; r <= round; r++) {
    x = slots[b + r];
    gap |= x == kSentinel;
  }
  if (!gap) return x;
  int taken = 0;  // a gapped view: the round-th neighbour past the gaps
  for (uint64_t j = b; j < e; j++) {
    const uint32_t y = slots[j];
    if (y != kSentinel && taken++ == round) return y;
  }
  return kSentinel;
}

// The first sampling round: every vertex under its first neighbour where that
// is smaller, by one store.  The edges to larger ones are left to k_cc_sample.
__global__ void k_cc_first(const uint64_t *__restrict__ off, const uint32_t *__restrict__ slots, uint32_t *p,
                           uint64_t n) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x)
    p[v] = min((uint32_t)v, cc_sampled(off, slots, v, 0));  // kSentinel (no neighbour) is larger than v
}

// What the first round left: the edges to a larger first neighbour, then every
// vertex to its second.
// (kFar: *few, whether few of the parents are equal.)
template <bool kFar>
__global__ void k_cc_sample(const uint64_t *__restrict__ off, const uint32_t *__restrict__ slots,
                            uint32_t *p, uint64_t n, const unsigned long long *few) {
  const bool equal = !kFar || !*few;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t x = cc_sampled(off, slots, v, 0);
    if (x == kSentinel) continue;
    if (x > v) cc_link<kFar>(p, (uint32_t)v, x, equal);
    const uint32_t y = cc_sampled(off, slots, v, 1);
    if (y != kSentinel) cc_link<kFar>(p, (uint32_t)v, y, equal);
  }
}

// v to its root, by pointer jumping.  Only v's thread writes p[v]: a store into
// another vertex's entry could land after its own thread wrote its root there,
// and leave a stale ancestor behind the last pass.  Every step is stored, for
// the first round may leave chains as long as the graph (a path, a grid's
// columns), and the threads on a chain halve it together.
__device__ __forceinline__ uint32_t cc_compress(uint32_t *p, uint32_t v) {
  uint32_t cur = ld_parent(p, v), next = ld_parent(p, cur);
  while (next != cur) {
    __stcg(p + v, next);
    cur = next;
    next = ld_parent(p, cur);
  }
  return cur;
}
__global__ void k_cc_compress(uint32_t *p, uint64_t n) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x)
    cc_compress(p, (uint32_t)v);
}

// The vertex that probe i of a fixed hash draws.
__device__ __forceinline__ uint32_t cc_probe(uint64_t n, uint32_t i) {
  uint64_t z = 0x5EEDull + (uint64_t)(i + 1) * 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (uint32_t)(((z & 0xFFFFFFFFull) * n) >> 32);
}
// The most frequent root among a warp's (ties: the smallest).
__device__ __forceinline__ uint32_t cc_mode(uint32_t root) {
  const uint32_t same = __popc(__match_any_sync(kFull, root));
  const uint32_t most = __reduce_max_sync(kFull, same);
  return __reduce_min_sync(kFull, same == most ? root : kSentinel);
}

// The compress between the rounds, then hooking passes over the edges to the
// second neighbours where they pay (see cc_run), a compress after each: the
// larger parent of an edge's ends goes under the smaller, by one atomicMin and no
// search.  At the start of a pass every parent is a root, and only roots get a
// new one, so what was joined before stays joined.  A root that two edges
// lower keeps the lower one, so a pass can lose the other edge's union; the
// linking that follows makes it again, so the passes only prepare, and a grid
// barrier that gave up would end them early and nothing else.  Parents stay
// below their children throughout.  One cooperative kernel: where the passes are
// not wanted it costs a barrier.
__device__ __forceinline__ void cc_hook(uint32_t *p, uint32_t v, uint32_t x) {
  const uint32_t pv = ld_parent(p, v), px = ld_parent(p, x);
  const uint32_t hi = max(pv, px), lo = min(pv, px);
  if (hi != lo && ld_parent(p, hi) > lo) atomicMin(p + hi, lo);
}
// Three passes: two are 10% faster on skewed graphs and up to 1.7x slower on uniform
// ones (1 M vertices of degree 2: 417 against 240 us), four are 3 to 10% slower.
constexpr int kCcHookBlock = 1024, kCcHooks = 3;
constexpr uint64_t kCcHookLeast = 1 << 15;
constexpr uint64_t kCcFar = 1 << 24;  // 64 MB of parents
__global__ void __launch_bounds__(kCcHookBlock, 2) k_cc_hook(const uint64_t *__restrict__ off,
                                                             const uint32_t *__restrict__ slots,
                                                             const uint32_t *__restrict__ deg, uint32_t *p, uint64_t n,
                                                             unsigned long long *trees, unsigned long long *few,
                                                             int passes, GridBar *bar) {
  __shared__ unsigned int sm[kCcHookBlock / 32 + 1];
  __shared__ uint32_t cand;
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, nthr = (uint64_t)gridDim.x * blockDim.x;
  unsigned int mine = 0;
  for (uint64_t v = tid; v < n; v += nthr) mine += cc_compress(p, (uint32_t)v) == (uint32_t)v && deg[v];
  mine = block_sum(mine, sm);
  if (threadIdx.x == 0 && mine) atomicAdd(trees, (unsigned long long)mine);
  if (!grid_sync(bar, gridDim.x)) return;
  if (__ldcg(trees) * 256 <= n) return;
  const uint32_t probe = cc_probe(n, threadIdx.x), root = ld_parent(p, probe);
  if (threadIdx.x < 32) {
    const uint32_t c = cc_mode(root);
    if (threadIdx.x == 0) cand = c;
  }
  __syncthreads();
  const int joined = __syncthreads_count(deg[probe] != 0);
  if (__syncthreads_count(root == cand) * 5 >= joined) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) *few = 1;
  if (!passes || !grid_sync(bar, gridDim.x)) return;  // every block has probed
  for (int pass = 0; pass < passes; pass++) {
    for (uint64_t v = tid; v < n; v += nthr) {
      const uint32_t x = cc_sampled(off, slots, v, 0);
      if (x == kSentinel) continue;
      if (x > v) cc_hook(p, (uint32_t)v, x);
      const uint32_t y = cc_sampled(off, slots, v, 1);
      if (y != kSentinel) cc_hook(p, (uint32_t)v, y);
    }
    if (!grid_sync(bar, gridDim.x)) return;
    for (uint64_t v = tid; v < n; v += nthr) cc_compress(p, (uint32_t)v);
    if (!grid_sync(bar, gridDim.x)) return;
  }
}

// Every vertex to its root, and the list of those whose remaining edges must be
// linked: more than kSample neighbours (the first kSample are linked by the
// sampling rounds) and a root other than the giant component's, the most
// frequent one among 32 probes (links are over, so every block finds the same).
// A vertex inside the giant component is skipped entirely: each of its
// neighbours outside it will link the edge from its own side, and roots only
// merge, so a vertex found inside stays inside.
__global__ void __launch_bounds__(256) k_cc_outside(const uint32_t *__restrict__ deg, uint32_t *p, uint64_t n,
                                                    uint32_t *list, unsigned long long *count) {
  __shared__ uint32_t giant;
  if (threadIdx.x < 32) {
    const uint32_t v = cc_probe(n, threadIdx.x), c = cc_mode(cc_find<false>(p, v, ld_parent(p, v)));
    if (threadIdx.x == 0) giant = c;
  }
  __syncthreads();
  for (uint64_t base = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) & ~31ull; base < n;
       base += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t v = base + lane_id();
    const bool keep = v < n && cc_compress(p, (uint32_t)v) != giant && deg[v] > (uint32_t)kSample;
    const uint64_t at = warp_append(keep, count);
    if (keep) list[at] = (uint32_t)v;
  }
}

// Remaining edges of the listed vertices, GS lanes per vertex.
template <int GS>
__global__ void __launch_bounds__(256) k_cc_finish(const uint64_t *__restrict__ off,
                                                   const uint32_t *__restrict__ slots, uint32_t *p,
                                                   const uint32_t *__restrict__ list,
                                                   const unsigned long long *__restrict__ count) {
  const uint64_t nl = *count;
  const unsigned gl = threadIdx.x % GS;
  const uint64_t gid = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / GS;
  const uint64_t ng = ((uint64_t)gridDim.x * blockDim.x) / GS;
  for (uint64_t t = gid; t < nl; t += ng) {
    const uint32_t v = list[t];
    const uint64_t b = off[v], e = off[v + 1];
    // skip the first kSample non-gap neighbours: already linked
    uint64_t start = b;
    for (int taken = 0; start < e && taken < kSample; start++)
      if (slots[start] != kSentinel) taken++;
    for (uint64_t j = start + gl; j < e; j += GS) {
      uint32_t u = slots[j];
      if (u == kSentinel) continue;
      cc_link(p, v, u);
    }
  }
}

int cc_run(byo_graph *g, uint32_t *d_label) {
  byo_ctx *ctx = g->ctx;
  const uint64_t n = g->n;
  if (n == 0) return BYO_OK;
  uint32_t *p = d_label;
  const dim3 grid_v(grid_for(ctx, n, 256));
  uint32_t *words = nullptr, *list = nullptr;
  // [0..1] count of listed vertices, [2..3] trees, [4..5] whether no tree holds
  // much, then the barrier
  BYO_TRY(ws(g, WS_MISC, 6 + sizeof(GridBar) / 4, &words));
  BYO_TRY(ws(g, WS_FRONT_LIST_A, n, &list));
  unsigned long long *count = reinterpret_cast<unsigned long long *>(words), *trees = count + 1, *few = count + 2;
  GridBar *bar = reinterpret_cast<GridBar *>(words + 6);
  BYO_CU(ctx, cudaMemsetAsync(words, 0, 24 + sizeof(GridBar), ctx->stream));
  const uint64_t *off = g->d_off;
  const uint32_t *slots = g->d_slots, *deg = g->d_deg;
  launch(ctx, k_cc_first, grid_v, dim3(256), 0, off, slots, p, n);
  // Where no tree of the first round holds much, the second round's links wait for
  // one another on a few growing trees, and hooking passes first leave them little
  // to join: uniform graphs of average degree 16, 40000 / 300007 / 4 M vertices,
  // 186 / 829 / 1529 us without and 76 / 149 / 969 with them; RMAT with permuted
  // ids, 2^17 / 2^22 vertices, 116 / 1881 and 79 / 501.  Where hubs gather the
  // trees (k_cc_hook sees one of a fifth of the vertices with neighbours or more; of
  // all vertices, RMAT 2^22 with 2^22 draws, half of them alone, took 311 us instead of
  // 222) they made it 1.3 to 2x slower, so
  // there the kernel only compresses, 4 to 8 us slower than k_cc_compress, which
  // smaller graphs keep (uniform, 10007: 68 us either way).  Nor do they pay below
  // an average degree of 1.6, where the trees stay small: 300007 vertices, degree
  // 1.2 / 1.5 / 1.7: 82 / 162 / 140 us without, 116 / 132 / 132 with.
  // Nor on uniform graphs whose parents are far larger than the L2, for each pass
  // gathers two of them a vertex from memory, and the links, halving at every step,
  // few: 2^24 / 2^25 / 2^26 vertices of degree 16 3.7 / 6.7 / 13.5 ms with the passes and
  // 2.8 / 3.6 / 6.8 without; of degree 12 2.9 / 5.4 / 10.8 and 4.7 / 3.6 / 8.0, of degree 8
  // 2.2 / 4.2 / 9.1 and 5.0 / 4.0 / 10.8.  There the kernel tells whether the links look
  // for equal parents first: uniform 2^26 of degree 16 7.9 ms with and 6.8 without,
  // RMAT 2^26 of degree 32 4.0 and 4.8.
  const bool far = n >= kCcFar && g->m >= (n < 2 * kCcFar ? 15 : 11) * n;
  if (n < kCcHookLeast || 5 * g->m < 8 * n) {
    launch(ctx, k_cc_compress, grid_v, dim3(256), 0, p, n);
  } else {
    int per_sm = 0, passes = far ? 0 : kCcHooks;
    BYO_CU(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cc_hook, kCcHookBlock, 0));
    void *args[] = {(void *)&off,   (void *)&slots, (void *)&deg,    (void *)&p,  (void *)&n,
                    (void *)&trees, (void *)&few,   (void *)&passes, (void *)&bar};
    BYO_CU(ctx, cudaLaunchCooperativeKernel((const void *)k_cc_hook, dim3(per_sm * ctx->num_sms), dim3(kCcHookBlock),
                                            args, 0, ctx->stream));
    ctx->launches++;
  }
  launch(ctx, far ? k_cc_sample<true> : k_cc_sample<false>, grid_v, dim3(256), 0, off, slots, p, n,
         (const unsigned long long *)few);
  launch(ctx, k_cc_outside, dim3(grid_for(ctx, n, 256)), dim3(256), 0, deg, p, n, list, count);
  const double avg = (double)g->m / (double)n;
  const int GS = avg >= 24 ? 16 : avg >= 8 ? 8 : 4;
  const int grid = grid_for(ctx, n * GS, 256, 16);
  if (GS == 16)
    launch_t(ctx, "cc_finish", k_cc_finish<16>, dim3(grid), dim3(256), 0, (const uint64_t *)g->d_off,
             (const uint32_t *)g->d_slots, p, (const uint32_t *)list, (const unsigned long long *)count);
  else if (GS == 8)
    launch_t(ctx, "cc_finish", k_cc_finish<8>, dim3(grid), dim3(256), 0, (const uint64_t *)g->d_off,
             (const uint32_t *)g->d_slots, p, (const uint32_t *)list, (const unsigned long long *)count);
  else
    launch_t(ctx, "cc_finish", k_cc_finish<4>, dim3(grid), dim3(256), 0, (const uint64_t *)g->d_off,
             (const uint32_t *)g->d_slots, p, (const uint32_t *)list, (const unsigned long long *)count);
  launch(ctx, k_cc_compress, grid_v, dim3(256), 0, p, n);
  return check_launch(ctx, "cc");
}

// ---------------------------------------------------------------- BFS-CC

__global__ void k_bfscc_isolated(const uint32_t *__restrict__ deg, uint64_t n, uint32_t *label) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x)
    label[v] = deg[v] == 0 ? (uint32_t)v : kSentinel;
}

__global__ void k_bfscc_first_unlabeled(const uint32_t *__restrict__ label, uint64_t n,
                                        unsigned int *out) {
  uint32_t best = kSentinel;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x)
    if (label[v] == kSentinel) {
      best = (uint32_t)v;
      break;  // grid-stride order: first hit per thread is its smallest
    }
  if (best != kSentinel) atomicMin(out, best);
}

// label every vertex reached by the traversal (lp set) that has no label yet
__global__ void k_bfscc_assign(const uint64_t *__restrict__ lp, uint64_t n, uint32_t src,
                               uint32_t *label) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x)
    if (label[v] == kSentinel && lp[v] != kNone64) label[v] = src;
}

__global__ void k_trav_seed(uint64_t *lp, uint32_t *visited, uint32_t src) {
  lp[src] = src;
  atomicOr(visited + (src >> 5), 1u << (src & 31));
}

int bfs_cc_run(byo_graph *g, uint32_t *d_label) {
  // BFSCC/Connectivity.h:57-88: components in order of their smallest vertex,
  // one edgeMap traversal each; isolated vertices label themselves.  After
  // kMaxBfs traversals the remaining (small) components are finished by the
  // union-find pass, whose labels (component minimum) are the same.
  byo_ctx *ctx = g->ctx;
  const uint64_t n = g->n, W = (n + 31) / 32;
  if (n == 0) return BYO_OK;
  constexpr int kMaxBfs = 64;
  TravState st;
  Frontier fa, fb;
  BYO_TRY(ws(g, WS_LP, n, &st.lp));
  BYO_TRY(ws(g, WS_VISITED, W, &st.visited));
  BYO_TRY(ws(g, WS_FRONT_LIST_A, n, &fa.list));
  BYO_TRY(ws(g, WS_FRONT_LIST_B, n, &fb.list));
  BYO_TRY(ws(g, WS_FRONT_BITS_A, W, &fa.bits));
  BYO_TRY(ws(g, WS_FRONT_BITS_B, W, &fb.bits));
  unsigned int *d_first = nullptr;
  BYO_TRY(ws(g, WS_MISC, 4, (uint32_t **)&d_first));
  launch(ctx, k_bfscc_isolated, dim3(grid_for(ctx, n, 256)), dim3(256), 0, (const uint32_t *)g->d_deg, n,
         d_label);
  BYO_TRY(trav_init(g, st, 0));
  // start from an empty traversal state: no vertex visited
  BYO_CU(ctx, cudaMemsetAsync(st.lp, 0xFF, n * 8, ctx->stream));
  BYO_CU(ctx, cudaMemsetAsync(st.visited, 0, W * 4, ctx->stream));
  BYO_TRY(memset_async(ctx, fa.bits, 0, W * 4));
  BYO_TRY(memset_async(ctx, fb.bits, 0, W * 4));
  const EngineTuning tune = default_tuning(g);
  uint32_t *h = nullptr;
  BYO_TRY(pinned(ctx, 4096, (void **)&h));
  for (int it = 0; it < kMaxBfs; it++) {
    BYO_CU(ctx, cudaMemsetAsync(d_first, 0xFF, 4, ctx->stream));
    launch(ctx, k_bfscc_first_unlabeled, dim3(grid_for(ctx, n, 256)), dim3(256), 0,
           (const uint32_t *)d_label, n, d_first);
    BYO_CU(ctx, cudaMemcpyAsync(h, d_first, 4, cudaMemcpyDeviceToHost, ctx->stream));
    BYO_CU(ctx, cudaStreamSynchronize(ctx->stream));
    const uint32_t s = h[0];
    if (s == kSentinel) return check_launch(ctx, "bfs_cc");
    launch(ctx, k_trav_seed, dim3(1), dim3(1), 0, st.lp, st.visited, s);
    BYO_CU(ctx, cudaMemcpyAsync(fa.list, &s, 4, cudaMemcpyHostToDevice, ctx->stream));
    BYO_TRY(memset_async(ctx, fa.bits, 0, W * 4));
    BYO_TRY(memset_async(ctx, fb.bits, 0, W * 4));
    uint32_t ds = 0;
    BYO_CU(ctx, cudaMemcpyAsync(&ds, g->d_deg + s, 4, cudaMemcpyDeviceToHost, ctx->stream));
    BYO_CU(ctx, cudaStreamSynchronize(ctx->stream));
    fa.size = 1;
    fa.outdeg = ds;
    fa.dense = false;
    fa.has_list = true;
    fa.has_bits = false;
    fb.size = 0;
    fb.has_list = true;
    st.round = 1;
    Frontier *cur = &fa, *nxt = &fb;
    while (cur->size > 0 && cur->outdeg > 0) {
      int mode = m20_mode(g, *cur, -1, MODE_PUSH);
      BYO_TRY(clear_frontier_bits(g, *nxt));
      BYO_TRY(edge_map_round(g, st, *cur, *nxt, mode, tune));
      std::swap(cur, nxt);
    }
    // clear both bitmaps for the next traversal
    launch(ctx, k_bfscc_assign, dim3(grid_for(ctx, n, 256)), dim3(256), 0, (const uint64_t *)st.lp, n,
           s, d_label);
  }
  // finish with union-find over the whole graph; keep traversal labels (equal)
  uint32_t *lab2 = nullptr;
  BYO_TRY(ws(g, WS_LABEL, n, &lab2));
  BYO_TRY(cc_run(g, lab2));
  BYO_CU(ctx, cudaMemcpyAsync(d_label, lab2, n * 4, cudaMemcpyDeviceToDevice, ctx->stream));
  return check_launch(ctx, "bfs_cc");
}

// ================================================================ PageRank

template <typename T>
struct Acc {
  T s, c;
};

template <bool kComp, typename T>
__device__ __forceinline__ void acc_add(T &s, T &c, T x) {
  if constexpr (kComp) {
    T t = s + x;
    T bb = t - s;
    c += (s - (t - bb)) + (x - bb);
    s = t;
  } else {
    s += x;
  }
}

template <bool kComp, typename T, int GS>
__device__ __forceinline__ T group_total(T s, T c) {
#pragma unroll
  for (int o = GS / 2; o > 0; o >>= 1) {
    T s2 = __shfl_xor_sync(kFull, s, o, GS);
    T c2 = __shfl_xor_sync(kFull, c, o, GS);
    if constexpr (kComp) {
      T t = s + s2;
      T bb = t - s;
      T e = (s - (t - bb)) + (s2 - bb);
      s = t;
      c = c + c2 + e;
    } else {
      s += s2;
    }
  }
  return kComp ? s + c : s;
}

// ---------------------------------------------------------------- PageRank plan
// Work units of at most kPrTile + kPrLightMax slots, all processed by one
// kernel so every CTA streams the same amount:
//   light tile   consecutive vertices with runs <= kPrLightMax; one run of
//                slots; FP32 finishes its vertices, FP64 writes their sums
//   heavy chunk  kPrTile consecutive slots of one heavier vertex; its
//                compensated partial goes to part[chunk] and k_pr_combine sums
//                a vertex's chunks in order
// A warp gathers a unit's p_div values with plain loads, 16 independent
// loads per lane in flight, into its own stage in shared memory, then reduces
// from the stage (k_pr_units; light tiles by pr_light_tile).
constexpr int kPrTile = 512;            // slots per warp tile / heavy chunk
constexpr uint32_t kPrLightMax = 128;   // longest run of a light vertex
constexpr int kPrBlock = 256;
constexpr int kPrStage = kPrTile + kPrLightMax;  // staged values per warp

struct InLightLen {
  const uint64_t *off;
  __device__ uint64_t operator()(uint64_t v) const {
    uint64_t len = off[v + 1] - off[v];
    return len <= kPrLightMax ? len : 0;
  }
};

// tile starts: v == 0, v heavy, v-1 heavy, the light prefix crossed a
// multiple of kPrTile between v-1 and v, or v is a multiple of kPrTile (so a
// tile never holds more than kPrTile vertices, however many have no edges)
struct InTileStart {
  const uint64_t *off;
  const uint64_t *pre;
  __device__ uint64_t operator()(uint64_t v) const {
    if (v == 0 || v % kPrTile == 0) return 1;
    bool heavy = off[v + 1] - off[v] > kPrLightMax;
    bool prev_heavy = off[v] - off[v - 1] > kPrLightMax;
    return (heavy || prev_heavy || (pre[v] / kPrTile) != (pre[v - 1] / kPrTile)) ? 1 : 0;
  }
};
struct OutTileStart {
  uint32_t *starts;
  __device__ void operator()(uint64_t v, uint64_t pre, uint64_t f) const {
    if (f) starts[pre] = (uint32_t)v;
  }
};
// heavy vertices and their chunk counts
struct InHeavy {
  const uint64_t *off;
  __device__ uint64_t operator()(uint64_t v) const { return off[v + 1] - off[v] > kPrLightMax ? 1 : 0; }
};
struct OutHeavy {
  uint32_t *heavy;
  __device__ void operator()(uint64_t v, uint64_t pre, uint64_t f) const {
    if (f) heavy[pre] = (uint32_t)v;
  }
};
struct InChunks {
  const uint64_t *off;
  const uint32_t *heavy;
  __device__ uint64_t operator()(uint64_t h) const {
    uint32_t v = heavy[h];
    return (off[v + 1] - off[v] + kPrTile - 1) / kPrTile;
  }
};

// Unit descriptor (built once per PageRank call): slot range and either a
// light tile's vertices [v0, v1) or a heavy chunk (v1 == kNoVertex).
struct PrDesc {
  uint64_t s0, s1;
  uint32_t v0, v1;
  uint32_t chunk, pad;
};
constexpr uint32_t kNoVertex = 0xFFFFFFFFu;

// light tiles that are not a lone heavy vertex
struct InLightTile {
  const uint64_t *off;
  const uint32_t *tstart;
  __device__ uint64_t operator()(uint64_t t) const {
    uint32_t v0 = tstart[t], v1 = tstart[t + 1];
    return (v1 - v0 == 1 && off[v1] - off[v0] > kPrLightMax) ? 0 : 1;
  }
};
struct OutLightTile {
  const uint64_t *off;
  const uint32_t *tstart;
  PrDesc *desc;
  __device__ void operator()(uint64_t t, uint64_t pre, uint64_t f) const {
    if (!f) return;
    PrDesc d;
    d.v0 = tstart[t];
    d.v1 = tstart[t + 1];
    d.s0 = off[d.v0];
    d.s1 = off[d.v1];
    d.chunk = 0;
    d.pad = 0;
    desc[pre] = d;
  }
};

// heavy chunks after the light tiles (their count read on the device)
__global__ void k_pr_desc_chunks(const uint64_t *__restrict__ off, const uint32_t *__restrict__ heavy,
                                 const uint64_t *__restrict__ cbase, uint64_t nheavy,
                                 const uint64_t *__restrict__ nlight, PrDesc *desc) {
  const uint64_t base = *nlight;
  for (uint64_t h = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; h < nheavy;
       h += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = heavy[h];
    const uint64_t b = off[v], e = off[v + 1];
    for (uint64_t k = 0; k < cbase[h + 1] - cbase[h]; k++) {
      PrDesc d;
      d.s0 = b + k * kPrTile;
      d.s1 = d.s0 + kPrTile < e ? d.s0 + kPrTile : e;
      d.v0 = v;
      d.v1 = kNoVertex;
      d.chunk = (uint32_t)(cbase[h] + k);
      d.pad = cbase[h + 1] - cbase[h] == 1;  // the vertex's only chunk
      desc[base + cbase[h] + k] = d;
    }
  }
}

// State of the iteration loop (device side).
struct PrLoop {
  double l1;
  uint32_t iters;
  int32_t last;  // -1: no iteration ran; 0: the last iterate is in pb; 1: in pa
};

// One iteration: what its three kernels read and write.
template <typename T>
struct PrIter {
  const uint64_t *off;
  const uint32_t *slots, *deg;
  const PrDesc *desc;
  const uint64_t *counts;  // light tiles, heavy chunks
  const uint32_t *heavy;
  const uint64_t *cbase;
  uint64_t nheavy, n;
  const T *pdiv_in, *p_curr, *rdeg;  // rdeg: 1 / degree (FP64 only)
  T *p_next, *pdiv_out;
  T *part, *sum;  // chunk partials; every vertex's sum over its neighbours
  T damping, added;
  double *l1;          // the iteration's L1 distance, 0 between iterations
  unsigned int *done;  // blocks of the last kernel that are done
  PrLoop *loop;
  double eps;
  uint32_t max_iters;
  int half, in_graph;
  cudaGraphConditionalHandle h_if, h_while;
};

// Where vertices are finished (their iterate, shares and L1 distance, from their
// sums).  An FP64 instruction takes the SM's FP64 pipe 19 cycles however many
// lanes are active, and finishing takes ~30 of them in FP64 and 4 in FP32 (the L1
// norm is FP64 in every precision).  FP32: by the warp that has the sum, hidden
// behind its gathers (a kernel of its own takes 45 us an iteration at RMAT 2^22
// and saves the units 4).  FP64: by k_pr_finish with full warps; the units, with one
// heavy vertex or a tile's few at a time, kept the pipe 57% busy with it.  At RMAT
// 2^20 with 2^24 draws, an iteration: units 322 -> 157 us, combining 19, finishing
// 22; 20 iterations 6.9 -> 4.3 ms.
template <typename T>
constexpr bool kPrInPlace = sizeof(T) == 4;

// p / d from r = 1 / d: the quotient's error is computed exactly by a fused
// multiply-add and corrected (Markstein, IBM J. Res. Dev. 34, 1990: correctly
// rounded when r is, away from the ends of the exponent range).  3 FP64
// instructions where a division takes about 12.
__device__ __forceinline__ double pr_divide(double p, double d, double r) {
  const double q = __dmul_rn(p, r);
  if ((__double2hiint(q) & 0x7FF00000) == 0x7FF00000) return q;  // infinite or NaN
  return __fma_rn(__fma_rn(-q, d, p), r, q);
}
__device__ __forceinline__ float pr_divide(float p, float d, float) { return p / d; }

template <typename T>
__device__ __forceinline__ void pr_finish(const PrIter<T> &a, uint64_t v, T tot, double &l1loc) {
  const T p = a.damping * tot + a.added;
  const uint32_t d = __ldg(a.deg + v);
  const T before = __ldg(a.p_curr + v);
  const T r = sizeof(T) == 8 ? __ldg(a.rdeg + v) : T(0);
  a.p_next[v] = p;
  a.pdiv_out[v] = d ? pr_divide(p, (T)d, r) : (T)INFINITY;
  l1loc += fabs((double)before - (double)p);
}

// The end of an iteration's last kernel: the last block to finish records the
// distance, clears the accumulators and, in a graph, tells the loop whether
// another iteration runs (PageRank.h:176-190: stop when L1 < eps or after
// max_iters).  half 0 ends the first iteration of a loop body (pa -> pb) and
// sets both conditions; half 1 ends the second (pb -> pa) and sets the loop's.
template <typename T>
__device__ __forceinline__ void pr_end(const PrIter<T> &a, double l1loc, double *sm) {
  if (__syncthreads_or(l1loc != 0.0)) l1loc = block_sum(l1loc, sm);  // FP64 adds: 64 cycles each, in a row
  if (threadIdx.x) return;
  if (gridDim.x > 1) {
    if (l1loc != 0.0) atomicAdd(a.l1, l1loc);
    __threadfence();
    if (atomicAdd(a.done, 1u) != gridDim.x - 1) return;
    __threadfence();
    l1loc = 0.0;
  }
  const uint32_t it = ++a.loop->iters;
  const double L = __ldcg(a.l1) + l1loc;
  a.loop->l1 = L;
  a.loop->last = a.half;
  *a.l1 = 0.0;
  *a.done = 0;
  if (!a.in_graph) return;  // the host reads the state and decides
  const unsigned cont = (!(L < a.eps) && it < a.max_iters) ? 1u : 0u;
  if (a.half == 0) cudaGraphSetConditional(a.h_if, cont);
  cudaGraphSetConditional(a.h_while, cont);
}

// (s, c) += (s2, c2), compensated when kComp (TwoSum of the sums, errors added)
template <bool kComp, typename T>
__device__ __forceinline__ void acc_merge(T &s, T &c, T s2, T c2) {
  if constexpr (kComp) {
    T t = s + s2;
    T bb = t - s;
    T e = (s - (t - bb)) + (s2 - bb);
    s = t;
    c = c + c2 + e;
  } else {
    s += s2;
  }
}

// Per-warp scratch of a light tile beside its stage: a head flag for the first
// slot of every non-empty run.
constexpr uint32_t kPrFlagWords = (kPrStage + 31) / 32;
template <typename T>
constexpr size_t pr_warp_smem() {
  return (size_t)kPrStage * sizeof(T) + kPrFlagWords * 4;
}

// Position of the last head flag below pos (there is one: slot 0 is a head).
__device__ __forceinline__ uint32_t last_head_below(const uint32_t *flags, uint32_t pos) {
  for (int w = (int)((pos - 1) >> 5); w >= 0; w--) {
    uint32_t word = flags[w];
    const uint32_t lim = pos - 32u * (uint32_t)w;  // bits below pos in this word
    if (lim < 32) word &= (1u << lim) - 1u;
    if (word) return 32u * (uint32_t)w + 31u - __clz(word);
  }
  return 0;
}

// Sums of a light tile's runs from the staged values buf[0, len).  Each lane
// takes an odd-length chunk of consecutive slots (odd, so the lanes' reads
// fall in different banks) and sums it in order; the partial of a run that
// crosses chunk boundaries is carried by an inclusive segmented warp scan (a
// lane holding a head starts a new segment) and the run open at a lane's
// start is completed by the lane that holds its end.  Each run's total is
// written over the staged value of its first slot, and a last pass finishes (or
// writes the sums of) the tile's vertices, a lane each (consecutive vertices,
// coalesced).  One fixed order per graph, so results are deterministic.
template <bool kComp, typename T>
__device__ __forceinline__ void pr_light_tile(const PrDesc &d, uint32_t len, T *buf, uint32_t *flags,
                                              const PrIter<T> &a, double &l1loc) {
  const uint64_t *__restrict__ off = a.off;
  const unsigned lane = lane_id();
  for (uint32_t w = lane; w < kPrFlagWords; w += 32) flags[w] = 0;
  __syncwarp();
  for (uint32_t x = d.v0 + lane; x < d.v1; x += 32) {
    const uint64_t b = off[x], e = off[x + 1];
    if (e > b) {
      const uint32_t r0 = (uint32_t)(b - d.s0);
      atomicOr(flags + (r0 >> 5), 1u << (r0 & 31));
    }
  }
  __syncwarp();
  const uint32_t C = ((len + 31) >> 5) | 1u;
  const uint32_t lo = min(lane * C, len), hi = min(lo + C, len);
  T s = T(0), c = T(0), hs = T(0), hc = T(0);
  bool head = false;
  uint32_t hpos = 0, fw = 0;
  for (uint32_t r = lo; r < hi; r++) {
    if (r == lo || (r & 31) == 0) fw = flags[r >> 5];
    if ((fw >> (r & 31)) & 1u) {
      if (!head) {
        hs = s;
        hc = c;
        head = true;
      } else {
        buf[hpos] = kComp ? s + c : s;  // a run inside this chunk
      }
      s = T(0);
      c = T(0);
      hpos = r;
    }
    acc_add<kComp>(s, c, buf[r]);
  }
  T ss = s, sc = c;
  int f = head ? 1 : 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T ps = __shfl_up_sync(kFull, ss, o), pc = __shfl_up_sync(kFull, sc, o);
    const int pf = __shfl_up_sync(kFull, f, o);
    if ((int)lane >= o) {
      if (!f) {
        T ts = ps, tc = pc;
        acc_merge<kComp>(ts, tc, ss, sc);
        ss = ts;
        sc = tc;
      }
      f |= pf;
    }
  }
  T cs = __shfl_up_sync(kFull, ss, 1), cc = __shfl_up_sync(kFull, sc, 1);
  __syncwarp();  // every lane's reads of the stage are done
  if (head && lo > 0) {  // the run open at lo ends in this chunk
    acc_merge<kComp>(cs, cc, hs, hc);
    buf[last_head_below(flags, lo)] = kComp ? cs + cc : cs;
  }
  if (lane == 31 && len)  // the run open at the tile's end
    buf[last_head_below(flags, len)] = kComp ? ss + sc : ss;
  __syncwarp();
  for (uint32_t x = d.v0 + lane; x < d.v1; x += 32) {
    const uint64_t b = off[x], e = off[x + 1];
    const T tot = e > b ? buf[b - d.s0] : T(0);
    if constexpr (kPrInPlace<T>) pr_finish(a, x, tot, l1loc); else a.sum[x] = tot;
  }
  __syncwarp();
}

// One warp per unit, no block-wide barriers: the warp gathers p_div of the
// unit's slots (16 independent loads per lane in flight) into its own stage in
// shared memory, then reduces.  Light tile: pr_light_tile.  Heavy chunk: warp
// partial to part[]; with kDirectHeavy (FP64) each lane sums its gathered slots
// lane, lane+32, ... in registers without the stage, in the same order:
// measured at RMAT 2^22, 20 FP64 iterations 34.0 -> 28.8 ms, while FP32 runs 1%
// faster staged.  FP64 takes 64 registers (4 CTAs an SM): 48 spill the gathers
// in flight, 263 against 207 us an iteration at RMAT 2^20.
template <bool kComp, typename T, bool kDirectHeavy>
__global__ void __launch_bounds__(kPrBlock, sizeof(T) == 8 ? 4 : 5) k_pr_units(PrIter<T> a) {
  extern __shared__ __align__(16) unsigned char pr_smem[];
  __shared__ double sm[kPrBlock / 32 + 1];
  double l1loc = 0.0;
  const uint64_t nunits = a.counts[0] + a.counts[1];  // light tiles + heavy chunks
  const T *__restrict__ pdiv_in = a.pdiv_in;
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
  T *buf = reinterpret_cast<T *>(pr_smem) + (size_t)warp * kPrStage;
  uint32_t *flags = reinterpret_cast<uint32_t *>(reinterpret_cast<T *>(pr_smem) + (size_t)(kPrBlock / 32) * kPrStage) +
                    (size_t)warp * kPrFlagWords;
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t t = gw; t < nunits; t += nw) {
    const PrDesc d = a.desc[t];
    const uint32_t len = (uint32_t)(d.s1 - d.s0);
    const uint32_t *__restrict__ id = a.slots + d.s0;
    if (d.v1 == kNoVertex && kDirectHeavy) {
      T s = T(0), c = T(0);
      for (uint32_t i = lane; i < len; i += 32 * 16) {
        uint32_t u[16];
#pragma unroll
        for (int q = 0; q < 16; q++) u[q] = i + 32 * q < len ? __ldcs(id + i + 32 * q) : kSentinel;
        T g[16];
#pragma unroll
        for (int q = 0; q < 16; q++) g[q] = u[q] != kSentinel ? __ldg(pdiv_in + u[q]) : T(0);
#pragma unroll
        for (int q = 0; q < 16; q++)
          if (i + 32 * q < len) acc_add<kComp>(s, c, g[q]);
      }
      T tot = group_total<kComp, T, 32>(s, c);
      if (lane == 0) a.part[d.chunk] = tot;
      continue;
    }
    for (uint32_t i = lane; i < len; i += 32 * 16) {
      uint32_t u[16];
#pragma unroll
      for (int q = 0; q < 16; q++) u[q] = i + 32 * q < len ? __ldcs(id + i + 32 * q) : kSentinel;
#pragma unroll
      for (int q = 0; q < 16; q++)
        if (i + 32 * q < len) buf[i + 32 * q] = u[q] != kSentinel ? __ldg(pdiv_in + u[q]) : T(0);
    }
    __syncwarp();
    if (d.v1 != kNoVertex) {
      pr_light_tile<kComp, T>(d, len, buf, flags, a, l1loc);
    } else {
      T s = T(0), c = T(0);
      for (uint32_t r = lane; r < len; r += 32) acc_add<kComp>(s, c, buf[r]);
      T tot = group_total<kComp, T, 32>(s, c);
      if (lane == 0) {
        if (kPrInPlace<T> && d.pad) pr_finish(a, d.v0, tot, l1loc); else a.part[d.chunk] = tot;
      }
    }
    __syncwarp();
  }
  if constexpr (kPrInPlace<T>) {
    l1loc = block_sum(l1loc, sm);
    if (threadIdx.x == 0 && l1loc != 0.0) atomicAdd(a.l1, l1loc);
  }
}

// FP32: a group of kCombineLanes lanes per heavy vertex of several chunks (most
// have a few): its chunk partials, lane l of the group taking chunks l, l + G,
// ... in order, summed by a fixed tree over the group; then the vertex is
// finished by the group's first lane.  Measured at RMAT 2^22 (ms per iteration
// of units + combine): groups of 32 / 8 / 4 lanes 0.563 / 0.543 / 0.549.
// FP64: the heavy vertices' sums, a lane each, for an addition costs a warp the
// same whatever lanes take part: up to 8 partials by the same tree in a lane,
// more by the warp.
constexpr int kCombineLanes = 8;
template <bool kComp, typename T>
__global__ void __launch_bounds__(256) k_pr_combine(PrIter<T> a) {
  __shared__ double sm[9];
  const unsigned lane = lane_id();
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  if constexpr (kPrInPlace<T>) {
    constexpr int kPer = 32 / kCombineLanes;
    const unsigned gl = lane % kCombineLanes;
    double l1loc = 0.0;
    for (uint64_t base = gw * kPer; base < a.nheavy; base += nw * kPer) {
      const uint64_t h = base + lane / kCombineLanes;
      T s = T(0), c = T(0);
      bool mine = false;  // a vertex of several chunks (one chunk: finished by its unit)
      if (h < a.nheavy) {
        const uint64_t c0 = a.cbase[h], c1 = a.cbase[h + 1];
        mine = c1 - c0 > 1;
        if (mine)
          for (uint64_t k = c0 + gl; k < c1; k += kCombineLanes) acc_add<kComp>(s, c, a.part[k]);
      }
      const T tot = group_total<kComp, T, kCombineLanes>(s, c);
      if (mine && gl == 0) pr_finish(a, a.heavy[h], tot, l1loc);
    }
    pr_end(a, l1loc, sm);
  } else {
    for (uint64_t base = gw * 32; base < a.nheavy; base += nw * 32) {
      const uint64_t h = base + lane;
      const uint64_t c0 = h < a.nheavy ? a.cbase[h] : 0, c1 = h < a.nheavy ? a.cbase[h + 1] : 0;
      const bool wide = c1 - c0 > kCombineLanes;
      T s[kCombineLanes], c[kCombineLanes];
#pragma unroll
      for (int k = 0; k < kCombineLanes; k++) {
        s[k] = !wide && c0 + k < c1 ? a.part[c0 + k] : T(0);
        c[k] = T(0);
      }
#pragma unroll
      for (int o = kCombineLanes / 2; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < o; k++) acc_merge<kComp>(s[k], c[k], s[k + o], c[k + o]);
      T tot = kComp ? s[0] + c[0] : s[0];
      for (unsigned m = __ballot_sync(kFull, wide); m; m &= m - 1) {
        const int o = __ffs(m) - 1;
        const uint64_t a0 = __shfl_sync(kFull, c0, o), a1 = __shfl_sync(kFull, c1, o);
        T x = T(0), y = T(0);
        for (uint64_t k = a0 + lane; k < a1; k += 32) acc_add<kComp>(x, y, a.part[k]);
        const T t = group_total<kComp, T, 32>(x, y);
        if ((int)lane == o) tot = t;
      }
      if (h < a.nheavy) a.sum[a.heavy[h]] = tot;
    }
  }
}

// FP64: the vertices from their sums, a thread each.
template <typename T>
__global__ void __launch_bounds__(256) k_pr_finish(PrIter<T> a) {
  __shared__ double sm[9];
  double l1loc = 0.0;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < a.n; v += (uint64_t)gridDim.x * blockDim.x)
    pr_finish(a, v, a.sum[v], l1loc);
  pr_end(a, l1loc, sm);
}

template <typename T>
__global__ void k_pr_init(const uint32_t *__restrict__ deg, uint64_t n, T *p_curr, T *pdiv, T *rdeg, T one_over_n) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t d = deg[v];
    p_curr[v] = one_over_n;
    pdiv[v] = one_over_n / (T)d;
    if (rdeg && d) rdeg[v] = T(1) / (T)d;
  }
}

template <typename T>
__global__ void k_to_f64(const T *__restrict__ in, uint64_t n, double *out) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x)
    out[v] = (double)in[v];
}

template <bool kComp, typename T>
static int pagerank_impl(byo_graph *g, double eps, uint32_t max_iters, double *d_p, uint32_t *iters_out,
                         double *l1_out) {
  byo_ctx *ctx = g->ctx;
  const uint64_t n = g->n;
  T *pa, *pb, *da, *db;
  BYO_TRY(ws(g, WS_PR_A, n + 2, &pa));
  BYO_TRY(ws(g, WS_PR_B, n, &pb));
  BYO_TRY(ws(g, WS_PR_C, n, &da));
  BYO_TRY(ws(g, WS_PR_D, n + 2 + (sizeof(PrLoop) + sizeof(T) - 1) / sizeof(T) + 2, &db));  // p_div, loop state
  // plan
  uint64_t *pre = nullptr;
  uint32_t *lists = nullptr;
  BYO_TRY(ws(g, WS_SCAN, 2 * n + 4, &pre));
  uint64_t *cbase = pre + n + 2;
  BYO_TRY(ws(g, WS_BUCKETS, 2 * n + 8, &lists));
  uint32_t *tstart = lists, *heavy = lists + (n + 4);
  double *d_l1 = nullptr;
  BYO_TRY(ws(g, WS_MISC, 8, (uint32_t **)&d_l1));
  uint64_t *counts = reinterpret_cast<uint64_t *>(d_l1 + 2);  // [0] light tiles, [1] heavy chunks
  uint64_t *h = nullptr;
  BYO_TRY(pinned(ctx, 4096, (void **)&h));
  const uint64_t *tot = nullptr;
  BYO_TRY(scan_apply(ctx, n, InLightLen{g->d_off}, OutPrefix{pre}, &tot));
  BYO_TRY(scan_apply(ctx, n, InTileStart{g->d_off, pre}, OutTileStart{tstart}, &tot));
  BYO_CU(ctx, cudaMemcpyAsync(h, tot, 8, cudaMemcpyDeviceToHost, ctx->stream));
  BYO_TRY(scan_apply(ctx, n, InHeavy{g->d_off}, OutHeavy{heavy}, &tot));
  BYO_CU(ctx, cudaMemcpyAsync(h + 1, tot, 8, cudaMemcpyDeviceToHost, ctx->stream));
  BYO_CU(ctx, cudaStreamSynchronize(ctx->stream));
  const uint64_t ntiles = h[0], nheavy = h[1];
  // From here the plan stays on the device: the counts of light tiles and
  // heavy chunks go to `counts`, which k_pr_desc_chunks and k_pr_units read,
  // and the buffers and grid are sized by upper bounds (a heavy vertex of d
  // slots makes ceil(d / kPrTile) chunks), so the host builds the graph
  // below while the GPU finishes the plan.
  BYO_TRY(scan_apply(ctx, nheavy, InChunks{g->d_off, heavy}, OutPrefix{cbase}, &tot));
  BYO_CU(ctx, cudaMemcpyAsync(cbase + nheavy, tot, 8, cudaMemcpyDeviceToDevice, ctx->stream));
  BYO_CU(ctx, cudaMemcpyAsync(counts + 1, tot, 8, cudaMemcpyDeviceToDevice, ctx->stream));
  h[3] = n;  // h[3] is not written again before the next synchronisation
  BYO_CU(ctx, cudaMemcpyAsync(tstart + ntiles, h + 3, 4, cudaMemcpyHostToDevice, ctx->stream));
  T *sum = nullptr, *rdeg = nullptr;
  if (!kPrInPlace<T>) {
    BYO_TRY(ws(g, WS_LP, n, &sum));
    BYO_TRY(ws(g, WS_FRONT_LIST_A, n, &rdeg));
  }
  launch(ctx, k_pr_init<T>, dim3(grid_for(ctx, n, 256)), dim3(256), 0, (const uint32_t *)g->d_deg, n, pa, da, rdeg,
         (T)(1.0 / (double)n));
  const uint64_t max_chunks = g->nslots / kPrTile + nheavy + 1;
  // descriptors: compacted light tiles, then heavy chunks
  PrDesc *desc = nullptr;
  BYO_TRY(ws(g, WS_TC_NBR, (ntiles + max_chunks + 1) * sizeof(PrDesc) / 4, (uint32_t **)&desc));
  BYO_TRY(scan_apply(ctx, ntiles, InLightTile{g->d_off, tstart}, OutLightTile{g->d_off, tstart, desc}, &tot));
  BYO_CU(ctx, cudaMemcpyAsync(counts, tot, 8, cudaMemcpyDeviceToDevice, ctx->stream));
  if (nheavy)
    launch(ctx, k_pr_desc_chunks, dim3(grid_for(ctx, nheavy, 256)), dim3(256), 0, (const uint64_t *)g->d_off,
           (const uint32_t *)heavy, (const uint64_t *)cbase, nheavy, (const uint64_t *)counts, desc);
  T *part = nullptr;
  BYO_TRY(ws(g, WS_TC_CNT, max_chunks + 2, &part));
  const T damping = (T)0.85;
  const T added = (T)((1 - 0.85) * (1 / (double)n));
  const int grid_c = grid_for(ctx, kPrInPlace<T> ? nheavy * kCombineLanes : nheavy, 256, 8);
  const size_t units_smem = (size_t)(kPrBlock / 32) * pr_warp_smem<T>();
  BYO_CU(ctx, cudaFuncSetAttribute(k_pr_units<kComp, T, sizeof(T) == 8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)units_smem));
  int units_per_sm = 0;
  BYO_CU(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&units_per_sm, k_pr_units<kComp, T, sizeof(T) == 8>,
                                                            kPrBlock, units_smem));
  const int grid_u = grid_for(ctx, (ntiles + max_chunks) * 32, kPrBlock, units_per_sm > 0 ? units_per_sm : 1);
  // The iterations run as one CUDA graph: a WHILE node whose body holds two
  // iterations (pa -> pb, then under an IF node pb -> pa), each ending in
  // pr_end, which sets the conditions from the L1 norm on the device.
  // No host round trip happens between iterations.
  PrLoop *loop = reinterpret_cast<PrLoop *>((reinterpret_cast<uintptr_t>(db + n + 2) + 7) & ~(uintptr_t)7);
  unsigned int *done = reinterpret_cast<unsigned int *>(d_l1 + 1);
  BYO_CU(ctx, cudaMemsetAsync(d_l1, 0, 16, ctx->stream));
  {
    PrLoop z{0.0, 0u, -1};
    BYO_CU(ctx, cudaMemcpyAsync(loop, &z, sizeof(PrLoop), cudaMemcpyHostToDevice, ctx->stream));
  }
  PrIter<T> iter[2];
  for (int h : {0, 1})
    iter[h] = PrIter<T>{g->d_off, g->d_slots, g->d_deg, desc, counts, heavy, cbase, nheavy, n, h ? db : da,
                        h ? pb : pa, rdeg, h ? pa : pb, h ? da : db, part, sum, damping, added, d_l1, done, loop, eps,
                        max_iters, h, ctx->pr_graphs ? 1 : 0, 0, 0};
  const int grid_f = grid_for(ctx, n, 256);
  uint32_t it = 0;
  double L1 = 0.0;
  const T *last = pa;
  if (max_iters > 0 && !ctx->pr_graphs) {
    // one stream launch per kernel and a host check of the residual after
    // each iteration (the same kernels in the same order: the same results)
    PrLoop *hs = nullptr;
    BYO_TRY(pinned(ctx, 4096, (void **)&hs));
    for (int hh = 0;; hh ^= 1) {
      launch_t(ctx, "pr_pull", k_pr_units<kComp, T, sizeof(T) == 8>, dim3(grid_u), dim3(kPrBlock), units_smem, iter[hh]);
      if (nheavy || kPrInPlace<T>)
        launch_t(ctx, "pr_pull", k_pr_combine<kComp, T>, dim3(grid_c), dim3(256), 0, iter[hh]);
      if (!kPrInPlace<T>) launch_t(ctx, "pr_pull", k_pr_finish<T>, dim3(grid_f), dim3(256), 0, iter[hh]);
      BYO_CU(ctx, cudaMemcpyAsync(hs, loop, sizeof(PrLoop), cudaMemcpyDeviceToHost, ctx->stream));
      BYO_CU(ctx, cudaStreamSynchronize(ctx->stream));
      if (hs->l1 < eps || hs->iters >= max_iters) break;
    }
    it = hs->iters;
    L1 = hs->l1;
    last = hs->last == 0 ? pb : pa;
  } else if (max_iters > 0) {
    cudaGraph_t graph = nullptr, body = nullptr, second = nullptr;
    cudaGraphExec_t exec = nullptr;
    int rc = BYO_OK;
    auto fail = [&](const char *what, cudaError_t e) {
      if (rc == BYO_OK) rc = set_error(ctx, BYO_EDEVICE, what, e);
    };
    cudaError_t e = cudaGraphCreate(&graph, 0);
    if (e != cudaSuccess) fail("pagerank graph", e);
    cudaGraphConditionalHandle h_while = 0, h_if = 0;
    cudaGraphNode_t wnode = nullptr, inode = nullptr;
    if (rc == BYO_OK && (e = cudaGraphConditionalHandleCreate(&h_while, graph, 1, cudaGraphCondAssignDefault)) !=
                            cudaSuccess)
      fail("pagerank loop condition", e);
    if (rc == BYO_OK) {
      cudaGraphNodeParams wp = {};
      wp.type = cudaGraphNodeTypeConditional;
      wp.conditional.handle = h_while;
      wp.conditional.type = cudaGraphCondTypeWhile;
      wp.conditional.size = 1;
      if ((e = cudaGraphAddNode(&wnode, graph, nullptr, nullptr, 0, &wp)) != cudaSuccess) fail("pagerank loop", e);
      else body = wp.conditional.phGraph_out[0];
    }
    if (rc == BYO_OK &&
        (e = cudaGraphConditionalHandleCreate(&h_if, graph, 0, cudaGraphCondAssignDefault)) != cudaSuccess)
      fail("pagerank half condition", e);
    // one iteration: units, combine, FP64's finish; returns its last node
    for (int h : {0, 1}) {
      iter[h].h_if = h_if;
      iter[h].h_while = h_while;
    }
    auto add_iter = [&](cudaGraph_t gr, int h, cudaGraphNode_t dep, cudaGraphNode_t *lastn) {
      cudaGraphNode_t prev = dep;
      auto add = [&](void *func, int grid, int block, size_t smem, const char *what) {
        if (rc != BYO_OK) return;
        void *args[] = {&iter[h]};
        cudaKernelNodeParams kp = {};
        kp.func = func;
        kp.gridDim = dim3(grid);
        kp.blockDim = dim3(block);
        kp.sharedMemBytes = (unsigned)smem;
        kp.kernelParams = args;
        cudaGraphNode_t node = nullptr;
        const cudaError_t x = cudaGraphAddKernelNode(&node, gr, prev ? &prev : nullptr, prev ? 1 : 0, &kp);
        if (x != cudaSuccess) return fail(what, x);
        prev = node;
      };
      add((void *)k_pr_units<kComp, T, sizeof(T) == 8>, grid_u, kPrBlock, units_smem, "pagerank units node");
      if (nheavy || kPrInPlace<T>) add((void *)k_pr_combine<kComp, T>, grid_c, 256, 0, "pagerank combine node");
      if (!kPrInPlace<T>) add((void *)k_pr_finish<T>, grid_f, 256, 0, "pagerank finish node");
      *lastn = prev;
    };
    cudaGraphNode_t k0 = nullptr, k1 = nullptr;
    add_iter(body, 0, nullptr, &k0);
    if (rc == BYO_OK) {
      cudaGraphNodeParams ip = {};
      ip.type = cudaGraphNodeTypeConditional;
      ip.conditional.handle = h_if;
      ip.conditional.type = cudaGraphCondTypeIf;
      ip.conditional.size = 1;
      if ((e = cudaGraphAddNode(&inode, body, &k0, nullptr, 1, &ip)) != cudaSuccess) fail("pagerank half", e);
      else second = ip.conditional.phGraph_out[0];
    }
    add_iter(second, 1, nullptr, &k1);
    if (rc == BYO_OK && (e = cudaGraphInstantiate(&exec, graph, 0)) != cudaSuccess) fail("pagerank instantiate", e);
    if (rc == BYO_OK) {
      const bool timed = !ctx->ktag.empty() && ktimer_begin(ctx, "pr_pull");
      if ((e = cudaGraphLaunch(exec, ctx->stream)) != cudaSuccess) fail("pagerank launch", e);
      if (timed) ktimer_end(ctx);
      ctx->launches += 1;
    }
    PrLoop hs{0.0, 0u, -1};
    if (rc == BYO_OK && (e = cudaMemcpyAsync(&hs, loop, sizeof(PrLoop), cudaMemcpyDeviceToHost, ctx->stream)) !=
                            cudaSuccess)
      fail("pagerank state", e);
    if (rc == BYO_OK && (e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess) fail("pagerank sync", e);
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    BYO_TRY(rc);
    ctx->launches += (uint64_t)(1 + (nheavy || kPrInPlace<T>) + !kPrInPlace<T>) * hs.iters - 1;  // kernels the graph ran
    it = hs.iters;
    L1 = hs.l1;
    last = hs.last == 0 ? pb : pa;
  }
  // the last computed iterate (the reference's final swap would hand back the
  // zeroed previous one when max_iters ends the loop, PageRank.h:181-192)
  launch(ctx, k_to_f64<T>, dim3(grid_for(ctx, n, 256)), dim3(256), 0, last, n, d_p);
  if (iters_out) *iters_out = it;
  if (l1_out) *l1_out = L1;
  return check_launch(ctx, "pagerank");
}

int pagerank_run(byo_graph *g, double eps, uint32_t max_iters, int precision, double *d_p,
                 uint32_t *iters, double *l1) {
  if (g->n == 0) return BYO_OK;
  switch (precision) {
    case BYO_PR_FP32_KAHAN: return pagerank_impl<true, float>(g, eps, max_iters, d_p, iters, l1);
    case BYO_PR_FP64: return pagerank_impl<false, double>(g, eps, max_iters, d_p, iters, l1);
    case BYO_PR_FP32: return pagerank_impl<false, float>(g, eps, max_iters, d_p, iters, l1);
    default: return set_error(g->ctx, BYO_EINVAL, "pagerank: unknown precision");
  }
}

}  // namespace byo
