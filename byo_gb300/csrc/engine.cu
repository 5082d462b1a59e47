// engine.cu -- edgeMap rounds (push / blocked / pull) and the BFS driver.
// See engine.h for the design.  Algorithmic bytes of one BFS traversal:
// 4 B per adjacency entry of every reached vertex + 8 B offsets per vertex
// + 8 B lp written per reached vertex (parent/level split is 8 B more).
#include <algorithm>
#include <cstring>

#include "device.cuh"
#include "engine.h"
#include "policy.cuh"
#include "internal.h"
#include "scan.cuh"

namespace byo {

__host__ __device__ __forceinline__ int log4_bin(uint32_t d) {
#ifdef __CUDA_ARCH__
  int b = d ? (31 - __clz(d)) / 2 : 0;  // 0:[0,4) 1:[4,16) ...
#else
  int b = d ? (31 - __builtin_clz(d)) / 2 : 0;
#endif
  return b > 7 ? 7 : b;
}

// The degree sketch of the next frontier is counted per block in shared
// memory (a warp adds one count per bin it holds) and added to the round's
// statistics once per block, so no global counter sees one atomic per vertex.
__device__ __forceinline__ void hist_init(unsigned long long *sh) {
  if (threadIdx.x < 8) sh[threadIdx.x] = 0;
  __syncthreads();
}
__device__ __forceinline__ void hist_warp_add(unsigned long long *sh, bool has, uint32_t d) {
  if (!__ballot_sync(kFull, has)) return;
  const int bin = log4_bin(d);
#pragma unroll
  for (int b = 0; b < 8; b++) {
    const unsigned m = __ballot_sync(kFull, has && bin == b);
    if (m && lane_id() == 0) atomicAdd(sh + b, (unsigned long long)__popc(m));
  }
}
__device__ __forceinline__ void hist_flush(unsigned long long *sh, RoundStats *st) {
  __syncthreads();
  if (threadIdx.x < 8 && sh[threadIdx.x]) atomicAdd(&st->hist[threadIdx.x], sh[threadIdx.x]);
}

// Emits v (if `emit`) to the next frontier list and bitmap; accumulates its
// degree for the round statistics.  Warp-collective.
__device__ __forceinline__ void emit_next(bool emit, uint32_t v, uint32_t *out_list,
                                          uint32_t *out_bits, RoundStats *st,
                                          const uint32_t *__restrict__ deg, uint64_t &dsum,
                                          WarpList<> &wl, unsigned long long *sh) {
  wl.add(emit, v, out_list, &st->count);
  uint32_t d = 0;
  if (emit) {
    atomicOr(out_bits + (v >> 5), 1u << (v & 31));
    d = deg[v];
    dsum += d;
  }
  hist_warp_add(sh, emit, d);
}

// Where the parts of a block's warps go in a list that they append to: s[w] holds
// the counts, then the places, by one add to the list's counter.  By one warp.
__device__ __forceinline__ void list_places(unsigned long long *s /* [32] */, uint32_t nw, unsigned long long *counter) {
  const uint32_t lane = lane_id(), c = lane < nw ? (uint32_t)s[lane] : 0, upto = warp_inclusive_scan(c);
  const uint32_t total = __shfl_sync(kFull, upto, 31);
  unsigned long long base = 0;
  if (lane == 0 && total) base = atomicAdd(counter, (unsigned long long)total);
  base = __shfl_sync(kFull, base, 0);
  if (lane < nw) s[lane] = base + upto - c;
}

// A visiting kernel's end: what its warps still hold of the next frontier (and of
// a second list, the pull's deferred vertices), by one add a block, and its part of
// the round's statistics, a warp each, so that the adds are waited for together.
// Warps that see a word or two each come here with all they found, and an add a
// warp was a quarter of a pull round at 2^18 vertices (three rounds: 47 -> 36 us) and
// 8% of a BFS on a uniform graph of 2 M (337 -> 308).  Block-collective, 4 warps or more.
template <uint32_t kCap>
__device__ __forceinline__ void round_flush(WarpList<kCap> &wl, uint32_t *out_list, RoundStats *st, uint64_t dsum,
                                            unsigned long long *sh, WarpList<kCap> *wd = nullptr,
                                            uint32_t *defer = nullptr) {
  __shared__ unsigned long long s_at[32], s_defer[32], s_sum[32];
  const uint32_t w = threadIdx.x >> 5, lane = lane_id(), nw = blockDim.x >> 5;
  dsum = warp_sum(dsum);
  if (lane == 0) {
    s_at[w] = wl.count;
    if (wd) s_defer[w] = wd->count;
    s_sum[w] = dsum;
  }
  __syncthreads();
  if (w == 0) list_places(s_at, nw, &st->count);
  if (w == 1 && wd) list_places(s_defer, nw, &st->ndefer);
  if (w == 2) {
    dsum = warp_sum(lane < nw ? s_sum[lane] : 0ull);
    if (lane == 0 && dsum) atomicAdd(&st->outdeg, (unsigned long long)dsum);
  }
  if (w == 3 && lane < 8 && sh[lane]) atomicAdd(&st->hist[lane], sh[lane]);
  __syncthreads();
  for (uint32_t i = lane; i < wl.count; i += 32) out_list[s_at[w] + i] = wl.buf[i];
  if (wd)
    for (uint32_t i = lane; i < wd->count; i += 32) defer[s_defer[w] + i] = wd->buf[i];
}

// Visits edge u->v for BFS_F: cond(v) = not visited before this round;
// updateAtomic keeps the smallest (level, parent); the first writer emits.
__device__ __forceinline__ bool visit(uint32_t u, uint32_t v, uint64_t lvl, uint64_t *lp,
                                      const uint32_t *__restrict__ visited) {
  if (v == kSentinel) return false;
  if (test_bit_cg(visited, v)) return false;
  unsigned long long old = atomicMin((unsigned long long *)(lp + v), (unsigned long long)(lvl | u));
  return old == kNone64;
}

// R edges u[q] -> v[q] a lane (v kSentinel: none): their bits, then their atomics, then
// the emissions, so R edges wait for each access once.  Warp-collective.
template <int R>
__device__ __forceinline__ void visit_emit(const uint32_t (&u)[R], const uint32_t (&v)[R], uint64_t lvl, uint64_t *lp,
                                           const uint32_t *__restrict__ visited, uint32_t *out_list,
                                           uint32_t *out_bits, RoundStats *st, const uint32_t *__restrict__ deg,
                                           uint64_t &dsum, WarpList<> &wl, unsigned long long *sh) {
  bool open[R];
#pragma unroll
  for (int q = 0; q < R; q++) open[q] = v[q] != kSentinel && !test_bit_cg(visited, v[q]);
#pragma unroll
  for (int q = 0; q < R; q++)
    if (open[q]) open[q] = atomicMin((unsigned long long *)(lp + v[q]), (unsigned long long)(lvl | u[q])) == kNone64;
#pragma unroll
  for (int q = 0; q < R; q++) emit_next(open[q], v[q], out_list, out_bits, st, deg, dsum, wl, sh);
}

// ---------------------------------------------------------------- push
// Slots of a hub a CTA takes (hub, chunk).  One CTA for a whole hub held the
// round of a 2^22-vertex RMAT graph's largest hubs up for 1.3 ms; 0.11 in chunks.
constexpr uint32_t kHubChunk = 2048;

// Eight CTAs an SM: at 40 registers, six, a BFS by pushes alone on RMAT 2^22 / 2^26
// draws took 2300 us instead of 2000.
template <int GS>
__global__ void __launch_bounds__(256, 8) k_push(const uint64_t *__restrict__ off,
                                              const uint32_t *__restrict__ slots,
                                              const uint32_t *__restrict__ deg,
                                              const uint32_t *__restrict__ F, uint64_t fsize,
                                              uint64_t *lp, const uint32_t *__restrict__ visited,
                                              uint32_t *out_list, uint32_t *out_bits,
                                              RoundStats *st, uint64_t lvl, uint2 *hubs, uint64_t hub_cap,
                                              uint32_t hub_min) {
  __shared__ unsigned long long s_hist[8];
  hist_init(s_hist);
  __shared__ uint32_t s_list[8][kWarpListCap];
  WarpList<> wl{s_list[threadIdx.x >> 5]};
  constexpr int PER_WARP = 32 / GS;
  const unsigned lane = lane_id(), g = lane / GS, gl = lane % GS;
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint64_t dsum = 0;
  for (uint64_t i0 = gw * PER_WARP; i0 < fsize; i0 += nw * PER_WARP) {
    uint64_t i = i0 + g;
    uint32_t u = 0;
    uint64_t b = 0, e = 0;
    if (i < fsize) {
      u = F[i];
      b = off[u];
      e = off[u + 1];
    }
    // a hub's lanes list its chunks; where the list is full (a frontier that
    // holds ids twice) the places left say so and the group walks the hub itself
    const uint32_t nc = e - b >= hub_min ? (uint32_t)((e - b + kHubChunk - 1) / kHubChunk) : 0;
    unsigned long long at = 0;
    if (nc && gl == 0) at = atomicAdd(&st->ndefer, (unsigned long long)nc);
    at = __shfl_sync(kFull, at, g * GS);
    if (nc) {
      const bool fits = at + nc <= hub_cap;
      for (uint32_t c = gl; c < nc && at + c < hub_cap; c += GS) hubs[at + c] = make_uint2(fits ? u : kSentinel, c);
      if (fits) e = b;
    }
    uint64_t chunks = (e - b + GS - 1) / GS;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      uint64_t t = __shfl_xor_sync(kFull, chunks, o);
      chunks = t > chunks ? t : chunks;
    }
    for (uint64_t c = 0; c < chunks; c++) {
      const uint64_t j = b + c * GS + gl;
      const uint32_t us[1] = {u}, v[1] = {j < e ? slots[j] : kSentinel};
      visit_emit(us, v, lvl, lp, visited, out_list, out_bits, st, deg, dsum, wl, s_hist);
    }
  }
  round_flush(wl, out_list, st, dsum, s_hist);
}

// edgeMapDenseForward (edge_map_data.h:180-247): every vertex of a dense
// frontier pushes to its neighbours; a warp takes a 32-vertex bitmap word and
// walks the adjacency of each of its set bits with all lanes.
__global__ void __launch_bounds__(256) k_push_dense_fwd(const uint64_t *__restrict__ off,
                                                        const uint32_t *__restrict__ slots,
                                                        const uint32_t *__restrict__ deg,
                                                        const uint32_t *__restrict__ Fbits, uint64_t n,
                                                        uint64_t *lp, const uint32_t *__restrict__ visited,
                                                        uint32_t *out_list, uint32_t *out_bits, RoundStats *st,
                                                        uint64_t lvl) {
  __shared__ unsigned long long s_hist[8];
  hist_init(s_hist);
  __shared__ uint32_t s_list[8][kWarpListCap];
  WarpList<> wl{s_list[threadIdx.x >> 5]};
  const unsigned lane = lane_id();
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t W = (n + 31) / 32;
  uint64_t dsum = 0;
  for (uint64_t w = gw; w < W; w += nw) {
    unsigned word = Fbits[w];
    while (word) {
      const uint32_t u = (uint32_t)(w * 32 + __ffs(word) - 1);
      word &= word - 1;
      const uint64_t b = off[u], e = off[u + 1];
      for (uint64_t base = b; base < e; base += 32) {
        const uint64_t j = base + lane;
        bool em = false;
        uint32_t v = kSentinel;
        if (j < e) {
          v = slots[j];
          em = visit(u, v, lvl, lp, visited);
        }
        emit_next(em, v, out_list, out_bits, st, deg, dsum, wl, s_hist);
      }
    }
  }
  round_flush(wl, out_list, st, dsum, s_hist);
}

// A CTA per chunk of a hub (degree >= hub_min).
__global__ void __launch_bounds__(256) k_push_hubs(const uint64_t *__restrict__ off,
                                                   const uint32_t *__restrict__ slots,
                                                   const uint32_t *__restrict__ deg,
                                                   const uint2 *__restrict__ hubs, uint64_t hub_cap,
                                                   uint64_t *lp, const uint32_t *__restrict__ visited,
                                                   uint32_t *out_list, uint32_t *out_bits,
                                                   RoundStats *st, uint64_t lvl) {
  __shared__ unsigned long long s_hist[8];
  hist_init(s_hist);
  __shared__ uint32_t s_list[8][kWarpListCap];
  WarpList<> wl{s_list[threadIdx.x >> 5]};
  const uint64_t nd = *(volatile unsigned long long *)&st->ndefer, nh = nd < hub_cap ? nd : hub_cap;
  uint64_t dsum = 0;
  for (uint64_t h = blockIdx.x; h < nh; h += gridDim.x) {
    const uint32_t u = hubs[h].x;
    if (u == kSentinel) continue;
    const uint64_t b = off[u] + (uint64_t)hubs[h].y * kHubChunk, end = off[u + 1];
    const uint64_t e = b + kHubChunk < end ? b + kHubChunk : end;
    for (uint64_t base = b; base < e; base += 4 * blockDim.x) {
      uint32_t v[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint64_t j = base + q * blockDim.x + threadIdx.x;
        v[q] = j < e ? slots[j] : kSentinel;
      }
      const uint32_t us[4] = {u, u, u, u};
      visit_emit(us, v, lvl, lp, visited, out_list, out_bits, st, deg, dsum, wl, s_hist);
    }
  }
  round_flush(wl, out_list, st, dsum, s_hist);
}

// ---------------------------------------------------------------- blocked
// The last i in [0, n) with pre[i] <= x (pre[0] <= x), by a warp: 32 probes a
// step, so 2^20 entries take four waits for memory.
__device__ __forceinline__ uint64_t warp_last_le(const uint64_t *__restrict__ pre, uint64_t n, uint64_t x) {
  uint64_t lo = 0, len = n;  // the answer is in [lo, lo + len)
  while (len > 1) {
    const uint64_t step = (len + 31) / 32, at = lo + lane_id() * step;
    const unsigned m = __ballot_sync(kFull, lane_id() * step < len && pre[at] <= x);
    const int k = 31 - __clz((int)m);
    lo += (uint64_t)k * step;
    len = len - (uint64_t)k * step < step ? len - (uint64_t)k * step : step;
  }
  return lo;
}

// Edge-balanced: tile t covers frontier-edge ranks [t*TILE, (t+1)*TILE) of
// the exclusive degree prefix `pre`; each rank is mapped to its frontier
// vertex by binary search (the merge-path split of rank space).  The tile's
// part of the prefix and the vertices' slots are staged in shared memory, so an
// edge's search waits for no global memory, and a thread has 4 edges in flight
// (RMAT 2^20, a round over half the graph: 420 -> 375 us).
constexpr uint32_t kBlockedStage = 2048;
__global__ void __launch_bounds__(256) k_push_blocked(const uint64_t *__restrict__ off,
                                                      const uint32_t *__restrict__ slots,
                                                      const uint32_t *__restrict__ deg,
                                                      const uint32_t *__restrict__ F, uint64_t fsize,
                                                      const uint64_t *__restrict__ pre,
                                                      uint64_t *lp,
                                                      const uint32_t *__restrict__ visited,
                                                      uint32_t *out_list, uint32_t *out_bits,
                                                      RoundStats *st, uint64_t lvl, int tile) {
  __shared__ unsigned long long s_hist[8];
  hist_init(s_hist);
  __shared__ uint32_t s_list[8][kWarpListCap];
  WarpList<> wl{s_list[threadIdx.x >> 5]};
  __shared__ uint64_t s_slot[kBlockedStage];  // slot of a rank: rank + s_slot
  __shared__ uint32_t s_pre[kBlockedStage], s_u[kBlockedStage];
  __shared__ uint64_t s_lo, s_hi;
  const uint64_t total = pre[fsize];
  const uint64_t ntiles = (total + tile - 1) / tile;
  uint64_t dsum = 0;
  for (uint64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const uint64_t e0 = t * tile;
    const uint64_t e1 = e0 + tile < total ? e0 + tile : total;
    if (threadIdx.x < 64) {  // the first and the last vertex, a warp each
      const uint64_t i = warp_last_le(pre, fsize, threadIdx.x < 32 ? e0 : e1 - 1);
      if (threadIdx.x == 0) s_lo = i;
      if (threadIdx.x == 32) s_hi = i;
    }
    __syncthreads();
    const uint64_t vlo = s_lo, vhi = s_hi;
    // (a frontier may hold any number of vertices without slots)
    const bool staged = vhi - vlo < kBlockedStage;
    const uint32_t nv = (uint32_t)(vhi - vlo + 1);
    if (staged) {
      for (uint32_t i = threadIdx.x; i < nv; i += blockDim.x) {
        const uint32_t u = F[vlo + i];
        const uint64_t p = pre[vlo + i];
        s_u[i] = u;
        s_pre[i] = p > e0 ? (uint32_t)(p - e0) : 0;
        s_slot[i] = off[u] - p;
      }
      __syncthreads();
    }
    for (uint64_t base = e0; base < e1; base += 4 * blockDim.x) {
      uint32_t u[4], v[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint64_t e = base + q * blockDim.x + threadIdx.x;
        u[q] = 0;
        v[q] = kSentinel;
        if (e >= e1) continue;
        if (staged) {
          uint32_t lo = 0, hi = nv;
          while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (s_pre[mid] <= (uint32_t)(e - e0)) lo = mid; else hi = mid;
          }
          u[q] = s_u[lo];
          v[q] = slots[e + s_slot[lo]];
        } else {
          uint64_t lo = vlo, hi = vhi + 1;
          while (hi - lo > 1) {
            const uint64_t mid = (lo + hi) >> 1;
            if (pre[mid] <= e) lo = mid; else hi = mid;
          }
          u[q] = F[lo];
          v[q] = slots[off[u[q]] + (e - pre[lo])];
        }
      }
      visit_emit(u, v, lvl, lp, visited, out_list, out_bits, st, deg, dsum, wl, s_hist);
    }
    __syncthreads();
  }
  round_flush(wl, out_list, st, dsum, s_hist);
}

// ---------------------------------------------------------------- pull
__device__ __forceinline__ bool in_frontier(const uint32_t *s_bits, int stage_words,
                                            const uint32_t *__restrict__ Fbits, uint32_t u) {
  uint32_t w = u >> 5;
  uint32_t word = (w < (uint32_t)stage_words) ? s_bits[w] : __ldg(Fbits + w);
  return (word >> (u & 31)) & 1u;
}

// A thread per unvisited vertex.  Found and deferred vertices go out through
// WarpLists: an add to the two counters from every warp held the first dense
// round at RMAT 2^22 up by a third (138 us, 96 now).  The lists take what L1 has
// for the ids and bits of a round that finds few: BFS by pulls alone on a uniform
// graph of 10^6 vertices and degree 16 594 us with room for 96 entries, words and
// slots counted in 64 bits (which spills) and an add after the other at the end;
// 584 without those two; 560 with room for 64 as well (without lists 557).
constexpr uint32_t kPullListCap = 64;
__global__ void __launch_bounds__(1024, 2) k_pull(const uint64_t *__restrict__ off,
                                               const uint32_t *__restrict__ slots,
                                               const uint32_t *__restrict__ deg,
                                               const uint32_t *__restrict__ Fbits, uint64_t n,
                                               uint64_t *__restrict__ lp, uint32_t *visited,
                                               uint32_t *out_list, uint32_t *out_bits,
                                               RoundStats *st, uint64_t lvl, uint32_t *defer,
                                               int cap, int stage_words) {
  extern __shared__ uint32_t s_bits[];
  __shared__ unsigned long long s_hist[8];
  __shared__ uint32_t s_list[2][32][kPullListCap];
  WarpList<kPullListCap> wl{s_list[0][threadIdx.x >> 5]}, wdefer{s_list[1][threadIdx.x >> 5]};
  for (int i = threadIdx.x; i < stage_words; i += blockDim.x) s_bits[i] = Fbits[i];
  if (threadIdx.x < 8) s_hist[threadIdx.x] = 0;
  __syncthreads();
  const uint32_t W = (uint32_t)((n + 31) >> 5);
  const unsigned lane = lane_id();
  const uint32_t nw = gridDim.x * (blockDim.x >> 5);
  uint64_t dsum = 0;
  for (uint32_t w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < W; w += nw) {
    const uint32_t vword = visited[w];
    if (vword == kFull) continue;
    const uint32_t v = w * 32 + lane;
    bool found = false, deferred = false;
    uint32_t parent = 0;
    if (v < n && !((vword >> lane) & 1u)) {
      const uint64_t b = off[v], len = off[v + 1] - b;
      const uint32_t *const ids = slots + b;
      const uint32_t lim = (uint32_t)min(len, (uint64_t)cap);
      // eight neighbours at a time: their ids, then their frontier bits, are
      // loaded together; the first hit in slot order is the parent
      for (uint32_t j0 = 0; j0 < lim && !found; j0 += 8) {
        uint32_t u[8];
#pragma unroll
        for (int q = 0; q < 8; q++) u[q] = j0 + q < lim ? ids[j0 + q] : kSentinel;
        bool h[8];
#pragma unroll
        for (int q = 0; q < 8; q++) h[q] = u[q] != kSentinel && in_frontier(s_bits, stage_words, Fbits, u[q]);
#pragma unroll
        for (int q = 7; q >= 0; q--)
          if (h[q]) {
            found = true;
            parent = u[q];
          }
      }
      deferred = !found && len > lim;
    }
    if (found) lp[v] = lvl | parent;
    const unsigned fb = __ballot_sync(kFull, found);
    if (lane == 0 && fb) {
      out_bits[w] = fb;
      visited[w] |= fb;
    }
    wl.add(found, v, out_list, &st->count);
    uint32_t d = 0;
    if (found) {
      d = deg[v];
      dsum += d;
    }
    hist_warp_add(s_hist, found, d);
    wdefer.add(deferred, v, defer, &st->ndefer);
  }
  round_flush(wl, out_list, st, dsum, s_hist, &wdefer, defer);
}

// Warp per deferred vertex: 32 neighbours per step, ballot, lowest lane wins.
__global__ void __launch_bounds__(256) k_pull_long(const uint64_t *__restrict__ off,
                                                   const uint32_t *__restrict__ slots,
                                                   const uint32_t *__restrict__ deg,
                                                   const uint32_t *__restrict__ Fbits,
                                                   uint64_t *__restrict__ lp, uint32_t *visited,
                                                   uint32_t *out_list, uint32_t *out_bits,
                                                   RoundStats *st, uint64_t lvl,
                                                   const uint32_t *__restrict__ defer, int cap, PolicyTail pt) {
  __shared__ float4 sP[kParamChunks];
  __shared__ unsigned long long s_hist[8];
  policy_prefetch(pt, sP);
  hist_init(s_hist);
  const uint64_t nd = *(volatile unsigned long long *)&st->ndefer;
  const unsigned lane = lane_id();
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t i = gw; i < nd; i += nw) {
    const uint32_t v = defer[i];
    const uint64_t b = off[v] + cap, e = off[v + 1];
    bool found = false;
    uint32_t parent = 0;
    for (uint64_t base = b; base < e && !found; base += 32) {
      uint64_t j = base + lane;
      uint32_t u = j < e ? slots[j] : kSentinel;
      bool hit = u != kSentinel && ((__ldg(Fbits + (u >> 5)) >> (u & 31)) & 1u);
      unsigned m = __ballot_sync(kFull, hit);
      if (m) {
        found = true;
        parent = __shfl_sync(kFull, u, __ffs(m) - 1);
      }
    }
    uint32_t d = 0;
    if (found && lane == 0) {
      lp[v] = lvl | parent;
      atomicOr(out_bits + (v >> 5), 1u << (v & 31));
      atomicOr(visited + (v >> 5), 1u << (v & 31));
      unsigned long long slot = atomicAdd(&st->count, 1ull);
      out_list[slot] = v;
      d = deg[v];
      atomicAdd(&st->outdeg, (unsigned long long)d);
    }
    hist_warp_add(s_hist, found && lane == 0, d);
  }
  hist_flush(s_hist, st);
  policy_tail(pt, st, sP);
}

// ---------------------------------------------------------------- bookkeeping
__global__ void k_mark_visited(const uint32_t *__restrict__ list, RoundStats *st, uint32_t *visited,
                               PolicyTail pt) {
  __shared__ float4 sP[kParamChunks];
  policy_prefetch(pt, sP);
  const uint64_t cnt = st->count;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < cnt;
       i += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t v = list[i];
    atomicOr(visited + (v >> 5), 1u << (v & 31));
  }
  policy_tail(pt, st, sP);
}

__global__ void k_clear_words_from_list(const uint32_t *__restrict__ list, uint64_t cnt,
                                        uint32_t *bits) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < cnt;
       i += (uint64_t)gridDim.x * blockDim.x)
    bits[list[i] >> 5] = 0;  // every set bit of `bits` belongs to some list entry
}

__global__ void k_set_bits_from_list(const uint32_t *__restrict__ list, uint64_t cnt, uint32_t *bits) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < cnt;
       i += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t v = list[i];
    atomicOr(bits + (v >> 5), 1u << (v & 31));
  }
}

__global__ void k_trav_init(uint64_t *lp, uint32_t *visited, uint64_t n, uint32_t src) {
  const uint64_t W = (n + 31) >> 5;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    lp[i] = (i == src) ? (uint64_t)src : kNone64;
    if (i < W) visited[i] = (i == (src >> 5)) ? (1u << (src & 31)) : 0u;
  }
}

// Everything a BFS from src starts from: lp, visited, both frontier bitmaps and
// the first frontier.
__global__ void k_bfs_start(uint64_t *lp, uint32_t *visited, uint32_t *list, uint32_t *bits, uint32_t *next_bits,
                            uint64_t n, uint32_t src) {
  const uint64_t W = (n + 31) >> 5;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    lp[i] = (i == src) ? (uint64_t)src : kNone64;
    if (i < W) {
      visited[i] = bits[i] = (i == (src >> 5)) ? (1u << (src & 31)) : 0u;
      next_bits[i] = 0;
    }
    if (i == 0) list[0] = src;
  }
}

__global__ void k_trav_extract(const uint64_t *__restrict__ lp, uint64_t n, uint32_t *parent,
                               uint32_t *level) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t x = lp[i];
    if (parent) parent[i] = x == kNone64 ? kSentinel : (uint32_t)x;
    if (level) level[i] = x == kNone64 ? kSentinel : (uint32_t)(x >> 32);
  }
}

// ---------------------------------------------------------------- host side

byo_tuning effective_tuning(const byo_graph *g) {
  byo_tuning t = g->tune;
  const double avg = g->n ? (double)g->m / (double)g->n : 0.0;
  if (!t.push_group) t.push_group = avg >= 24 ? 32 : avg >= 12 ? 16 : avg >= 6 ? 8 : 4;
  if (!t.hub_min) t.hub_min = 4096;
  if (!t.pull_cap) t.pull_cap = 32;
  if (!t.blocked_tile) t.blocked_tile = 2048;
  if (!t.ms_heavy_deg) t.ms_heavy_deg = 48;
  if (!t.ms_hub_deg) t.ms_hub_deg = 1024;
  if (!t.ms_push_div) t.ms_push_div = 20;
  if (!t.tc_stage) t.tc_stage = 40960;
  t.reserved = 0;
  if (!t.pull_stage_words) {
    const uint64_t W = (g->n + 31) / 32;
    t.pull_stage_words = (uint32_t)(W < 16384 ? (W < 256 ? 256 : W) : 16384);
  }
  return t;
}

// Shared memory of k_pull: what it has besides the staged words (its lists; the
// compiler's figure), the most words (check_tuning), and the bytes of words up to
// which two CTAs share an SM's 228 KB.
constexpr int kPullStatic = 17216, kPullMaxStage = 49152;
constexpr int kPullPairBytes = (228 * 1024) / 2 - 1024 - kPullStatic;

int check_tuning(byo_ctx *ctx, const byo_tuning *t) {
  const char *bad = nullptr;
  if (t->push_group && t->push_group != 4 && t->push_group != 8 && t->push_group != 16 && t->push_group != 32)
    bad = "push_group must be 4, 8, 16 or 32";
  else if (t->hub_min && t->hub_min < 32)
    bad = "hub_min must be >= 32";
  else if (t->pull_cap > 4096)
    bad = "pull_cap must be <= 4096";
  else if (t->blocked_tile && (t->blocked_tile < 64 || t->blocked_tile > 65536))
    bad = "blocked_tile must be in [64, 65536]";
  else if (t->ms_heavy_deg > 65536)
    bad = "ms_heavy_deg must be <= 65536";
  else if (t->ms_hub_deg && (t->ms_hub_deg < 32 || t->ms_hub_deg > (1u << 20)))
    bad = "ms_hub_deg must be in [32, 2^20]";
  else if (t->pull_stage_words && (t->pull_stage_words < 256 || t->pull_stage_words > kPullMaxStage))
    bad = "pull_stage_words must be in [256, 49152]";
  else if (t->tc_stage && (t->tc_stage < 512 || t->tc_stage > 49152))
    bad = "tc_stage must be in [512, 49152]";
  else if (t->reserved)
    bad = "reserved field must be zero";
  return bad ? set_error(ctx, BYO_EINVAL, bad) : BYO_OK;
}

EngineTuning default_tuning(const byo_graph *g) {
  EngineTuning t;
  const uint64_t W = (g->n + 31) / 32;
  const byo_tuning e = effective_tuning(g);
  t.pull_stage_words = (int)(W < e.pull_stage_words ? W : e.pull_stage_words);
  t.push_group = (int)e.push_group;
  t.hub_min = e.hub_min;
  t.pull_cap = (int)e.pull_cap;
  t.blocked_tile = (int)e.blocked_tile;
  return t;
}

int m20_mode(const byo_graph *g, const Frontier &f, int64_t threshold, int sparse_mode) {
  const uint64_t n = g->n, M = g->m;
  const uint64_t dense_threshold = threshold < 0 ? M / 20 : (uint64_t)threshold;
  if (f.dense && f.size > n / 10) return MODE_PULL;
  if (f.size + f.outdeg > dense_threshold) return MODE_PULL;
  return sparse_mode;
}

int trav_init(byo_graph *g, TravState &st, uint32_t src) {
  byo_ctx *ctx = g->ctx;
  launch(ctx, k_trav_init, dim3(grid_for(ctx, g->n, 256)), dim3(256), 0, st.lp, st.visited, g->n, src);
  st.round = 1;
  st.reached = 1;
  return check_launch(ctx, "trav_init");
}

int trav_extract(byo_graph *g, const TravState &st, uint32_t *d_parent, uint32_t *d_level) {
  byo_ctx *ctx = g->ctx;
  launch(ctx, k_trav_extract, dim3(grid_for(ctx, g->n, 256)), dim3(256), 0, (const uint64_t *)st.lp,
         g->n, d_parent, d_level);
  return check_launch(ctx, "trav_extract");
}

int clear_frontier_bits(byo_graph *g, Frontier &f) {
  byo_ctx *ctx = g->ctx;
  const uint64_t W = (g->n + 31) / 32;
  if (f.has_list && f.size < W / 8) {
    if (f.size)
      launch(ctx, k_clear_words_from_list, dim3(grid_for(ctx, f.size, 256)), dim3(256), 0,
             (const uint32_t *)f.list, f.size, f.bits);
  } else {
    BYO_TRY(memset_async(ctx, f.bits, 0, W * sizeof(uint32_t)));
  }
  return check_launch(ctx, "clear_frontier_bits");
}

int ensure_bits(byo_graph *g, Frontier &f) {
  if (f.has_bits) return BYO_OK;
  byo_ctx *ctx = g->ctx;
  const uint64_t W = (g->n + 31) / 32;
  BYO_TRY(memset_async(ctx, f.bits, 0, W * sizeof(uint32_t)));
  if (f.size)
    launch(ctx, k_set_bits_from_list, dim3(grid_for(ctx, f.size, 256)), dim3(256), 0,
           (const uint32_t *)f.list, f.size, f.bits);
  f.has_bits = true;
  return check_launch(ctx, "ensure_bits");
}

int edge_map_round(byo_graph *g, TravState &st, Frontier &in, Frontier &out, int mode,
                   const EngineTuning &tune, bool run_policy) {
  byo_ctx *ctx = g->ctx;
  RoundStats *d_st = nullptr;
  BYO_TRY(ws(g, WS_STATS, sizeof(RoundStats) / sizeof(uint64_t) + 2, (uint64_t **)&d_st));
  BYO_CU(ctx, cudaMemsetAsync(d_st, 0, sizeof(RoundStats) + 8, ctx->stream));
  // the policy for the next round runs as the epilogue of this round's last kernel
  PolicyTail pt;
  if (run_policy) BYO_TRY(policy_tail_args(g, (unsigned int *)(d_st + 1), st.reached, mode == MODE_PULL, &pt));
  // pull: deferred vertices; push: hub chunks (a frontier without repeats holds
  // at most so many)
  uint32_t *defer = nullptr;
  const uint64_t hub_cap = g->nslots / kHubChunk + g->nslots / tune.hub_min + 1;
  BYO_TRY(ws(g, WS_DEFER, std::max<uint64_t>(g->n + 1, 2 * hub_cap), &defer));
  const uint64_t lvl = (uint64_t)st.round << 32;
  if (mode == MODE_PULL) {
    BYO_TRY(ensure_bits(g, in));
    const int stage = tune.pull_stage_words, smem = stage * 4;
    // the attribute is the device's, and other contexts set it too: always the
    // same value, and no record of having set it
    BYO_CU(ctx, cudaFuncSetAttribute(k_pull, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kPullMaxStage));
    const uint64_t W = (g->n + 31) / 32;
    int block = 1024;
    int grid = (int)((W + 31) / 32);
    int maxg = ctx->num_sms * (smem > kPullPairBytes ? 1 : 2);
    if (grid > maxg) grid = maxg;
    if (grid < 1) grid = 1;
    launch_t(ctx, "bfs_pull", k_pull, dim3(grid), dim3(block), (size_t)smem, (const uint64_t *)g->d_off,
           (const uint32_t *)g->d_slots, (const uint32_t *)g->d_deg, (const uint32_t *)in.bits, g->n,
           st.lp, st.visited, out.list, out.bits, d_st, lvl, defer, tune.pull_cap, stage);
    pt.prefetch = 1;
    launch(ctx, k_pull_long, dim3(ctx->num_sms * 4), dim3(256), 0, (const uint64_t *)g->d_off,
           (const uint32_t *)g->d_slots, (const uint32_t *)g->d_deg, (const uint32_t *)in.bits, st.lp,
           st.visited, out.list, out.bits, d_st, lvl, (const uint32_t *)defer, tune.pull_cap, pt);
  } else {
    if (mode == MODE_DENSE_FWD) {
      BYO_TRY(ensure_bits(g, in));
      const uint64_t W = (g->n + 31) / 32;
      launch_t(ctx, "bfs_push", k_push_dense_fwd, dim3(grid_for(ctx, W * 32, 256, 16)), dim3(256), 0,
               (const uint64_t *)g->d_off, (const uint32_t *)g->d_slots, (const uint32_t *)g->d_deg,
               (const uint32_t *)in.bits, g->n, st.lp, (const uint32_t *)st.visited, out.list, out.bits, d_st, lvl);
    } else if (!in.has_list) {
      return set_error(ctx, BYO_EINVAL, "sparse round needs a frontier list");
    } else if (mode == MODE_PUSH) {
      const int grid = grid_for(ctx, (in.size * (uint64_t)tune.push_group + 255) / 256 * 256, 256, 16);
      switch (tune.push_group) {
#define PUSH_CASE(GS)                                                                            \
  case GS:                                                                                       \
    launch_t(ctx, "bfs_push", k_push<GS>, dim3(grid), dim3(256), 0, (const uint64_t *)g->d_off,                \
           (const uint32_t *)g->d_slots, (const uint32_t *)g->d_deg, (const uint32_t *)in.list,  \
           in.size, st.lp, (const uint32_t *)st.visited, out.list, out.bits, d_st, lvl,          \
           (uint2 *)defer, hub_cap, tune.hub_min);                                                                     \
    break;
        PUSH_CASE(4)
        PUSH_CASE(8)
        PUSH_CASE(16)
        PUSH_CASE(32)
#undef PUSH_CASE
        default:
          return set_error(ctx, BYO_EINVAL, "push group must be 4, 8, 16 or 32");
      }
      launch(ctx, k_push_hubs, dim3(ctx->num_sms * 2), dim3(256), 0, (const uint64_t *)g->d_off,
             (const uint32_t *)g->d_slots, (const uint32_t *)g->d_deg, (const uint2 *)defer, hub_cap, st.lp,
             (const uint32_t *)st.visited, out.list, out.bits, d_st, lvl);
    } else {
      uint64_t *pre = nullptr;
      BYO_TRY(ws(g, WS_SCAN, in.size + 1, &pre));
      // prefix over slot-range lengths (= degrees for a CSR; gaps included
      // for the PMA so ranks map to slots)
      BYO_TRY(scan_gather_range(ctx, g->d_off, in.list, in.size, pre));
      const uint64_t est_tiles = (in.outdeg + tune.blocked_tile - 1) / tune.blocked_tile;
      const int grid = grid_for(ctx, est_tiles ? est_tiles : 1, 1, 16);
      launch_t(ctx, "bfs_blocked", k_push_blocked, dim3(grid), dim3(256), 0, (const uint64_t *)g->d_off,
             (const uint32_t *)g->d_slots, (const uint32_t *)g->d_deg, (const uint32_t *)in.list,
             in.size, (const uint64_t *)pre, st.lp, (const uint32_t *)st.visited, out.list, out.bits,
             d_st, lvl, tune.blocked_tile);
    }
    const int mgrid = grid_for(ctx, in.outdeg + 1, 256);
    pt.prefetch = mgrid >= ctx->num_sms;
    launch(ctx, k_mark_visited, dim3(mgrid), dim3(256), 0, (const uint32_t *)out.list, d_st, st.visited, pt);
  }
  BYO_TRY(check_launch(ctx, "edge_map_round"));
  RoundStats *h = nullptr;
  BYO_TRY(pinned(ctx, 4096, (void **)&h));
  BYO_CU(ctx, cudaMemcpyAsync(h, d_st, sizeof(RoundStats), cudaMemcpyDeviceToHost, ctx->stream));
  BYO_CU(ctx, cudaStreamSynchronize(ctx->stream));
  out.size = h->count;
  out.outdeg = h->outdeg;
  for (int i = 0; i < 8; i++) out.hist[i] = h->hist[i];
  if (run_policy) {
    out.next_mode = (int)h->mode;
    for (int i = 0; i < 16; i++) out.feat[i] = h->feat[i];
  }
  out.dense = (mode == MODE_PULL || mode == MODE_DENSE_FWD);
  out.has_list = true;
  out.has_bits = true;
  st.round++;
  st.reached += out.size;
  return BYO_OK;
}

// ---------------------------------------------------------------- BFS driver

int bfs_run(byo_graph *g, uint32_t src, uint32_t *d_parent, uint32_t *d_level, int policy,
            uint32_t *rounds) {
  byo_ctx *ctx = g->ctx;
  if (src >= g->n) return set_error(ctx, BYO_EINVAL, "bfs: src >= n");
  const uint64_t n = g->n, W = (n + 31) / 32;
  TravState st;
  Frontier fa, fb;
  BYO_TRY(ws(g, WS_LP, n, &st.lp));
  BYO_TRY(ws(g, WS_VISITED, W, &st.visited));
  BYO_TRY(ws(g, WS_FRONT_LIST_A, n, &fa.list));
  BYO_TRY(ws(g, WS_FRONT_LIST_B, n, &fb.list));
  BYO_TRY(ws(g, WS_FRONT_BITS_A, W, &fa.bits));
  BYO_TRY(ws(g, WS_FRONT_BITS_B, W, &fb.bits));
  launch(ctx, k_bfs_start, dim3(grid_for(ctx, n, 256)), dim3(256), 0, st.lp, st.visited, fa.list, fa.bits, fb.bits, n,
         src);
  BYO_TRY(check_launch(ctx, "bfs_start"));
  st.round = 1;
  st.reached = 1;
  fa.size = 1;
  fa.has_list = fa.has_bits = true;
  fb.size = 0;
  fb.has_list = true;  // empty list: its bitmap is all zero
  const EngineTuning tune = default_tuning(g);
  ctx->rounds.clear();
  // features (and the learned choice) are computed on the device after every
  // round when the learned policy runs or rounds are being logged
  const bool run_policy = policy == BYO_POLICY_LEARNED || ctx->time_rounds;
  Frontier *cur = &fa, *nxt = &fb;
  uint32_t nr = 0;
  // small push rounds run back to back in one persistent kernel (not while
  // rounds are timed one by one for the policy's training samples)
  const bool small_ok = !ctx->time_rounds &&
                        (policy == BYO_POLICY_M20 || policy == BYO_POLICY_LEARNED || policy == BYO_POLICY_PUSH);
  // The learned policy inspects frontiers near the m/20 threshold and those
  // holding a vertex of degree >= 4^5; a rule does not, and up to kSmallEdges
  // edges a round costs less there (under 10 us) than any round driven from the
  // host (~30 us).
  const bool gate_hub = policy == BYO_POLICY_LEARNED;
  const uint64_t small_limit = gate_hub ? std::max<uint64_t>(4096, g->m / 20 / 64) : kSmallEdges;
  if (small_ok && !gate_hub) {
    // start there without asking the host for the source's degree
    BYO_TRY(bfs_small_rounds(g, st, cur, nxt, small_limit, false, nullptr, &nr));
  } else {
    uint32_t dsrc = 0;
    BYO_CU(ctx, cudaMemcpyAsync(&dsrc, g->d_deg + src, 4, cudaMemcpyDeviceToHost, ctx->stream));
    BYO_CU(ctx, cudaStreamSynchronize(ctx->stream));
    fa.outdeg = dsrc;
    fa.hist[log4_bin(dsrc)] = 1;
    if (run_policy) {
      RoundStats *d_st = nullptr, *h = nullptr;
      BYO_TRY(ws(g, WS_STATS, sizeof(RoundStats) / sizeof(uint64_t) + 2, (uint64_t **)&d_st));
      BYO_TRY(pinned(ctx, 4096, (void **)&h));
      std::memset(h, 0, sizeof(RoundStats));
      h->count = 1;
      h->outdeg = dsrc;
      int bin = dsrc ? (31 - __builtin_clz(dsrc)) / 2 : 0;
      h->hist[bin > 7 ? 7 : bin] = 1;
      BYO_CU(ctx, cudaMemcpyAsync(d_st, h, sizeof(RoundStats), cudaMemcpyHostToDevice, ctx->stream));
      BYO_TRY(round_policy(g, d_st, 0, false));
      BYO_CU(ctx, cudaMemcpyAsync(h, d_st, sizeof(RoundStats), cudaMemcpyDeviceToHost, ctx->stream));
      BYO_CU(ctx, cudaStreamSynchronize(ctx->stream));
      fa.next_mode = (int)h->mode;
      for (int i = 0; i < 16; i++) fa.feat[i] = h->feat[i];
    }
  }
  while (cur->size > 0) {
    int mode;
    switch (policy) {
      case BYO_POLICY_PUSH: mode = MODE_PUSH; break;
      case BYO_POLICY_PULL: mode = MODE_PULL; break;
      case BYO_POLICY_BLOCKED: mode = MODE_BLOCKED; break;
      case BYO_POLICY_M20_BLOCKED: mode = m20_mode(g, *cur, -1, MODE_BLOCKED); break;
      case BYO_POLICY_LEARNED: mode = cur->next_mode; break;  // network, or m/20 if untrained
      default: mode = m20_mode(g, *cur, -1, MODE_PUSH); break;
    }
    if (mode != MODE_PULL && cur->outdeg == 0) break;  // edge_map_data.h:290
    // next's bitmap still holds the frontier before `cur`: clear it
    BYO_TRY(clear_frontier_bits(g, *nxt));
    bool hub = false;
    for (int q = 5; q < 8; q++) hub |= cur->hist[q] != 0;
    if (small_ok && mode != MODE_BLOCKED && (mode == MODE_PUSH || !gate_hub) && cur->has_list &&
        cur->outdeg && cur->size + cur->outdeg <= std::min(small_limit, kSmallEdges) && !(gate_hub && hub)) {
      RoundStats *d_st = nullptr;
      BYO_TRY(ws(g, WS_STATS, sizeof(RoundStats) / sizeof(uint64_t) + 2, (uint64_t **)&d_st));
      uint32_t R = 0;
      BYO_TRY(bfs_small_rounds(g, st, cur, nxt, small_limit, gate_hub, run_policy ? d_st : nullptr, &R));
      nr += R;
      if (R == 0) return set_error(ctx, BYO_EDEVICE, "bfs: small rounds did not run");
      if (run_policy && cur->size > 0) {
        // the policy for the frontier the kernel stopped at
        RoundStats *h = nullptr;
        BYO_TRY(round_policy(g, d_st, st.reached - cur->size, false));
        BYO_TRY(pinned(ctx, 4096, (void **)&h));
        BYO_CU(ctx, cudaMemcpyAsync(h, d_st, sizeof(RoundStats), cudaMemcpyDeviceToHost, ctx->stream));
        BYO_CU(ctx, cudaStreamSynchronize(ctx->stream));
        cur->next_mode = (int)h->mode;
        for (int i = 0; i < 16; i++) cur->feat[i] = h->feat[i];
      }
      continue;
    }
    byo_round_log lg{};
    lg.round = st.round;
    lg.mode = (uint32_t)mode;
    lg.frontier = cur->size;
    lg.frontier_deg = cur->outdeg;
    lg.unvisited = n - st.reached;
    for (int i = 0; i < 16; i++) lg.features[i] = cur->feat[i];
    if (ctx->time_rounds) BYO_CU(ctx, cudaEventRecord(ctx->ev[0], ctx->stream));
    nxt->size = 0;
    BYO_TRY(edge_map_round(g, st, *cur, *nxt, mode, tune, run_policy));
    if (ctx->time_rounds) {
      BYO_CU(ctx, cudaEventRecord(ctx->ev[1], ctx->stream));
      BYO_CU(ctx, cudaEventSynchronize(ctx->ev[1]));
      cudaEventElapsedTime(&lg.ms, ctx->ev[0], ctx->ev[1]);
    }
    ctx->rounds.push_back(lg);
    nr++;
    Frontier *t = cur;
    cur = nxt;
    nxt = t;
  }
  if (rounds) *rounds = nr;
  return trav_extract(g, st, d_parent, d_level);
}

}  // namespace byo
