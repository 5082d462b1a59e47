// bfs_small.cu -- consecutive small push rounds of a BFS in one kernel, a
// cluster of 8 CTAs.
//
// A push round over a frontier of a few thousand edges takes a few
// microseconds of GPU work, but driving it from the host (launches, a copy of
// the round statistics, a stream synchronisation) costs ~30 us.  On graphs of
// high diameter (grids, road-like graphs) nearly every round is like that, and
// on small graphs every one.  This kernel runs such rounds back to back with
// the same visit rule as the push kernels (BFS_F's updateAtomic keeping the
// smallest (level, parent), BFS.h:30-45), so the result does not depend on
// which rounds it ran.  It leaves as soon as the next frontier is empty,
// grows past `limit` edges or (gate_hub) holds a vertex of degree >= 4^5, and
// hands the host the frontier in the engine's form (list + bitmap, its size,
// out-degree and degree sketch), so the round loop continues from there.  It
// counts slots as edges: a BFS runs on a view without gaps (traversal_view).
//
// A round is bound by the chain of dependent L2 accesses, so the chain is
// kept short: a frontier entry carries its slot range, fetched when the vertex
// was discovered, beside the atomicMin; a CTA appends to its own segment
// through a shared counter; and the barrier is between the CTAs' shared
// memories (an arrival is a remote add, the wait a local poll), carrying the
// segments' sizes.  One barrier a round: a vertex counts as unvisited when its
// lp was never written, so no bitmap has to be settled between rounds.
// Grid 1277 x 1531, 2800 rounds: 7.6 ms, 2.7 us a round; a cooperative grid of two
// CTAs an SM with two barriers in global memory took 5.9 us a round, and left the
// rounds of more than 4096 edges to the host: 38 ms.  A 4096-vertex RMAT graph:
// 201 -> 67 us.
#include <algorithm>
#include <cstring>
#include <vector>

#include "device.cuh"
#include "engine.h"
#include "gridsync.cuh"
#include "internal.h"

namespace byo {

namespace {

constexpr int kSmallBlock = 1024;
constexpr uint32_t kSmallCtas = 8;
constexpr uint32_t kSmallWarps = kSmallCtas * kSmallBlock / 32;
constexpr uint32_t kSmallLog = 1u << 16;  // rounds one launch may run (and log)
// Entries of up to kSmallLen slots take 4 to 32 lanes; a longer one's slots are cut
// into pieces of kSmallPiece, a warp each: the first with the entry itself, the
// others listed beside it.  Pieces that find no room there belong to a frontier
// of more than kSmallEdges slots, which ends the run.
constexpr uint32_t kSmallLen = 64, kSmallPiece = 512, kSmallPieces = kSmallEdges / kSmallPiece;

// A frontier vertex and its slots.
struct __align__(16) SmallEntry {
  uint64_t b;
  uint32_t len, v;
};

// What the host reads: every word is written by the kernel.
struct SmallOut {
  unsigned long long size, edges, first_edges;  // of the frontier reached; the first frontier's slots
  unsigned long long hist[kSmallCtas][8];
  unsigned int rounds, pad, err[kSmallCtas];
};

struct SmallArgs {
  const uint64_t *off;
  const uint32_t *slots;
  uint64_t *lp;
  uint32_t *visited;
  uint32_t *list;  // the frontier to start from, then the one reached
  uint32_t *bits;
  uint64_t size, limit;
  uint32_t round0;
  int gate_hub;
  uint32_t limit_ms, extra;  // the barrier's time limit and the test hook's extra arrivals
  SmallEntry *seg;           // [2][kSmallCtas][cap + kSmallPieces]
  uint64_t cap;
  SmallOut *out;
  unsigned long long *log;  // per round: |F| and the next frontier's out-degree
};

__device__ __forceinline__ int small_bin(uint32_t d) {
  int b = d ? (31 - __clz(d)) / 2 : 0;
  return b > 7 ? 7 : b;
}

// What a CTA found in a round: short entries from the front of its segment,
// longer ones from the back and pieces of those behind it, their slots,
// whether one has 4^5 or more (kSmallBig in `hub`, as published).
struct __align__(16) SmallFound {
  unsigned int small, hub;
  unsigned long long edges;
  unsigned int pieces, pad[3];
};
constexpr unsigned kSmallBig = 1u << 31;

struct SmallShared {
  SmallFound from[2][kSmallCtas];    // published with the barrier, by parity
  SmallFound mine;                   // being collected
  unsigned int mine_big;
  unsigned int arrived;              // arrivals of all CTAs, over all barriers
  unsigned int pre[kSmallCtas + 1];  // short entries before each segment
  unsigned int long_pre[2 * kSmallCtas + 1];  // longer entries, then pieces, before each
  unsigned int hubs[kSmallCtas];
  unsigned int nhub, big, ok;
  unsigned long long edges;
};

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t remote_addr(uint32_t local, uint32_t cta) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(cta));
  return r;
}
__device__ __forceinline__ void cluster_hw_sync() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}

// The end of a round: publishes what this CTA found, waits (for a bounded
// time) until all have, and lays the segments out.  Lane i of the first warp
// writes to CTA i and releases it with an add to its arrival count.
__device__ __forceinline__ bool small_sync(SmallShared &s, const SmallArgs &a, unsigned rank, unsigned turn) {
  __syncthreads();
  if (threadIdx.x < 32) {
    const unsigned lane = threadIdx.x;
    if (lane < kSmallCtas) {
      const uint32_t to = remote_addr(smem_addr(&s.from[turn & 1][rank]), lane);
      const unsigned hub = s.mine.hub | (s.mine_big ? kSmallBig : 0u);
      asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(to), "r"(s.mine.small), "r"(hub),
                   "r"((unsigned)s.mine.edges), "r"((unsigned)(s.mine.edges >> 32))
                   : "memory");
      asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(to + 16), "r"(min(s.mine.pieces, kSmallPieces)) : "memory");
      asm volatile("red.release.cluster.shared::cluster.add.u32 [%0], %1;" ::"r"(
                       remote_addr(smem_addr(&s.arrived), lane)),
                   "r"(1u)
                   : "memory");
    }
    const unsigned need = (turn + 1) * (kSmallCtas + a.extra);
    const uint64_t limit = a.limit_ms ? (uint64_t)a.limit_ms * 1000000ull : kBarrierNs;
    const uint64_t t0 = globaltimer_ns();
    bool ok = true;
    for (unsigned spin = 1;; spin++) {
      unsigned got;
      asm volatile("ld.acquire.cluster.shared::cta.u32 %0, [%1];" : "=r"(got) : "r"(smem_addr(&s.arrived)) : "memory");
      if (got >= need) break;
      if (spin % 256 == 0 && globaltimer_ns() - t0 > limit) {
        ok = false;
        break;
      }
    }
    ok = !__any_sync(kFull, !ok);
    SmallFound f{};
    if (ok && lane < kSmallCtas) f = s.from[turn & 1][lane];
    const bool big = __any_sync(kFull, (f.hub & kSmallBig) != 0);
    const unsigned hub = f.hub & ~kSmallBig;
    unsigned small = f.small, hubs = hub, pieces = f.pieces;  // inclusive scans over the 8 lanes
    unsigned long long edges = f.edges;
#pragma unroll
    for (int o = 1; o < (int)kSmallCtas; o <<= 1) {
      const unsigned ps = __shfl_up_sync(kFull, small, o, kSmallCtas), ph = __shfl_up_sync(kFull, hubs, o, kSmallCtas);
      const unsigned pp = __shfl_up_sync(kFull, pieces, o, kSmallCtas);
      const unsigned long long pe = __shfl_up_sync(kFull, edges, o, kSmallCtas);
      if (lane % kSmallCtas >= (unsigned)o) {
        small += ps;
        hubs += ph;
        pieces += pp;
        edges += pe;
      }
    }
    const unsigned nhub = __shfl_sync(kFull, hubs, kSmallCtas - 1);
    if (lane < kSmallCtas) {
      s.pre[lane] = small - f.small;
      s.long_pre[lane] = hubs - hub;
      s.long_pre[kSmallCtas + lane] = nhub + pieces - f.pieces;
      s.hubs[lane] = hub;
    }
    if (lane == kSmallCtas - 1) {
      s.pre[kSmallCtas] = small;
      s.long_pre[2 * kSmallCtas] = nhub + pieces;
      s.nhub = nhub;
      s.edges = edges;
      s.big = big;
      s.ok = ok;
      s.mine = SmallFound{};
      s.mine_big = 0;
    }
  }
  __syncthreads();
  return s.ok != 0;
}

// Adds v to the CTA's segment.
__device__ __forceinline__ void small_add(SmallShared &s, SmallEntry *seg, uint64_t cap, uint32_t v, uint64_t b,
                                          uint32_t len) {
  if (len <= kSmallLen) {
    seg[atomicAdd(&s.mine.small, 1u)] = SmallEntry{b, len, v};
    return;
  }
  seg[cap - 1 - atomicAdd(&s.mine.hub, 1u)] = SmallEntry{b, len, v};
  if (len <= kSmallPiece || len > kSmallEdges) return;  // (past the limit: the run ends)
  const uint32_t n = (len - 1) / kSmallPiece, at = atomicAdd(&s.mine.pieces, n);
  for (uint32_t k = 0; k < n && at + k < kSmallPieces; k++)
    seg[cap + at + k] = SmallEntry{b + (k + 1) * kSmallPiece, min(len - (k + 1) * kSmallPiece, kSmallPiece), v};
}

// Up to four edges u -> slots[j], slots[j + step], ... of each lane: the atomics
// and the slot ranges of their ends go out together.
__device__ __forceinline__ void small_visit(SmallShared &s, const SmallArgs &a, SmallEntry *seg, uint64_t j,
                                            uint64_t step, uint64_t e, uint64_t key, unsigned long long &edges, bool &big) {
  uint32_t v[4];
#pragma unroll
  for (int q = 0; q < 4; q++) v[q] = j + q * step < e ? a.slots[j + q * step] : kSentinel;
  unsigned long long old[4];
  uint64_t b[4], end[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    old[q] = 0;
    b[q] = end[q] = 0;
    if (v[q] == kSentinel) continue;
    old[q] = atomicMin((unsigned long long *)(a.lp + v[q]), (unsigned long long)key);
    b[q] = a.off[v[q]];
    end[q] = a.off[v[q] + 1];
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    if (old[q] != kNone64) continue;
    const uint32_t len = (uint32_t)(end[q] - b[q]);
    atomicOr(a.visited + (v[q] >> 5), 1u << (v[q] & 31));
    small_add(s, seg, a.cap, v[q], b[q], len);
    edges += len;
    big |= len >= 1024;
  }
}

__device__ __forceinline__ SmallEntry small_load(const SmallEntry *p) {
  const uint4 x = __ldcg(reinterpret_cast<const uint4 *>(p));
  return SmallEntry{(uint64_t)x.y << 32 | x.x, x.z, x.w};
}

__global__ void __cluster_dims__(kSmallCtas, 1, 1) __launch_bounds__(kSmallBlock, 1) k_bfs_small(SmallArgs a) {
  __shared__ SmallShared s;
  __shared__ unsigned int hist[8];
  const unsigned rank = blockIdx.x;  // one cluster: the CTA's rank
  const unsigned tid = rank * kSmallBlock + threadIdx.x, nthr = kSmallCtas * kSmallBlock;
  if (threadIdx.x == 0) {
    s.arrived = 0;
    s.mine = SmallFound{};
    s.mine_big = 0;
  }
  if (threadIdx.x < 8) hist[threadIdx.x] = 0;
  cluster_hw_sync();  // every CTA's shared memory is ready
  const uint64_t stride = a.cap + kSmallPieces;
  SmallEntry *const segs[2] = {a.seg, a.seg + kSmallCtas * stride};
  unsigned long long edges = 0;
  bool big = false;
  auto flush = [&]() {  // a warp's edge count and hub flag to the CTA's
    __syncwarp();
    if (!__any_sync(kFull, edges != 0)) return;
    // a lane's edges stay below 2^40: two 32-bit sums
    const unsigned lo = __reduce_add_sync(kFull, (unsigned)edges & 0xFFFF);
    const unsigned hi = __reduce_add_sync(kFull, (unsigned)(edges >> 16));
    big = __any_sync(kFull, big);
    if (lane_id() == 0) atomicAdd(&s.mine.edges, ((unsigned long long)hi << 16) + lo);
    if (lane_id() == 0 && big) s.mine_big = 1;
    edges = 0;
    big = false;
  };
  // the first frontier's entries
  for (uint64_t i = tid; i < a.size; i += nthr) {
    const uint32_t v = a.list[i];
    const uint64_t b = a.off[v];
    const uint32_t len = (uint32_t)(a.off[v + 1] - b);
    small_add(s, segs[0] + rank * stride, a.cap, v, b, len);
    edges += len;
    big |= len >= 1024;
  }
  flush();
  unsigned turn = 0;
  bool ok = small_sync(s, a, rank, turn++);
  uint32_t r = 0;
  int cur = 0;
  const unsigned long long first_edges = s.edges;
  bool stop = !ok || !s.edges || a.size + s.edges > a.limit || (a.gate_hub && s.big);
  const bool ran = !stop;
  if (ran)  // the first frontier's bitmap: all its bits belong to its list
    for (uint64_t i = tid; i < a.size; i += nthr) a.bits[a.list[i] >> 5] = 0;
  while (!stop) {
    const SmallEntry *const from = segs[cur];
    SmallEntry *const to = segs[cur ^ 1] + rank * stride;
    const uint32_t F = s.pre[kSmallCtas], H = s.long_pre[2 * kSmallCtas];
    const uint64_t lvl = (uint64_t)(a.round0 + r) << 32;
    // lanes to an entry: enough groups for every entry, at least 4 lanes
    const uint32_t lg = F <= nthr / 32 ? 5 : F <= nthr / 16 ? 4 : F <= nthr / 8 ? 3 : 2, gs = 1u << lg;
    for (uint32_t i = tid >> lg; i < F; i += nthr >> lg) {
      uint32_t c = 0;
#pragma unroll
      for (uint32_t k = 1; k < kSmallCtas; k++) c += i >= s.pre[k];
      const SmallEntry u = small_load(from + c * stride + (i - s.pre[c]));
      for (uint32_t k = tid & (gs - 1); k < u.len; k += 4 * gs)
        small_visit(s, a, to, u.b + k, gs, u.b + u.len, lvl | u.v, edges, big);
    }
    for (uint32_t i = tid >> 5; i < H; i += kSmallWarps) {  // longer entries and pieces, a warp each
      uint32_t c = 0;
      while (i >= s.long_pre[c + 1]) c++;
      const uint32_t at = i - s.long_pre[c];
      const SmallEntry u = small_load(c < kSmallCtas ? from + c * stride + (a.cap - 1 - at)
                                                     : from + (c - kSmallCtas) * stride + (a.cap + at));
      const uint32_t len = min(u.len, kSmallPiece);
      for (uint32_t k = lane_id(); k < len; k += 128)
        small_visit(s, a, to, u.b + k, 32, u.b + len, lvl | u.v, edges, big);
    }
    flush();
    if (tid == 0) a.log[2 * r] = F + s.nhub;
    ok = small_sync(s, a, rank, turn++);
    const uint32_t fn = s.pre[kSmallCtas] + s.nhub;
    if (tid == 0) a.log[2 * r + 1] = s.edges;
    cur ^= 1;
    r++;
    stop = !ok || fn == 0 || (uint64_t)fn + s.edges > a.limit || (a.gate_hub && s.big) || r == kSmallLog;
  }
  // the frontier reached, in the engine's form
  const uint32_t F = s.pre[kSmallCtas], fn = F + s.nhub;
  if (ok) {
    uint32_t hubs_before = 0;
    for (uint32_t c = 0; c < kSmallCtas; c++) {
      const SmallEntry *const seg = segs[cur] + c * stride;
      const uint32_t nsmall = s.pre[c + 1] - s.pre[c], nhub = s.hubs[c];
      for (uint32_t i = tid; i < nsmall + nhub; i += nthr) {
        const SmallEntry u = small_load(i < nsmall ? seg + i : seg + (a.cap - 1 - (i - nsmall)));
        atomicAdd(hist + small_bin(u.len), 1u);
        if (!ran) continue;  // the list and the bitmap it came with
        a.list[i < nsmall ? s.pre[c] + i : F + hubs_before + (i - nsmall)] = u.v;
        atomicOr(a.bits + (u.v >> 5), 1u << (u.v & 31));
      }
      hubs_before += nhub;
    }
  }
  __syncthreads();
  if (threadIdx.x < 8) a.out->hist[rank][threadIdx.x] = hist[threadIdx.x];
  if (threadIdx.x == 0) {
    a.out->err[rank] = ok ? 0 : 1;
    if (rank == 0) {
      a.out->size = fn;
      a.out->edges = s.edges;
      a.out->first_edges = first_edges;
      a.out->rounds = r;
    }
  }
  cluster_hw_sync();  // no CTA leaves while another may still add to its shared memory
}

}  // namespace

int bfs_small_rounds(byo_graph *g, TravState &st, Frontier *&cur, Frontier *&nxt, uint64_t limit, bool gate_hub,
                     RoundStats *d_st, uint32_t *rounds_run) {
  byo_ctx *ctx = g->ctx;
  *rounds_run = 0;
  // SmallOut and the log, read back together up to kFast rounds
  constexpr uint32_t kFast = 96;
  constexpr size_t kHead = (sizeof(SmallOut) + 15) & ~(size_t)15;
  unsigned char *buf = nullptr;
  BYO_TRY(ws(g, WS_BUCKETS, kHead + 16ull * kSmallLog, &buf));
  SmallArgs a;
  a.limit = std::min<uint64_t>(limit, kSmallEdges);
  // a round finds at most as many vertices as its frontier has edges, and no
  // more than there are; the first frontier is dealt out
  a.cap = std::min<uint64_t>(std::max<uint64_t>(a.limit, cur->size), g->n) + 1;
  BYO_TRY(ws(g, WS_DEFER, 2 * kSmallCtas * (a.cap + kSmallPieces) * sizeof(SmallEntry) / 4, (uint32_t **)&a.seg));
  a.off = g->d_off;
  a.slots = g->d_slots;
  a.lp = st.lp;
  a.visited = st.visited;
  a.list = cur->list;
  a.bits = cur->bits;
  a.size = cur->size;
  a.round0 = st.round;
  a.gate_hub = gate_hub ? 1 : 0;
  a.limit_ms = ctx->bar_limit_ms;
  a.extra = ctx->bar_extra;
  a.out = reinterpret_cast<SmallOut *>(buf);
  a.log = reinterpret_cast<unsigned long long *>(buf + kHead);
  launch(ctx, k_bfs_small, dim3(kSmallCtas), dim3(kSmallBlock), 0, a);
  BYO_TRY(check_launch(ctx, "bfs_small"));
  unsigned char *hbuf = nullptr;
  BYO_TRY(pinned(ctx, 4096, (void **)&hbuf));
  static_assert(kHead + 16 * kFast <= 4096, "the head and the fast log fit the pinned page");
  BYO_CU(ctx, cudaMemcpyAsync(hbuf, buf, kHead + 16 * kFast, cudaMemcpyDeviceToHost, ctx->stream));
  BYO_CU(ctx, cudaStreamSynchronize(ctx->stream));
  SmallOut h;
  std::memcpy(&h, hbuf, sizeof(h));
  for (uint32_t c = 0; c < kSmallCtas; c++)
    if (h.err[c]) return set_error(ctx, BYO_ETIMEDOUT, "bfs: cluster barrier timed out");
  const uint32_t R = h.rounds;
  std::vector<unsigned long long> lg(2ull * R);
  std::memcpy(lg.data(), hbuf + kHead, 16ull * std::min(R, kFast));
  if (R > kFast) {
    BYO_CU(ctx, cudaMemcpyAsync(lg.data() + 2 * kFast, a.log + 2 * kFast, 16ull * (R - kFast), cudaMemcpyDeviceToHost,
                                ctx->stream));
    BYO_CU(ctx, cudaStreamSynchronize(ctx->stream));
  }
  uint64_t reached = 0;
  for (uint32_t r = 0; r < R; r++) {
    byo_round_log e{};
    e.round = st.round + r;
    e.mode = MODE_PUSH;
    e.frontier = lg[2 * r];
    e.frontier_deg = r == 0 ? h.first_edges : lg[2 * (r - 1) + 1];
    e.unvisited = 0;
    ctx->rounds.push_back(e);
    reached += r + 1 < R ? lg[2 * (r + 1)] : h.size;
  }
  cur->size = h.size;
  cur->outdeg = h.edges;
  for (int q = 0; q < 8; q++) {
    cur->hist[q] = 0;
    for (uint32_t c = 0; c < kSmallCtas; c++) cur->hist[q] += h.hist[c][q];
  }
  cur->dense = false;
  cur->has_list = cur->has_bits = true;
  nxt->size = 0;
  st.reached += reached;
  st.round += R;
  if (d_st) {
    // the statistics the policy reads for the round after (a pageable source:
    // the copy has consumed it when the call returns)
    RoundStats rs{};
    rs.count = cur->size;
    rs.outdeg = cur->outdeg;
    for (int q = 0; q < 8; q++) rs.hist[q] = cur->hist[q];
    BYO_CU(ctx, cudaMemcpyAsync(d_st, &rs, sizeof(RoundStats), cudaMemcpyHostToDevice, ctx->stream));
  }
  *rounds_run = R;
  return BYO_OK;
}

}  // namespace byo
