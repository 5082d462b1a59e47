// edgemap.cu -- edgeMap over the device functors other than BFS_F, and
// vertexMap / vertexFilter.
//
// The reference's edgeMap (gbbs/edge_map_data.h:254-315) takes any struct
// with update / updateAtomic / cond; a GPU kernel cannot call a host lambda,
// so the functors are a closed set of device structs, each mirroring one
// GBBS functor:
//   LabelF    BFS_ComponentLabel_F (benchmarks/Connectivity/BFSCC/Connectivity.h:31-50)
//   PrF       PR_F                 (benchmarks/PageRank/PageRank.h:33-50)
//   PrDeltaF  delta::PR_Delta_F    (benchmarks/PageRank/PageRank.h:200-226)
// BFS_F keeps the traversal engine of engine.cu.
//
// Rounds:
//   sparse (edgeMapSparse, gbbs/edge_map_blocked.h:18-92) and blocked: a warp
//     per frontier vertex walks its neighbour run with coalesced loads and
//     applies cond + updateAtomic; a vertex enters the output once (its bit is
//     claimed by atomicOr, the winner appends it by warp ballot).
//   dense (edgeMapDense, gbbs/edge_map_data.h:47-175): every vertex whose
//     cond holds scans its neighbours in order and applies update (one writer
//     per vertex) to those in the frontier, leaving at the first !cond.  A
//     lane takes a vertex of <= kDenseShort slots; longer runs go to a warp
//     that loads and tests 32 neighbours at a time and applies the updates in
//     order.  PR_F and PR_Delta_F have kernels of their own, whose sums are
//     bit-identical to a sequential scan: a round on its own a lane, a warp or a CTA
//     a vertex (k_em_sum_direct, k_em_sum_warps, k_em_sum_ctas), rounds of one
//     plan lanes by class (k_em_sum_lanes).
//   dense forward (edgeMapDenseForward, gbbs/edge_map_data.h:180-247): the
//     frontier's members push with updateAtomic, as the sparse round does.
// The output is a list and a bitmap kept together (the engine's Frontier).
//
// Arithmetic that feeds parity with the FP64 oracle uses explicitly rounded
// operations (__dadd_rn, __dmul_rn, __ddiv_rn): no fused multiply-add, so
// every result equals the oracle's separately rounded C expression.
#include "device.cuh"
#include "engine.h"
#include "internal.h"
#include "seqsum.cuh"

namespace byo {

namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kDenseShort = 64;  // slots a lane scans alone in a dense round

struct LabelF {
  uint32_t *P;
  uint32_t src;
  __device__ bool cond(uint32_t d) const { return *(volatile uint32_t *)(P + d) == kNone; }
  __device__ bool update(uint32_t, uint32_t d) const {
    if (P[d] != src) {
      P[d] = src;
      return true;
    }
    return false;
  }
  __device__ bool updateAtomic(uint32_t, uint32_t d) const { return atomicCAS(P + d, kNone, src) == kNone; }
};

struct PrF {
  const double *pc;
  double *pn;
  const uint32_t *deg;
  __device__ double value(uint32_t s) const { return __ddiv_rn(pc[s], (double)deg[s]); }
  __device__ bool cond(uint32_t) const { return true; }
  __device__ bool update(uint32_t s, uint32_t d) const {
    pn[d] = __dadd_rn(pn[d], value(s));
    return true;
  }
  __device__ bool updateAtomic(uint32_t s, uint32_t d) const {
    atomicAdd(pn + d, value(s));
    return true;
  }
};

struct PrDeltaF {
  const double *delta;  // [2n]: delta, delta / degree
  double *ngh;
  __device__ double value(uint32_t s) const { return delta[2 * (uint64_t)s + 1]; }
  __device__ bool cond(uint32_t) const { return true; }
  __device__ bool update(uint32_t s, uint32_t d) const {
    const double old = ngh[d];
    ngh[d] = __dadd_rn(old, value(s));
    return old == 0.0;
  }
  __device__ bool updateAtomic(uint32_t s, uint32_t d) const {
    unsigned long long *a = reinterpret_cast<unsigned long long *>(ngh + d);
    const double x = value(s);
    unsigned long long old = *(volatile unsigned long long *)a, seen;
    do {
      seen = old;
      old = atomicCAS(a, seen, __double_as_longlong(__dadd_rn(__longlong_as_double(seen), x)));
    } while (old != seen);
    return __longlong_as_double(seen) == 0.0;
  }
};

// Output of a round: the bit of v claimed once, the winner appends v.
__device__ __forceinline__ void emit_out(bool want, uint32_t v, uint32_t *out_list, uint32_t *out_bits,
                                         const uint32_t *deg, unsigned long long *cnt, uint64_t &outdeg) {
  bool emit = false;
  if (want) {
    const uint32_t bit = 1u << (v & 31);
    emit = !(atomicOr(out_bits + (v >> 5), bit) & bit);
  }
  const uint64_t slot = warp_append(emit, cnt);
  if (emit) {
    out_list[slot] = v;
    outdeg += deg[v];
  }
}

template <class F>
__global__ void __launch_bounds__(256) k_em_push(const uint64_t *__restrict__ off, const uint32_t *__restrict__ slots,
                                                 const uint32_t *__restrict__ deg, F f,
                                                 const uint32_t *__restrict__ list, uint64_t size, int output,
                                                 uint32_t *out_list, uint32_t *out_bits, unsigned long long *cnt) {
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint64_t outdeg = 0;
  for (uint64_t i = gw; i < size; i += nw) {
    const uint32_t u = list[i];
    const uint64_t b = off[u], e = off[u + 1];
    for (uint64_t base = b; base < e; base += 32) {
      const uint64_t j = base + lane_id();
      bool hit = false;
      uint32_t v = 0;
      if (j < e) {
        v = slots[j];
        if (v != kSentinel && f.cond(v)) hit = f.updateAtomic(u, v);
      }
      emit_out(hit && output, v, out_list, out_bits, deg, cnt, outdeg);
    }
  }
  outdeg = warp_sum(outdeg);
  if (lane_id() == 0 && outdeg) atomicAdd(cnt + 1, (unsigned long long)outdeg);
}

template <class F>
__global__ void __launch_bounds__(256) k_em_pull(const uint64_t *__restrict__ off, const uint32_t *__restrict__ slots,
                                                 const uint32_t *__restrict__ deg, F f, const uint32_t *__restrict__ fb,
                                                 uint64_t n, int output, uint32_t *out_list, uint32_t *out_bits,
                                                 unsigned long long *cnt, uint32_t *defer) {
  const uint64_t W = (n + 31) / 32;
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint64_t outdeg = 0;
  for (uint64_t w = gw; w < W; w += nw) {
    const uint64_t v = w * 32 + lane_id();
    bool marked = false, lng = false;
    if (v < n) {
      const uint64_t b = off[v], e = off[v + 1];
      if (e - b > kDenseShort) {
        lng = true;
      } else if (f.cond((uint32_t)v)) {
        for (uint64_t j = b; j < e; j++) {
          const uint32_t u = slots[j];
          if (u == kSentinel) continue;
          if (test_bit(fb, u) && f.update(u, (uint32_t)v)) marked = true;
          if (!f.cond((uint32_t)v)) break;
        }
      }
    }
    const uint64_t slot = warp_append(lng, cnt + 2);
    if (lng) defer[slot] = (uint32_t)v;
    marked = marked && output;
    const unsigned m = __ballot_sync(kFull, marked);
    if (lane_id() == 0 && m) atomicOr(out_bits + w, m);
    const uint64_t s2 = warp_append(marked, cnt);
    if (marked) {
      out_list[s2] = (uint32_t)v;
      outdeg += deg[v];
    }
  }
  outdeg = warp_sum(outdeg);
  if (lane_id() == 0 && outdeg) atomicAdd(cnt + 1, (unsigned long long)outdeg);
}

// A long run in order, a warp at a time: returns whether any update marked v
// (warp-uniform).  Generic form: lane 0 applies the updates one by one.
template <class F>
__device__ __forceinline__ bool warp_pull_run(const F &f, uint32_t v, const uint32_t *slots, uint64_t b, uint64_t e,
                                              const uint32_t *fb) {
  bool marked = false;
  for (uint64_t base = b; base < e; base += 32) {
    const uint64_t j = base + lane_id();
    const uint32_t u = j < e ? slots[j] : kSentinel;
    unsigned in = __ballot_sync(kFull, u != kSentinel && test_bit(fb, u));
    bool stop = false;
    while (in && !stop) {
      const int k = __ffs(in) - 1;
      in &= in - 1;
      const uint32_t uk = __shfl_sync(kFull, u, k);
      int r = 0, c = 1;
      if (lane_id() == 0) {
        r = f.update(uk, v) ? 1 : 0;
        c = f.cond(v) ? 1 : 0;
      }
      r = __shfl_sync(kFull, r, 0);
      c = __shfl_sync(kFull, c, 0);
      marked |= r != 0;
      stop = !c;
    }
    if (stop) break;
  }
  return marked;
}

template <class F>
__global__ void __launch_bounds__(256) k_em_pull_long(const uint64_t *__restrict__ off,
                                                      const uint32_t *__restrict__ slots,
                                                      const uint32_t *__restrict__ deg, F f,
                                                      const uint32_t *__restrict__ fb, int output,
                                                      uint32_t *out_list, uint32_t *out_bits, unsigned long long *cnt,
                                                      const uint32_t *__restrict__ defer) {
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t nd = cnt[2];
  uint64_t outdeg = 0;
  for (uint64_t i = gw; i < nd; i += nw) {
    const uint32_t v = defer[i];
    bool marked = false;
    if (__shfl_sync(kFull, f.cond(v) ? 1 : 0, 0)) marked = warp_pull_run(f, v, slots, off[v], off[v + 1], fb);
    const bool want = lane_id() == 0 && marked && output;
    emit_out(want, v, out_list, out_bits, deg, cnt, outdeg);
  }
  outdeg = warp_sum(outdeg);
  if (lane_id() == 0 && outdeg) atomicAdd(cnt + 1, (unsigned long long)outdeg);
}

// ---------------------------------------------------------------- dense rounds of the sums
// Runs in classes of similar length, each a list of vertices: a lane takes a
// run of the first ones, a warp one of the next to last and a CTA one of the
// last.  A warp's FP64 addition takes the pipe 19 cycles however many lanes
// add, so 32 runs of one length cost a warp what a single one would.
constexpr uint32_t kSumLaneMax = 128, kSumWarpMax = 4096;
constexpr int kSumLanes = 11, kSumWarp = kSumLanes, kSumCta = kSumLanes + 1, kSumClasses = kSumLanes + 2;
__device__ __forceinline__ int sum_class(uint64_t len) {  // 1..2, 3..4, ..8, ..12, ..16, 24, 32, .. kSumLaneMax
  if (len <= 8) return len <= 2 ? 0 : len <= 4 ? 1 : 2;
  if (len > kSumLaneMax) return len <= kSumWarpMax ? kSumWarp : kSumCta;
  const int lg = 31 - __clz((int)len - 1);  // 8 < len: len - 1 in [2^lg, 2^(lg+1))
  return 3 + 2 * (lg - 3) + (int)(((len - 1) >> (lg - 1)) & 1);
}
struct SumPlan {
  uint32_t *list;             // the classes' vertices, one class after the other
  unsigned long long *count;  // [kSumClasses] vertices, [kSumClasses] cursors, [1] next warp run
  // of a round on its own: the warps' runs only, and the CTAs' from the end of n
  bool direct;
  __device__ const uint32_t *runs(int c, uint64_t n) const {
    if (direct) return c == kSumCta ? list + (n - count[c]) : list;
    uint64_t start = 0;
    for (int k = 0; k < c; k++) start += count[k];
    return list + start;
  }
};
constexpr int kSumCounts = 2 * kSumClasses + 1;

// What one neighbour adds: a value computed once per vertex (PR_F: n divisions
// instead of one an edge; FP64 division is slow here), or read in place, or
// (kDivide, small views) divided there.
struct SumArgs {
  const uint64_t *off;
  const uint32_t *slots;
  const uint32_t *deg;
  const uint32_t *fb;    // the frontier; null: every vertex
  const double *val;     // value of vertex u at val[u * stride + at]
  uint32_t stride, at;
  uint64_t n;
  double *sum;
  int zero_marks, output;
  uint32_t *out_list, *out_bits;
  unsigned long long *cnt;  // members out, their degrees
  SumPlan plan;
  template <bool kDivide = false>
  __device__ double value(uint32_t u) const {
    const double x = __ldg(val + (uint64_t)u * stride + at);
    return kDivide ? __ddiv_rn(x, (double)deg[u]) : x;
  }
  __device__ bool member(uint32_t u) const { return u != kSentinel && (!fb || test_bit(fb, u)); }
};

// kPlace = false counts the classes, true writes the lists: a CTA counts its
// 4096 vertices in shared memory and takes a place in each list at once.
template <bool kPlace>
__global__ void __launch_bounds__(1024) k_sum_plan(const uint64_t *__restrict__ off, uint64_t n, SumPlan p) {
  __shared__ unsigned int cnt[kSumClasses];
  __shared__ unsigned long long at[kSumClasses];
  for (uint64_t base = blockIdx.x * 4096ull; base < n; base += gridDim.x * 4096ull) {
    if (threadIdx.x < kSumClasses) cnt[threadIdx.x] = 0;
    __syncthreads();
    int c[4];
    unsigned int slot[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const uint64_t v = base + q * 1024 + threadIdx.x;
      const uint64_t len = v < n ? off[v + 1] - off[v] : 0;
      c[q] = len ? sum_class(len) : -1;
      const unsigned peers = __match_any_sync(kFull, c[q]);
      const int leader = __ffs(peers) - 1;
      unsigned int b = 0;
      if (c[q] >= 0 && (int)lane_id() == leader) b = atomicAdd(cnt + c[q], (unsigned)__popc(peers));
      slot[q] = __shfl_sync(kFull, b, leader) + __popc(peers & lanemask_lt());
    }
    __syncthreads();
    if (threadIdx.x < kSumClasses && cnt[threadIdx.x]) {
      unsigned long long start = 0;
      if (kPlace)
        for (int k = 0; k < (int)threadIdx.x; k++) start += p.count[k];
      at[threadIdx.x] = start + atomicAdd(p.count + (kPlace ? kSumClasses : 0) + threadIdx.x,
                                          (unsigned long long)cnt[threadIdx.x]);
    }
    __syncthreads();
    if (kPlace) {
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (c[q] >= 0) p.list[at[c[q]] + slot[q]] = (uint32_t)(base + q * 1024 + threadIdx.x);
    }
    __syncthreads();
  }
}

__global__ void k_em_values(PrF f, uint64_t n, double *val) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
    val[v] = f.value((uint32_t)v);
}

// A lane per run: 32 runs of one class, kWin terms of each at a time gathered
// by the whole warp (the runs' ids in pieces of kWin) and staged, then added
// by the runs' lanes.  Bound by a warp's own chain (64 cycles an FP64 addition,
// two gathers a window), so longer runs than kSumLaneMax are composed by a warp
// instead: with lanes up to 512 slots, one warp's 32 windows took 285 us.
// Chung-Lu n = 10^6, 16 M edges: 90 us a round; a lane that walked its own run
// of up to 64 slots with a division for every term took 270.
template <int kWin, bool kMarks>
__device__ __forceinline__ void sum_lane_runs(const SumArgs &a, const uint32_t *list, uint64_t runs, uint64_t group,
                                              double *stage, uint64_t &outdeg) {
  const unsigned lane = lane_id();
  const uint64_t i = group * 32 + lane;
  uint32_t v = 0;
  uint64_t b = 0;
  uint32_t len = 0;
  if (i < runs) {
    v = list[i];
    b = a.off[v];
    len = (uint32_t)(a.off[v + 1] - b);
  }
  double acc = len ? a.sum[v] : 0.0;
  bool any = false, zero = false;
  for (uint32_t w0 = 0; __ballot_sync(kFull, w0 < len); w0 += kWin) {
    uint32_t u[kWin];
#pragma unroll
    for (int q = 0; q < kWin; q++) {  // position q * 32 + lane: run / kWin, term % kWin
      const int run = q * (32 / kWin) + lane / kWin;
      const uint32_t k = w0 + lane % kWin;
      const uint64_t rb = __shfl_sync(kFull, b, run);
      const uint32_t rl = __shfl_sync(kFull, len, run);
      u[q] = k < rl ? a.slots[rb + k] : kSentinel;
    }
    uint32_t has = 0;
#pragma unroll
    for (int q = 0; q < kWin; q++) {
      const bool in = kMarks ? a.member(u[q]) : u[q] != kSentinel;
      if (in) stage[(q * (32 / kWin) + lane / kWin) * (kWin + 1) + lane % kWin] = a.value(u[q]);
      const unsigned m = __ballot_sync(kFull, in);
      if ((int)(lane / (32 / kWin)) == q) has = m >> (lane % (32 / kWin) * kWin);
    }
    __syncwarp();
    has &= (1u << kWin) - 1u;
    any |= has != 0;
#pragma unroll
    for (int k = 0; k < kWin; k++)
      if ((has >> k) & 1u) {
        if (kMarks) zero |= seq_zero(acc);
        acc = __dadd_rn(acc, stage[lane * (kWin + 1) + k]);
      }
    __syncwarp();
  }
  if (any) a.sum[v] = acc;
  if (kMarks) emit_out(a.output && (a.zero_marks ? zero : any), v, a.out_list, a.out_bits, a.deg, a.cnt, outdeg);
}

// kMarks: a frontier, or members out (not in PageRank's rounds).
template <bool kMarks>
__global__ void __launch_bounds__(256) k_em_sum_lanes(SumArgs a) {
  __shared__ double stage[8][32 * 17];
  __shared__ uint64_t first[kSumLanes + 1], vert[kSumLanes + 1];  // groups and vertices before each class
  if (threadIdx.x == 0) {
    uint64_t g = 0, v = 0;
    for (int c = 0; c < kSumLanes; c++) {
      first[c] = g;
      vert[c] = v;
      g += (a.plan.count[c] + 31) / 32;
      v += a.plan.count[c];
    }
    first[kSumLanes] = g;
    vert[kSumLanes] = v;
  }
  __syncthreads();
  // neighbouring groups, which are of one length, on different SMs
  const uint64_t gw = (uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  double *st = stage[threadIdx.x >> 5];
  uint64_t outdeg = 0;
  int c = kSumLanes - 1;  // the longest runs first
  for (uint64_t t = gw; t < first[kSumLanes]; t += nw) {
    const uint64_t g = first[kSumLanes] - 1 - t;
    while (g < first[c]) c--;
    const uint32_t *list = a.plan.list + vert[c];
    const uint64_t runs = vert[c + 1] - vert[c];
    if (c <= 1)
      sum_lane_runs<4, kMarks>(a, list, runs, g - first[c], st, outdeg);
    else if (c == 2)
      sum_lane_runs<8, kMarks>(a, list, runs, g - first[c], st, outdeg);
    else
      sum_lane_runs<16, kMarks>(a, list, runs, g - first[c], st, outdeg);
  }
  if (!kMarks) return;
  outdeg = warp_sum(outdeg);
  if (lane_id() == 0 && outdeg) atomicAdd(a.cnt + 1, (unsigned long long)outdeg);
}

// One run by a warp, 256 neighbours a step; stage: seq_at<8>(256) values, mask: 8 words.
template <bool kDivide>
__device__ __forceinline__ SeqSum sum_warp_run(const SumArgs &a, uint32_t v, uint64_t b, uint64_t e, double *stage,
                                               uint32_t *mask) {
  const unsigned lane = lane_id();
  SeqSum s{a.sum[v], false, false};
  for (uint64_t j0 = b; j0 < e; j0 += 256) {
    uint32_t u[8];
#pragma unroll
    for (int r = 0; r < 8; r++) u[r] = j0 + r * 32 + lane < e ? a.slots[j0 + r * 32 + lane] : kSentinel;
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const bool has = a.member(u[r]);
      const unsigned word = __ballot_sync(kFull, has);
      stage[seq_at<8>(r * 32 + lane)] = has ? a.value<kDivide>(u[r]) : 0.0;
      if (lane == 0) mask[r] = word;
    }
    __syncwarp();
    double x[8];
#pragma unroll
    for (int r = 0; r < 8; r++) x[r] = stage[seq_at<8>(8 * lane + r)];
    seq_warp(s, x, reinterpret_cast<const unsigned char *>(mask)[lane]);
    __syncwarp();
  }
  if (lane == 0 && s.any) a.sum[v] = s.acc;
  return s;
}

// The listed runs of the warps, each warp the next one.
template <bool kDivide>
__device__ __forceinline__ void sum_warp_runs(const SumArgs &a, double *stage, uint32_t *mask) {
  const unsigned lane = lane_id();
  const uint32_t *runs = a.plan.runs(kSumWarp, a.n);
  const uint64_t nwarp = a.plan.count[kSumWarp];
  if (!nwarp) return;
  uint64_t outdeg = 0;
  for (;;) {
    unsigned long long i = 0;
    if (lane == 0) i = atomicAdd(a.plan.count + 2 * kSumClasses, 1ull);
    i = __shfl_sync(kFull, i, 0);
    if (i >= nwarp) break;
    const uint32_t v = runs[i];
    const SeqSum s = sum_warp_run<kDivide>(a, v, a.off[v], a.off[v + 1], stage, mask);
    emit_out(lane == 0 && a.output && (a.zero_marks ? s.zero : s.any), v, a.out_list, a.out_bits, a.deg, a.cnt, outdeg);
  }
  outdeg = warp_sum(outdeg);
  if (lane == 0 && outdeg) atomicAdd(a.cnt + 1, (unsigned long long)outdeg);
}

// A round on its own: planning it costs two passes and the launches of three
// streams, 12 us of a 40 us call on small graphs, and on uniform graphs there is
// little to tell apart (10^6 vertices of degree 16: 325 us a call by a plan, 290 so).
// A lane per vertex of up to kSumShort neighbours, kBatch of its slots in flight; the
// longer runs are listed for the other kernel.  At 32 neighbours instead of 64:
// uniform 10^6 vertices of degree 24 / 32 / 48 330 / 371 / 451 -> 356 / 757 / 1229 us, Chung-Lu
// and RMAT graphs as fast.
// On a view with gaps (kGaps) so few neighbours may lie in a run of any length: a
// lane takes it up to twice as many slots (a vector of runs has no more), its warp
// at once up to kGapRun (a leaf's gap).
constexpr uint32_t kSumShort = 64, kGapRun = 512;
enum { kRunLane, kRunGap, kRunWarp, kRunCta };
template <bool kGaps>
__device__ __forceinline__ int sum_run(const SumArgs &a, uint64_t v, uint64_t len) {
  if (len <= kSumShort) return kRunLane;
  if (kGaps && len <= kGapRun && a.deg[v] <= kSumShort) return len <= 2 * kSumShort ? kRunLane : kRunGap;
  return len <= kSumWarpMax ? kRunWarp : kRunCta;
}

// Whether a round on its own is better planned, from 128 groups of 32 vertices: their
// lanes' runs so unlike that most lanes would wait (the longest of 32 against their
// mean: uniform graphs up to 2.7, Chung-Lu 2.2, for the hubs come first, RMAT 3.1 to
// 6.1), or many too long for a lane (uniform from an average degree of about 56).
constexpr int kSumProbes = 4;  // groups a warp
template <bool kGaps>
__global__ void __launch_bounds__(1024) k_sum_probe(SumArgs a, unsigned long long *plan) {
  __shared__ unsigned int s_sum, s_max, s_long;
  if (threadIdx.x == 0) s_sum = s_max = s_long = 0;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kSumProbes; q++) {
    const uint32_t i = q * 32 + (threadIdx.x >> 5);
    const uint64_t v = (((uint64_t)(i * 0x9E3779B1u) * ((a.n + 31) >> 5)) >> 32) * 32 + lane_id();
    const uint64_t len = v < a.n ? a.off[v + 1] - a.off[v] : 0;
    const uint32_t x = v < a.n ? min(kGaps ? a.deg[v] : (uint32_t)min(len, (uint64_t)kSumShort), kSumShort) : 0;
    const uint32_t sum = __reduce_add_sync(kFull, x), top = __reduce_max_sync(kFull, x);
    const uint32_t lng = __popc(__ballot_sync(kFull, len && sum_run<kGaps>(a, v, len) >= kRunWarp));
    if (lane_id() == 0) {
      atomicAdd(&s_sum, sum);
      atomicAdd(&s_max, top);
      atomicAdd(&s_long, lng);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) *plan = 32 * s_max > 3 * s_sum || 8 * s_long > 32 * kSumProbes * 32;
}

template <bool kDivide, bool kGaps, int kBatch>
__global__ void __launch_bounds__(256, kDivide || kGaps ? 4 : 5) k_em_sum_direct(SumArgs a) {
  __shared__ double stages[kGaps ? 8 : 1][kGaps ? seq_at<8>(256) : 1];
  __shared__ uint32_t masks[8][8];
  const uint64_t W = (a.n + 31) / 32;
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint64_t outdeg = 0;
  for (uint64_t w = gw; w < W; w += nw) {
    const uint64_t v = w * 32 + lane_id();
    const uint64_t b = v < a.n ? a.off[v] : 0, len = v < a.n ? a.off[v + 1] - b : 0;
    bool any = false, zero = false;
    const int run = sum_run<kGaps>(a, v, len);
    if (len && run == kRunLane) {
      const uint32_t *const ids = a.slots + b;
      double acc = 0.0;
      for (uint32_t j = 0; j < len; j += kBatch) {
        uint32_t u[kBatch];
        double x[kBatch];
        unsigned in = 0;
#pragma unroll
        for (int q = 0; q < kBatch; q++) u[q] = j + q < len ? ids[j + q] : kSentinel;
#pragma unroll
        for (int q = 0; q < kBatch; q++) in |= a.member(u[q]) ? 1u << q : 0u;
        if (!in) continue;
#pragma unroll
        for (int q = 0; q < kBatch; q++) x[q] = (in >> q) & 1u ? a.value<kDivide>(u[q]) : 0.0;
        if (!any) acc = a.sum[v];
        any = true;
#pragma unroll
        for (int q = 0; q < kBatch; q++)
          if ((in >> q) & 1u) {
            zero |= seq_zero(acc);
            acc = __dadd_rn(acc, x[q]);
          }
      }
      if (any) a.sum[v] = acc;
    }
    if constexpr (kGaps) {
      for (unsigned m = __ballot_sync(kFull, run == kRunGap); m; m &= m - 1) {
        const int k = __ffs(m) - 1;
        const uint64_t from = __shfl_sync(kFull, b, k);
        const SeqSum s = sum_warp_run<kDivide>(a, (uint32_t)(w * 32 + k), from, from + __shfl_sync(kFull, len, k),
                                               stages[threadIdx.x >> 5], masks[threadIdx.x >> 5]);
        if ((int)lane_id() == k) {
          any = s.any;
          zero = s.zero;
        }
      }
    }
    const uint64_t at = warp_append(run == kRunWarp, a.plan.count + kSumWarp);
    if (run == kRunWarp) a.plan.list[at] = (uint32_t)v;
    const uint64_t back = warp_append(run == kRunCta, a.plan.count + kSumCta);
    if (run == kRunCta) a.plan.list[a.n - 1 - back] = (uint32_t)v;
    emit_out(a.output && (a.zero_marks ? zero : any), (uint32_t)v, a.out_list, a.out_bits, a.deg, a.cnt, outdeg);
  }
  outdeg = warp_sum(outdeg);
  if (lane_id() == 0 && outdeg) atomicAdd(a.cnt + 1, (unsigned long long)outdeg);
}

// Runs above 4096 slots, a CTA each (seqsum.cuh), 4096 neighbours a step: bound by
// the largest hub's steps (1.4 us each).  Chung-Lu n = 10^6, whose hub has 500 K
// neighbours: 172 us a round; one lane adding a warp's values in turn took 20 ms.
// 64 registers instead of 128 spill the loads in flight: 364 us.  kRest: then the
// warps' runs too, on views where the launch saved is more than what fewer warps
// an SM (128 registers) cost: uniform 10^5 vertices of degree 8 50 -> 46 us a call, RMAT
// 2^18 235 -> 212.
constexpr int kSumBlock = 512, kSumTerms = 8;
template <bool kDivide, bool kRest>
__global__ void __launch_bounds__(kSumBlock, 1) k_em_sum_ctas(SumArgs a) {
  __shared__ double stage[seq_at<kSumTerms>(kSumTerms * kSumBlock)];
  __shared__ uint32_t mask[kSumTerms * kSumBlock / 32];
  __shared__ uint64_t sums[2][32];
  __shared__ SeqSum shared;
  const SeqBlockMem mem{stage, mask, sums, &shared};
  const uint32_t *runs = a.plan.runs(kSumCta, a.n);
  const uint64_t ncta = a.plan.count[kSumCta];
  uint64_t outdeg = 0;
  unsigned turn = 0;
  for (uint64_t i = blockIdx.x; i < ncta; i += gridDim.x) {
    const uint32_t v = runs[i];
    const uint64_t b = a.off[v], e = a.off[v + 1];
    SeqSum s{a.sum[v], false, false};
    // the values of the next step and the ids of the one after it load while
    // a step is added
    uint32_t u[kSumTerms];
    double x[kSumTerms];
    unsigned in = 0;
    auto ids = [&](uint64_t j0) {
#pragma unroll
      for (int r = 0; r < kSumTerms; r++) {
        const uint64_t j = j0 + r * kSumBlock + threadIdx.x;
        u[r] = j < e ? a.slots[j] : kSentinel;
      }
    };
    auto values = [&]() {
      in = 0;
#pragma unroll
      for (int r = 0; r < kSumTerms; r++) {
        const bool has = a.member(u[r]);
        in |= (has ? 1u : 0u) << r;
        x[r] = has ? a.value<kDivide>(u[r]) : 0.0;
      }
    };
    constexpr uint64_t kStep = kSumTerms * kSumBlock;
    ids(b);
    values();
    ids(b + kStep);
    for (uint64_t j = b; j < e; j += kStep) {
      double y[kSumTerms];
#pragma unroll
      for (int r = 0; r < kSumTerms; r++) y[r] = x[r];
      const unsigned had = in;
      values();
      ids(j + 2 * kStep);
      seq_block(s, y, had, mem, turn++);
    }
    if (threadIdx.x < 32) {
      if (threadIdx.x == 0 && s.any) a.sum[v] = s.acc;
      emit_out(threadIdx.x == 0 && a.output && (a.zero_marks ? s.zero : s.any), v, a.out_list, a.out_bits, a.deg,
               a.cnt, outdeg);
    }
  }
  if (threadIdx.x == 0 && outdeg) atomicAdd(a.cnt + 1, (unsigned long long)outdeg);
  if constexpr (kRest) {
    constexpr int kPart = seq_at<8>(256);
    static_assert(kPart * kSumBlock / 32 == seq_at<kSumTerms>(kSumTerms * kSumBlock), "a warp's part of the stage");
    __syncthreads();
    sum_warp_runs<kDivide>(a, stage + (threadIdx.x >> 5) * kPart, mask + (threadIdx.x >> 5) * 8);
  }
}

// Runs of kSumLaneMax to 4096 slots, a warp each: 108 us a round on the same graph
// (with the lanes' and the CTAs' runs side by side).
template <bool kDivide>
__global__ void __launch_bounds__(256) k_em_sum_warps(SumArgs a) {
  __shared__ double stages[8][seq_at<8>(256)];
  __shared__ uint32_t masks[8][8];
  sum_warp_runs<kDivide>(a, stages[threadIdx.x >> 5], masks[threadIdx.x >> 5]);
}

// ---------------------------------------------------------------- frontier forms

__global__ void k_bits_to_list(const uint32_t *__restrict__ bits, uint64_t n, const uint32_t *__restrict__ deg,
                               uint32_t *list, unsigned long long *cnt) {
  const uint64_t W = (n + 31) / 32;
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint64_t outdeg = 0;
  for (uint64_t w = gw; w < W; w += nw) {
    const uint64_t v = w * 32 + lane_id();
    const bool in = v < n && ((bits[w] >> lane_id()) & 1u);
    const uint64_t slot = warp_append(in, cnt);
    if (in) {
      list[slot] = (uint32_t)v;
      outdeg += deg[v];
    }
  }
  outdeg = warp_sum(outdeg);
  if (lane_id() == 0 && outdeg) atomicAdd(cnt + 1, (unsigned long long)outdeg);
}

// bits[w] = src[w] (or all ones) with the bits of ids >= n cleared
__global__ void k_bits_copy(const uint32_t *__restrict__ src, uint64_t n, uint32_t *bits) {
  const uint64_t W = (n + 31) / 32;
  for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < W; w += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t x = src ? src[w] : 0xFFFFFFFFu;
    if (w == W - 1 && (n & 31)) x &= (1u << (n & 31)) - 1u;
    bits[w] = x;
  }
}

// ---------------------------------------------------------------- vertex functions

struct VOp {
  int kind;
  double *a, *b, *c;
  double damping, eps2, added, one_over_n;
  const uint32_t *deg;
};

// PR_Vertex_F (PageRank.h:53-68), PR_Vertex_Reset (:71-78),
// delta::PR_Vertex_F_FirstRound (:252-281), delta::PR_Vertex_F (:294-318)
__device__ __forceinline__ bool vop_apply(const VOp &o, uint32_t i) {
  switch (o.kind) {
    case BYO_VOP_PR_UPDATE:
      o.a[i] = __dadd_rn(__dmul_rn(o.damping, o.a[i]), o.added);
      return true;
    case BYO_VOP_ZERO:
      o.a[i] = 0.0;
      return true;
    case BYO_VOP_PR_DELTA_FIRST: {
      const double pre = __dadd_rn(__dmul_rn(o.damping, o.c[i]), o.added);
      const double p = __dadd_rn(o.a[i], pre);
      o.a[i] = p;
      const double nd = __dsub_rn(pre, o.one_over_n);
      o.b[2 * (uint64_t)i] = nd;
      o.b[2 * (uint64_t)i + 1] = __ddiv_rn(nd, (double)o.deg[i]);
      return nd > __dmul_rn(o.eps2, p);
    }
    case BYO_VOP_PR_DELTA: {
      const double nd = __dmul_rn(o.c[i], o.damping);
      o.b[2 * (uint64_t)i] = nd;
      o.b[2 * (uint64_t)i + 1] = __ddiv_rn(nd, (double)o.deg[i]);
      if (fabs(nd) > __dmul_rn(o.eps2, o.a[i])) {
        o.a[i] = __dadd_rn(o.a[i], nd);
        return true;
      }
      return false;
    }
    default:
      return false;
  }
}

__global__ void __launch_bounds__(256) k_vertex_op(VOp o, const uint32_t *__restrict__ list, uint64_t size,
                                                   int filter, uint32_t *out_list, uint32_t *out_bits,
                                                   unsigned long long *cnt) {
  uint64_t outdeg = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i0 = blockIdx.x * (uint64_t)blockDim.x; i0 < size; i0 += stride) {
    const uint64_t i = i0 + threadIdx.x;
    bool keep = false;
    uint32_t v = 0;
    if (i < size) {
      v = list[i];
      keep = vop_apply(o, v);
    }
    if (filter) {
      keep = keep && i < size;
      if (keep) atomicOr(out_bits + (v >> 5), 1u << (v & 31));
      const uint64_t slot = warp_append(keep, cnt);
      if (keep) {
        out_list[slot] = v;
        outdeg += o.deg[v];
      }
    }
  }
  if (filter) {
    outdeg = warp_sum(outdeg);
    if (lane_id() == 0 && outdeg) atomicAdd(cnt + 1, (unsigned long long)outdeg);
  }
}

// Sum of |a[i] - b[i]| in 4096-vertex chunks (each summed in order), then
// the chunks in order: the oracle's reduction order, so the value is the
// oracle's to the last bit on the same inputs.  A CTA per chunk (seqsum.cuh);
// a thread per chunk took 800 us at n = 10^6, 51 here.
constexpr uint64_t kL1Chunk = 4096;
constexpr int kL1Block = 512, kL1Terms = 8;
template <class Term>
__device__ __forceinline__ double block_seq_sum(Term term, uint64_t lo, uint64_t hi) {
  __shared__ double stage[seq_at<kL1Terms>(kL1Terms * kL1Block)];
  __shared__ uint32_t mask[kL1Terms * kL1Block / 32];
  __shared__ uint64_t sums[2][32];
  __shared__ SeqSum shared;
  const SeqBlockMem mem{stage, mask, sums, &shared};
  SeqSum s{0.0, false, false};
  unsigned turn = 0;
  for (uint64_t i0 = lo; i0 < hi; i0 += kL1Terms * kL1Block) {
    double x[kL1Terms];
    unsigned in = 0;
#pragma unroll
    for (int r = 0; r < kL1Terms; r++) {
      const uint64_t i = i0 + r * kL1Block + threadIdx.x;
      in |= (i < hi ? 1u : 0u) << r;
      x[r] = i < hi ? term(i) : 0.0;
    }
    seq_block(s, x, in, mem, turn++);
  }
  __syncthreads();
  return s.acc;
}
__global__ void __launch_bounds__(kL1Block, 2) k_l1_chunks(const double *__restrict__ a, const double *__restrict__ b,
                                                        uint64_t n, double *part) {
  const uint64_t nch = (n + kL1Chunk - 1) / kL1Chunk;
  for (uint64_t c = blockIdx.x; c < nch; c += gridDim.x) {
    const double s = block_seq_sum([&](uint64_t i) { return fabs(__dsub_rn(a[i], b[i])); }, c * kL1Chunk,
                                   min((c + 1) * kL1Chunk, n));
    if (threadIdx.x == 0) part[c] = s;
  }
}
__global__ void __launch_bounds__(kL1Block) k_l1_total(const double *__restrict__ part, uint64_t nch, double *out) {
  const double s = block_seq_sum([&](uint64_t c) { return part[c]; }, 0, nch);
  if (threadIdx.x == 0) *out = s;
}

__global__ void k_fill_f64(double *a, uint64_t n, double x) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    a[i] = x;
}

// The runs of g in classes, for any number of rounds while g stays as it is.
int sum_plan(byo_graph *g, SumPlan *p) {
  byo_ctx *ctx = g->ctx;
  BYO_TRY(ws(g, WS_DEFER, g->n + 1, &p->list));
  BYO_TRY(ws(g, WS_BUCKETS, kSumCounts, &p->count));
  BYO_CU(ctx, cudaMemsetAsync(p->count, 0, kSumCounts * 8, ctx->stream));
  p->direct = false;
  const dim3 grid(grid_for(ctx, (g->n + 3) / 4, 1024, 2));
  launch(ctx, k_sum_plan<false>, grid, dim3(1024), 0, (const uint64_t *)g->d_off, g->n, *p);
  launch(ctx, k_sum_plan<true>, grid, dim3(1024), 0, (const uint64_t *)g->d_off, g->n, *p);
  return check_launch(ctx, "edge_map plan");
}

// A round of edgeMap: its counts on the device ([0..1] the members out and their
// edges, [2] k_em_pull's long runs, [3] k_sum_probe's word, from kEmCounts on those
// of a SumPlan).
constexpr int kEmCounts = 8, kEmWords = kEmCounts + kSumCounts;
struct EmRound {
  const SumPlan *plan;
  unsigned long long *cnt;
};

// A round on its own goes by a plan where most runs are too long for a lane (uniform
// 10^5 vertices of degree 64 / 100: 106 / 130 us a call, 131 / 136 without), and from
// kSumLarge slots on where k_sum_probe says so (8 us and a wait of the host: RMAT 2^24
// vertices, 16 draws each, 2.0 ms a call by a plan, 2.4 without; 2^20 no difference).
constexpr uint64_t kSumLarge = 1 << 23, kSumDense = 56, kSumDenseEdges = 1 << 22;

// A dense round of a functor that sums (PR_F, PR_Delta_F): by a plan, or on its
// own.
template <bool kDivide>
int sum_round(byo_graph *g, SumArgs a, Frontier &in, Frontier &out, bool output, EmRound &r) {
  byo_ctx *ctx = g->ctx;
  a.fb = nullptr;
  if (!in.all) {  // (a list may hold an id twice, so its size does not tell)
    BYO_TRY(ensure_bits(g, in));
    a.fb = in.bits;
  }
  a.off = g->d_off;
  a.slots = g->d_slots;
  a.deg = g->d_deg;
  a.n = g->n;
  a.output = output ? 1 : 0;
  a.out_list = out.list;
  a.out_bits = out.bits;
  a.cnt = r.cnt;
  const bool gaps = g->nslots != g->m;
  bool planned = r.plan || (g->m > kSumDenseEdges && g->m > kSumDense * g->n);
  if (!planned && g->nslots > kSumLarge) {
    uint64_t *h = nullptr;
    BYO_TRY(pinned(ctx, 4096, (void **)&h));
    launch(ctx, gaps ? k_sum_probe<true> : k_sum_probe<false>, dim3(1), dim3(1024), 0, a, r.cnt + 3);
    BYO_CU(ctx, cudaMemcpyAsync(h, r.cnt + 3, 8, cudaMemcpyDeviceToHost, ctx->stream));
    BYO_CU(ctx, cudaStreamSynchronize(ctx->stream));
    planned = *h != 0;
  }
  if (!planned) {
    a.plan.count = r.cnt + kEmCounts;
    a.plan.direct = true;
    BYO_TRY(ws(g, WS_DEFER, g->n + 1, &a.plan.list));
    const bool thin = g->nslots < 6 * g->n;  // half of 8 would be past the run's end
    const auto direct = gaps ? (thin ? k_em_sum_direct<kDivide, true, 4> : k_em_sum_direct<kDivide, true, 8>)
                             : (thin ? k_em_sum_direct<kDivide, false, 4> : k_em_sum_direct<kDivide, false, 8>);
    launch(ctx, direct, dim3(grid_for(ctx, (g->n + 31) / 32 * 32, 256)), dim3(256), 0, a);
    // if the longest run that there can be is long
    if ((gaps ? g->nslots : std::min(g->n, g->m)) > kSumShort)
      launch(ctx, k_em_sum_ctas<kDivide, true>, dim3(ctx->num_sms), dim3(kSumBlock), 0, a);
    return check_launch(ctx, "edge_map");
  }
  if (r.plan) {
    a.plan = *r.plan;
    BYO_CU(ctx, cudaMemsetAsync(a.plan.count + 2 * kSumClasses, 0, 8, ctx->stream));
  } else {
    BYO_TRY(sum_plan(g, &a.plan));
  }
  // the three take vertices of their own: side by side, the longest runs' few
  // CTAs leave room for the rest
  BYO_TRY(side_fork(ctx, 0));
  BYO_TRY(side_fork(ctx, 1));
  k_em_sum_ctas<kDivide, false><<<ctx->num_sms, kSumBlock, 0, ctx->side[0]>>>(a);
  k_em_sum_warps<kDivide><<<grid_for(ctx, g->nslots / kSumLaneMax * 32, 256), 256, 0, ctx->side[1]>>>(a);
  ctx->launches += 2;
  launch(ctx, a.fb || output ? k_em_sum_lanes<true> : k_em_sum_lanes<false>, dim3(grid_for(ctx, g->n, 256)), dim3(256),
         0, a);
  BYO_TRY(side_join(ctx, 0));
  BYO_TRY(side_join(ctx, 1));
  return check_launch(ctx, "edge_map");
}

// Slots up to which the divisions are made one an edge: one a vertex is a launch
// of its own (2.5 us), but a warp's 32 terms take a division's time if one needs it.
constexpr uint64_t kDivideSlots = 1 << 16;

int pull_round(byo_graph *g, const PrF &f, Frontier &in, Frontier &out, bool output, EmRound &r) {
  SumArgs a{};
  a.stride = 1;
  a.sum = f.pn;
  if (!r.plan && g->nslots <= kDivideSlots) {
    a.val = f.pc;
    return sum_round<true>(g, a, in, out, output, r);
  }
  double *val = nullptr;
  BYO_TRY(ws(g, WS_PR_D, g->n + 1, &val));
  launch(g->ctx, k_em_values, dim3(grid_for(g->ctx, g->n, 256)), dim3(256), 0, f, g->n, val);
  a.val = val;
  return sum_round<false>(g, a, in, out, output, r);
}

int pull_round(byo_graph *g, const PrDeltaF &f, Frontier &in, Frontier &out, bool output, EmRound &r) {
  SumArgs a{};
  a.val = f.delta;
  a.stride = 2;
  a.at = 1;
  a.sum = f.ngh;
  a.zero_marks = 1;
  return sum_round<false>(g, a, in, out, output, r);
}

int pull_round(byo_graph *g, const LabelF &f, Frontier &in, Frontier &out, bool output, EmRound &r) {
  byo_ctx *ctx = g->ctx;
  unsigned long long *const cnt = r.cnt;
  BYO_TRY(ensure_bits(g, in));
  uint32_t *defer = nullptr;
  BYO_TRY(ws(g, WS_DEFER, g->n + 1, &defer));
  const dim3 grid(grid_for(ctx, (g->n + 31) / 32 * 32, 256));
  launch(ctx, k_em_pull<LabelF>, grid, dim3(256), 0, (const uint64_t *)g->d_off, (const uint32_t *)g->d_slots,
         (const uint32_t *)g->d_deg, f, (const uint32_t *)in.bits, g->n, output ? 1 : 0, out.list, out.bits, cnt,
         defer);
  launch(ctx, k_em_pull_long<LabelF>, grid, dim3(256), 0, (const uint64_t *)g->d_off, (const uint32_t *)g->d_slots,
         (const uint32_t *)g->d_deg, f, (const uint32_t *)in.bits, output ? 1 : 0, out.list, out.bits, cnt,
         (const uint32_t *)defer);
  return check_launch(ctx, "edge_map");
}

template <class F>
int run_round(byo_graph *g, const F &f, Frontier &in, Frontier &out, int mode, bool output, EmRound &r) {
  byo_ctx *ctx = g->ctx;
  const int block = 256;
  if (mode == MODE_PULL) {
    BYO_TRY(pull_round(g, f, in, out, output, r));
  } else {  // sparse, blocked and dense forward: updateAtomic from the members
    BYO_TRY(ensure_list(g, in));
    if (in.size)
      launch(ctx, k_em_push<F>, dim3(grid_for(ctx, in.size * 32, block)), dim3(block), 0,
             (const uint64_t *)g->d_off, (const uint32_t *)g->d_slots, (const uint32_t *)g->d_deg, f,
             (const uint32_t *)in.list, in.size, output ? 1 : 0, out.list, out.bits, r.cnt);
  }
  return check_launch(ctx, "edge_map");
}

}  // namespace

int ensure_list(byo_graph *g, Frontier &f) {
  if (f.has_list) return BYO_OK;
  byo_ctx *ctx = g->ctx;
  unsigned long long *cnt = nullptr;
  BYO_TRY(ws(g, WS_STATS, 4, (uint64_t **)&cnt));
  BYO_CU(ctx, cudaMemsetAsync(cnt, 0, 16, ctx->stream));
  const uint64_t W = (g->n + 31) / 32;
  launch(ctx, k_bits_to_list, dim3(grid_for(ctx, W * 32, 256)), dim3(256), 0, (const uint32_t *)f.bits, g->n,
         (const uint32_t *)g->d_deg, f.list, cnt);
  unsigned long long h[2] = {0, 0};
  BYO_CU(ctx, cudaMemcpyAsync(h, cnt, 16, cudaMemcpyDeviceToHost, ctx->stream));
  BYO_CU(ctx, cudaStreamSynchronize(ctx->stream));
  f.size = h[0];
  f.outdeg = h[1];
  f.has_list = true;
  return check_launch(ctx, "frontier list");
}

int frontier_from_bits(byo_graph *g, const uint32_t *d_bits, Frontier &f) {
  byo_ctx *ctx = g->ctx;
  const uint64_t W = (g->n + 31) / 32;
  launch(ctx, k_bits_copy, dim3(grid_for(ctx, W, 256)), dim3(256), 0, d_bits, g->n, f.bits);
  f.has_bits = true;
  f.has_list = false;
  f.dense = true;
  f.all = d_bits == nullptr;
  BYO_TRY(ensure_list(g, f));
  return BYO_OK;
}

static int edge_map_planned(byo_graph *g, const FunctorArgs &fa, Frontier &in, Frontier &out, int mode, bool output,
                            const SumPlan *plan) {
  byo_ctx *ctx = g->ctx;
  EmRound r{plan, nullptr};
  BYO_TRY(ws(g, WS_STATS, kEmWords, (uint64_t **)&r.cnt));
  BYO_CU(ctx, cudaMemsetAsync(r.cnt, 0, kEmWords * 8, ctx->stream));
  switch (fa.kind) {
    case BYO_F_BFS_LABEL: BYO_TRY(run_round(g, LabelF{fa.parents, fa.src}, in, out, mode, output, r)); break;
    case BYO_F_PR: BYO_TRY(run_round(g, PrF{fa.p_curr, fa.p_next, g->d_deg}, in, out, mode, output, r)); break;
    case BYO_F_PR_DELTA: BYO_TRY(run_round(g, PrDeltaF{fa.delta, fa.ngh}, in, out, mode, output, r)); break;
    default: return set_error(ctx, BYO_EINVAL, "edge_map: unknown functor kind");
  }
  unsigned long long h[2] = {0, 0};
  if (output) {  // no output: the host waits for nothing
    BYO_CU(ctx, cudaMemcpyAsync(h, r.cnt, 16, cudaMemcpyDeviceToHost, ctx->stream));
    BYO_CU(ctx, cudaStreamSynchronize(ctx->stream));
  }
  out.size = h[0];
  out.outdeg = h[1];
  out.has_list = out.has_bits = true;
  out.dense = mode == MODE_PULL || mode == MODE_DENSE_FWD;
  return BYO_OK;
}

int generic_edge_map(byo_graph *g, const FunctorArgs &fa, Frontier &in, Frontier &out, int mode, bool output) {
  return edge_map_planned(g, fa, in, out, mode, output, nullptr);
}

int vertex_op_run(byo_graph *g, const VertexOpArgs &op, Frontier &in, Frontier *out) {
  byo_ctx *ctx = g->ctx;
  BYO_TRY(ensure_list(g, in));
  VOp o;
  o.kind = op.kind;
  o.a = op.a;
  o.b = op.b;
  o.c = op.c;
  o.damping = op.damping;
  o.eps2 = op.eps2;
  o.one_over_n = 1.0 / (double)g->n;
  o.added = (1.0 - op.damping) * o.one_over_n;
  o.deg = g->d_deg;
  unsigned long long *cnt = nullptr;
  BYO_TRY(ws(g, WS_STATS, 4, (uint64_t **)&cnt));
  BYO_CU(ctx, cudaMemsetAsync(cnt, 0, 16, ctx->stream));
  if (in.size)
    launch(ctx, k_vertex_op, dim3(grid_for(ctx, in.size, 256)), dim3(256), 0, o, (const uint32_t *)in.list,
           in.size, out ? 1 : 0, out ? out->list : nullptr, out ? out->bits : nullptr, cnt);
  BYO_TRY(check_launch(ctx, "vertex_map"));
  if (out) {
    unsigned long long h[2] = {0, 0};
    BYO_CU(ctx, cudaMemcpyAsync(h, cnt, 16, cudaMemcpyDeviceToHost, ctx->stream));
    BYO_CU(ctx, cudaStreamSynchronize(ctx->stream));
    out->size = h[0];
    out->outdeg = h[1];
    out->has_list = out->has_bits = true;
    out->dense = false;
  }
  return BYO_OK;
}

// The L1 distance of a and b on ctx->side[2], into h_out (pinned) when `done`
// has happened.
static int l1_diff(byo_graph *g, const double *a, const double *b, double *d_part, double *h_out, cudaEvent_t done) {
  byo_ctx *ctx = g->ctx;
  const uint64_t nch = (g->n + kL1Chunk - 1) / kL1Chunk;
  BYO_TRY(side_fork(ctx, 2));
  cudaStream_t st = ctx->side[2];
  k_l1_chunks<<<grid_for(ctx, nch * kL1Block, kL1Block, 4), kL1Block, 0, st>>>(a, b, g->n, d_part);
  k_l1_total<<<1, kL1Block, 0, st>>>(d_part, nch, d_part + nch);
  ctx->launches += 2;
  BYO_CU(ctx, cudaMemcpyAsync(h_out, d_part + nch, 8, cudaMemcpyDeviceToHost, st));
  BYO_CU(ctx, cudaEventRecord(done, st));
  return check_launch(ctx, "l1");
}

// PageRank_edgeMap (benchmarks/PageRank/PageRank.h:80-123) through the
// generic edgeMap: p_curr = 1/n, frontier = every vertex; each iteration
// edgeMap(PR_F, threshold 0, no_output) (always dense), vertexMap(PR_Vertex_F),
// L1 between the iterates, stop below eps; reset p_curr and swap.  Returns
// the last computed iterate (the reference's final swap would hand back the
// zeroed one when max_iters ends the loop).
//
// The L1 distance of an iteration is computed beside the next one, which writes
// the third of three buffers: when the distance ends the loop, that iteration
// is left unread.  So the host's wait and the L1 kernels (60 us, few CTAs) leave
// the chain of iterations.
int pagerank_edgemap_run(byo_graph *g, double eps, uint32_t max_iters, double *d_p, uint32_t *iters_out,
                         double *l1_out) {
  byo_ctx *ctx = g->ctx;
  const uint64_t n = g->n;
  const uint64_t W = (n + 31) / 32;
  const uint64_t nch = (n + kL1Chunk - 1) / kL1Chunk;
  double *p[3] = {}, *part = nullptr, *h = nullptr;
  BYO_TRY(ws(g, WS_PR_A, n + 1, &p[0]));
  BYO_TRY(ws(g, WS_PR_B, n + 1, &p[1]));
  BYO_TRY(ws(g, WS_LP, n + 1, &p[2]));
  BYO_TRY(ws(g, WS_PR_C, nch + 2, &part));
  BYO_TRY(pinned(ctx, 4096, (void **)&h));
  uint32_t *flist = nullptr, *fbits = nullptr;
  BYO_TRY(ws(g, WS_FRONT_LIST_A, n + 1, &flist));
  BYO_TRY(ws(g, WS_FRONT_BITS_A, W + 1, &fbits));
  Frontier all;
  all.list = flist;
  all.bits = fbits;
  BYO_TRY(frontier_from_bits(g, nullptr, all));
  Frontier none;  // no_output rounds write nothing
  SumPlan plan;   // of the view, which stays as it is
  BYO_TRY(sum_plan(g, &plan));
  launch(ctx, k_fill_f64, dim3(grid_for(ctx, n, 256)), dim3(256), 0, p[0], n, 1.0 / (double)n);
  uint32_t it = 0;  // iterations whose distance is known
  double L1 = 0.0;
  auto wait = [&](uint32_t t) -> int {  // for iteration t's distance
    BYO_CU(ctx, cudaEventSynchronize(ctx->ev[2 + (t & 1)]));
    L1 = h[t & 1];
    it = t + 1;
    return BYO_OK;
  };
  auto loop = [&]() -> int {
    for (uint32_t t = 0; t < max_iters; t++) {
      double *pc = p[t % 3], *pn = p[(t + 1) % 3];
      BYO_TRY(memset_async(ctx, pn, 0, n * 8));
      FunctorArgs f{};
      f.kind = BYO_F_PR;
      f.p_curr = pc;
      f.p_next = pn;
      BYO_TRY(edge_map_planned(g, f, all, none, MODE_PULL, false, &plan));
      VertexOpArgs vf{BYO_VOP_PR_UPDATE, pn, nullptr, nullptr, 0.85, 0.0};
      BYO_TRY(vertex_op_run(g, vf, all, nullptr));
      BYO_TRY(l1_diff(g, pc, pn, part, h + (t & 1), ctx->ev[2 + (t & 1)]));
      if (t) {
        BYO_TRY(wait(t - 1));
        if (L1 < eps) return BYO_OK;
      }
    }
    return max_iters ? wait(max_iters - 1) : BYO_OK;
  };
  const int rc = loop();
  if (max_iters) BYO_TRY(side_join(ctx, 2));
  BYO_TRY(rc);
  BYO_CU(ctx, cudaMemcpyAsync(d_p, p[it % 3], n * 8, cudaMemcpyDeviceToDevice, ctx->stream));
  if (iters_out) *iters_out = it;
  if (l1_out) *l1_out = L1;
  return check_launch(ctx, "pagerank_edgemap");
}

}  // namespace byo
