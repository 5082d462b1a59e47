// tc.cu -- triangle counting (Triangle_degree_ordering,
// benchmarks/TriangleCounting/ShunTangwongsan15/Triangle.h:167-204).
//
// Vertices are renamed by rank, 0 = the largest (degree, id), so an edge
// points from the larger rank to the smaller and N+(u) holds the neighbours of
// u with smaller ranks.  One pass over the adjacency writes every row in rank
// space as [N+ sorted | N-] (k_tc_rows, k_tc_rows_block).
//
// A triangle w < v < u is counted at its middle vertex v: N+(v) becomes a set
// in shared memory and, for every u of N-(v), the part of N+(u) below v is
// looked up in it.  The sorted prefix makes that sum over u of |N+(u)|^2 / 2
// lookups, where looking up all of N+(v) for every v of N+(u) makes sum over
// the edges of |N+(v)|: 7.2e9 against 2.9e10 at RMAT 2^22 with 2^26 draws
// (whose hash-set lookups took 613 ms a count; this one takes 13.3).
// The set of a v with a long N- is a map over the ranks below it (one shared
// load per lookup, no probe chain), made by a CTA; that of one with few
// neighbours a hash set, made by a warp.  The counts are whole numbers, so no order
// matters.
//
// N-(v) comes from v's own row, which has it where every edge is stored at both
// ends.  A graph of keys that were not symmetrised may not: then N- is made from
// the rows' N+ (k_tc_in).  Which it is the rows tell as they are written, by the sum
// of a keyed 64-bit mix of every u -> v in N+ less that of every one in N- (tc_mark):
// 0 where they are the same edges; where they are not, 0 with a chance of 2^-64,
// under another key (from the clock) for each count.  Looking for v in every list
// that the count reads anyway is exact and took 10%: 13.25 -> 14.54 ms on the graph
// above; this 13.27.
#include <algorithm>
#include <chrono>

#include "device.cuh"
#include "engine.h"
#include "internal.h"
#include "scan.cuh"

namespace byo {

namespace {

// Rows above this degree are split off to a CTA; the others fit a warp's stage.
constexpr uint32_t kTcRowMax = 1024;
// Longest N+ sorted in a CTA's shared memory; longer ones stay unsorted and
// are looked up whole.
constexpr uint32_t kTcSortCap = 16384;
// Maps of N-(v)'s CTAs: a byte per rank in 112 KB (two 1024-thread CTAs share an
// SM) for the v with a long N-, a bit per rank in 28 KB (eight 256-thread CTAs)
// for the rest below kTcMidRanks, a bit per rank in 112 KB above.
constexpr uint32_t kTcMapBytes = 112 * 1024, kTcMidBytes = 28 * 1024;
constexpr uint32_t kTcByteRanks = kTcMapBytes, kTcMidRanks = 8 * kTcMidBytes;
constexpr uint32_t kTcHashMax = 256;           // longest N+ in a warp's hash set
constexpr uint32_t kTcHash = 4 * kTcHashMax;   // its table's entries: load <= 1/4
constexpr uint32_t kTcHashFew = 16;            // longest N+ in half a warp's
constexpr uint32_t kTcHashSplit = 1 << 16;     // ranks from which they have a launch of their own
constexpr uint32_t kTcChunk = 4096;            // u's of one map work unit

// Which kernel counts v: a warp with a hash set when N+ is short and N- too
// short to pay for a CTA and its map.
enum { kTcByte = 0, kTcMid = 1, kTcFar = 2, kTcClasses = 3, kTcHashed = 3, kTcNone = 4 };
__device__ __forceinline__ int tc_class(uint32_t v, uint32_t nout, uint32_t nin) {
  if (nout == 0 || nin == 0) return kTcNone;
  if (nout <= kTcHashMax && nin < (v < kTcMidRanks ? 32u : 256u)) return kTcHashed;
  return v < kTcByteRanks && nin >= 512 ? kTcByte : v < kTcMidRanks ? kTcMid : kTcFar;
}

// A row holds its degree rounded up to 4, and 4 more: N+ from the start, padded
// to a multiple of 4 with kSentinel so that four entries load at once, N- at
// the end.
__host__ __device__ __forceinline__ uint64_t tc_round4(uint64_t x) { return (x + 3) & ~3ull; }

// A row's N+: start << 24 | length (rows start below 2^40; |N+| <= sqrt(2m)).
__device__ __forceinline__ uint64_t tc_row(uint64_t start, uint32_t len) { return start << 24 | len; }

__global__ void k_tc_rank_keys(const uint32_t *__restrict__ deg, uint64_t n, uint64_t *keys) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x)
    keys[v] = ((uint64_t)deg[v] << 32) | v;
}

// rank[vertex], and where the ranks of degree >= 2 (info[0]) and of degree >
// kTcRowMax (info[1]) end.
__global__ void k_tc_ranks(const uint64_t *__restrict__ sorted, uint64_t n, uint32_t *rank, uint64_t *info) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t k = sorted[i];
    const uint32_t d = (uint32_t)(k >> 32), below = i ? (uint32_t)(sorted[i - 1] >> 32) : 0;
    rank[(uint32_t)k] = (uint32_t)(n - 1 - i);
    if (d >= 2 && below < 2) info[0] = n - i;
    if (d > kTcRowMax && below <= kTcRowMax) info[1] = n - i;
  }
}

struct InRowSize {
  const uint64_t *sorted;
  uint64_t n;
  __device__ uint64_t operator()(uint64_t v) const { return tc_round4(sorted[n - 1 - v] >> 32) + 4; }
};

struct TcRows {
  const uint64_t *off;
  const uint32_t *slots;
  const uint32_t *rank;
  const uint64_t *sorted;  // (degree, vertex) ascending
  const uint64_t *roff;    // start of each rank's row
  uint64_t n;
  uint32_t n2;             // ranks of degree >= 2: no other vertex is in a triangle
  uint32_t *nbr;           // the rows
  uint64_t *row;           // N+ of each rank (tc_row)
  uint64_t *in;            // start of N- of each rank
  uint32_t *icnt;          // |N-| of each rank, vertices of degree 1 left out
  uint64_t seed;
  unsigned long long *differ;  // 0: N- holds the edges of N+
};

// The mix of an edge u -> v (the finalizer of SplitMix64, Steele, Lea & Flood 2014).
__device__ __forceinline__ uint64_t tc_mark(uint64_t seed, uint32_t u, uint32_t v) {
  uint64_t z = ((uint64_t)u << 32 | v) ^ seed;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// A warp per row: 128 neighbours' ranks in flight, N+ staged in shared memory
// and sorted there, N- written from the row's end.  Bound by the rank gathers
// (one sector each) and the chain vertex -> row -> neighbour -> rank, hidden by
// the warps in flight; with k_tc_rows_block 2.5 ms at RMAT 2^22 / 2^26 draws,
// where two passes of a warp per vertex (the hubs last) took 14.0.
__global__ void __launch_bounds__(256) k_tc_rows(TcRows a, uint32_t v0) {
  __shared__ uint32_t stage[8][kTcRowMax];
  __shared__ unsigned long long sm[9];
  uint32_t *st = stage[threadIdx.x >> 5];
  const unsigned lane = lane_id();
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  // the next row's place is loaded during this one, and the vertex after that
  auto vertex = [&](uint64_t t) { return t < a.n2 ? a.sorted[a.n - 1 - t] : 0; };
  uint64_t key = vertex(v0 + gw), key1 = vertex(v0 + gw + nw);
  uint64_t b = a.off[(uint32_t)key], e = a.off[(uint32_t)key + 1];
  unsigned long long mark = 0;
  for (uint64_t t = v0 + gw; t < a.n2; t += nw) {
    const uint32_t v = (uint32_t)t;
    const uint64_t key2 = vertex(t + 2 * nw), b1 = a.off[(uint32_t)key1], e1 = a.off[(uint32_t)key1 + 1];
    const uint64_t base = a.roff[t], end = base + tc_round4(key >> 32) + 4;
    uint32_t c = 0, ic = 0;
    if (e - b <= 32) {
      uint32_t x = b + lane < e ? a.slots[b + lane] : kSentinel;
      x = x != kSentinel ? __ldg(a.rank + x) : kSentinel;
      const bool out = x < v, in = x > v && x < a.n2;
      const unsigned mo = __ballot_sync(kFull, out), mi = __ballot_sync(kFull, in);
      const uint64_t m = tc_mark(a.seed, out ? v : x, out ? x : v);
      if (out) {
        st[__popc(mo & lanemask_lt())] = x;
        mark += m;
      }
      if (in) {
        a.nbr[end - 1 - __popc(mi & lanemask_lt())] = x;
        mark -= m;
      }
      c = __popc(mo);
      ic = __popc(mi);
      b = e;
    }
    for (uint64_t j0 = b; j0 < e; j0 += 128) {
      uint32_t x[4];
#pragma unroll
      for (int q = 0; q < 4; q++) x[q] = j0 + q * 32 + lane < e ? a.slots[j0 + q * 32 + lane] : kSentinel;
#pragma unroll
      for (int q = 0; q < 4; q++) x[q] = x[q] != kSentinel ? __ldg(a.rank + x[q]) : kSentinel;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const bool out = x[q] < v, in = x[q] > v && x[q] < a.n2;
        const unsigned mo = __ballot_sync(kFull, out), mi = __ballot_sync(kFull, in);
        const uint64_t m = tc_mark(a.seed, out ? v : x[q], out ? x[q] : v);
        if (out) st[c + __popc(mo & lanemask_lt())] = x[q];
        if (in) a.nbr[end - 1 - (ic + __popc(mi & lanemask_lt()))] = x[q];
        mark += out ? m : in ? 0 - m : 0;
        c += __popc(mo);
        ic += __popc(mi);
      }
    }
    __syncwarp();
    if (c <= 32) {
      uint32_t r = lane < c ? st[lane] : kSentinel;
#pragma unroll
      for (int size = 2; size <= 32; size <<= 1) {
        if (size > 8 && c <= size / 2) break;  // (the lanes past c hold kSentinel)
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
          const uint32_t o = __shfl_xor_sync(kFull, r, stride);
          r = (((lane & size) == 0) == ((lane & stride) == 0)) ? min(r, o) : max(r, o);
        }
      }
      if (lane < tc_round4(c)) a.nbr[base + lane] = r;
    } else {
      const uint32_t P = 1u << (32 - __clz((int)(c - 1)));
      for (uint32_t i = c + lane; i < P; i += 32) st[i] = kSentinel;
      for (uint32_t size = 2; size <= P; size <<= 1)
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
          __syncwarp();
          for (uint32_t i = lane; i < P / 2; i += 32) {
            const uint32_t lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
            const uint32_t x = st[lo], z = st[hi];
            if ((x > z) == ((lo & size) == 0)) {
              st[lo] = z;
              st[hi] = x;
            }
          }
        }
      __syncwarp();
      for (uint32_t i = lane; i < tc_round4(c); i += 32) a.nbr[base + i] = st[i];
    }
    if (lane == 0) {
      a.row[t] = tc_row(base, c);
      a.in[t] = end - ic;
      a.icnt[t] = ic;
    }
    __syncwarp();
    key = key1;
    key1 = key2;
    b = b1;
    e = e1;
  }
  mark = block_sum(mark, sm);
  if (threadIdx.x == 0 && mark) atomicAdd(a.differ, mark);
}

// A CTA per row above kTcRowMax: 4096 neighbours a step, placed by a block scan
// of the threads' counts (a row of 500 K neighbours takes 120 steps, so no
// row holds the launch up).  N+ up to `cap` entries is sorted in shared memory.
constexpr int kTcRowBlock = 1024;
__global__ void __launch_bounds__(kTcRowBlock) k_tc_rows_block(TcRows a, uint32_t v1, uint32_t cap) {
  extern __shared__ uint32_t buf[];  // next power of two >= cap entries
  __shared__ uint32_t sm[kTcRowBlock / 32 + 1];
  __shared__ unsigned long long sm64[kTcRowBlock / 32 + 1];
  unsigned long long mark = 0;
  for (uint32_t v = blockIdx.x; v < v1; v += gridDim.x) {
    const uint64_t key = a.sorted[a.n - 1 - v];
    const uint32_t y = (uint32_t)key;
    const uint64_t b = a.off[y], e = a.off[y + 1], base = a.roff[v], end = base + tc_round4(key >> 32) + 4;
    uint32_t c = 0, ic = 0;
    for (uint64_t j0 = b; j0 < e; j0 += 4 * kTcRowBlock) {
      uint32_t x[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint64_t j = j0 + q * kTcRowBlock + threadIdx.x;
        x[q] = j < e ? a.slots[j] : kSentinel;
      }
#pragma unroll
      for (int q = 0; q < 4; q++) x[q] = x[q] != kSentinel ? __ldg(a.rank + x[q]) : kSentinel;
      uint32_t mine = 0;  // N+ entries in the low half, N- entries in the high
#pragma unroll
      for (int q = 0; q < 4; q++) mine += x[q] < v ? 1u : x[q] > v && x[q] < a.n2 ? 1u << 16 : 0u;
      uint32_t tot;
      const uint32_t pre = block_exclusive_scan(mine, sm, &tot);
      uint32_t o = c + (pre & 0xFFFF), i = ic + (pre >> 16);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if (x[q] < v) {
          if (o < cap) buf[o] = x[q]; else a.nbr[base + o] = x[q];
          o++;
          mark += tc_mark(a.seed, v, x[q]);
        } else if (x[q] > v && x[q] < a.n2) {
          a.nbr[end - 1 - i++] = x[q];
          mark -= tc_mark(a.seed, x[q], v);
        }
      }
      c += tot & 0xFFFF;
      ic += tot >> 16;
    }
    __syncthreads();
    if (c > 1 && c <= cap) {
      const uint32_t P = 1u << (32 - __clz((int)(c - 1)));
      for (uint32_t i = c + threadIdx.x; i < P; i += blockDim.x) buf[i] = kSentinel;
      for (uint32_t size = 2; size <= P; size <<= 1)
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
          __syncthreads();
          for (uint32_t i = threadIdx.x; i < P / 2; i += blockDim.x) {
            const uint32_t lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
            const uint32_t x = buf[lo], z = buf[hi];
            if ((x > z) == ((lo & size) == 0)) {
              buf[lo] = z;
              buf[hi] = x;
            }
          }
        }
      __syncthreads();
    }
    for (uint32_t i = threadIdx.x; i < min(c, cap); i += blockDim.x) a.nbr[base + i] = buf[i];
    if (c + threadIdx.x < tc_round4(c)) a.nbr[base + c + threadIdx.x] = kSentinel;
    if (threadIdx.x == 0) {
      a.row[v] = tc_row(base, c);
      a.in[v] = end - ic;
      a.icnt[v] = ic;
    }
    __syncthreads();
  }
  mark = block_sum(mark, sm64);
  if (threadIdx.x == 0 && mark) atomicAdd(a.differ, mark);
}

// N- from the rows' N+, a warp a row: how long each is, then (kPlace, from icnt
// zero again) its entries at nbr + in (a start counts from nbr wherever the list is).
template <bool kPlace>
__global__ void __launch_bounds__(256) k_tc_in(uint32_t *nbr, const uint64_t *__restrict__ row, uint32_t n2,
                                               const uint64_t *__restrict__ in, uint32_t *icnt) {
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t u = gw; u < n2; u += nw) {
    const uint32_t *list = nbr + (row[u] >> 24);
    for (uint32_t i = lane_id(); i < ((uint32_t)row[u] & 0xFFFFFF); i += 32) {
      const uint32_t v = list[i], at = atomicAdd(icnt + v, 1u);
      if (kPlace) nbr[in[v] + at] = (uint32_t)u;
    }
  }
}
struct OutStart {
  uint64_t *start, base;
  __device__ void operator()(uint64_t i, uint64_t pre, uint64_t) const { start[i] = base + pre; }
};

// Work units of the map kernels: chunks of N-(v), v << 32 | chunk, class c's at
// units + c * cap, counted in nunits[c].
__global__ void __launch_bounds__(256) k_tc_units(const uint64_t *__restrict__ row, const uint32_t *__restrict__ icnt,
                                                  uint32_t n2, uint64_t *units, uint64_t cap,
                                                  unsigned long long *nunits) {
  for (uint64_t base = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) & ~31ull; base < n2;
       base += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t v = base + lane_id();
    const uint32_t nin = v < n2 ? icnt[v] : 0;
    const int c = v < n2 ? tc_class((uint32_t)v, (uint32_t)row[v] & 0xFFFFFF, nin) : kTcNone;
#pragma unroll
    for (int k = 0; k < kTcClasses; k++) {
      if (!__ballot_sync(kFull, c == k)) continue;
      const uint32_t mine = c == k ? (nin + kTcChunk - 1) / kTcChunk : 0;
      const uint32_t incl = warp_inclusive_scan(mine);
      unsigned long long at = 0;
      if (lane_id() == 31) at = atomicAdd(nunits + k, (unsigned long long)incl);
      at = __shfl_sync(kFull, at, 31) + incl - mine;
      for (uint32_t q = 0; q < mine; q++) units[k * cap + at + q] = v << 32 | q;
    }
  }
}

// Lookups of N+(u) below v, G lanes to a list, 4 entries a lane: left at the
// first entry >= v when the list is sorted (len <= sorted_cap).  in_set gives
// 1 for an entry of N+(v) and 0 for any other (kSentinel too).  Called by whole
// groups of G.
template <int G, class Set>
__device__ __forceinline__ uint32_t tc_lookup(const uint32_t *__restrict__ nbr, uint64_t row, uint32_t v,
                                              uint32_t sorted_cap, const Set &in_set) {
  const unsigned gm = ((1u << G) - 1) << (lane_id() & ~(G - 1));
  const uint32_t len = (uint32_t)row & 0xFFFFFF;
  const uint4 *list = reinterpret_cast<const uint4 *>(nbr + (row >> 24));
  uint32_t cnt = 0;
  for (uint32_t k = 4 * (lane_id() & (G - 1));; k += 4 * G) {
    uint4 x = make_uint4(kSentinel, kSentinel, kSentinel, kSentinel);
    if (k < len) x = __ldg(list + (k >> 2));
    cnt += in_set(x.x) + in_set(x.y) + in_set(x.z) + in_set(x.w);
    // the group's last entry is in its last lane (kSentinel past the end)
    if (__ballot_sync(gm, len <= sorted_cap ? x.w >= v : k + 4 >= len)) break;
  }
  return cnt;
}

// Lookups of the lists of u = ulist[i], ulist[i + kStep], ... below i1, the next
// list's place loaded while one is looked up.
template <int G, uint32_t kStep, class Set>
__device__ __forceinline__ uint64_t tc_lookups(const uint32_t *__restrict__ nbr, const uint64_t *__restrict__ row,
                                               const uint32_t *__restrict__ ulist, uint32_t i, uint32_t i1, uint32_t v,
                                               uint32_t sorted_cap, const Set &set) {
  uint64_t cnt = 0;
  uint64_t cur = i < i1 ? row[ulist[i]] : 0;
  while (i < i1) {
    i += kStep;
    const uint64_t nxt = i < i1 ? row[ulist[i]] : 0;
    cnt += tc_lookup<G>(nbr, cur, v, sorted_cap, set);
    cur = nxt;
  }
  return cnt;
}

// N+(v) over the ranks [w0, w0 + span), a byte or a bit each; the entry at
// span stays 0 and stands for every rank outside.
struct TcBytes {
  static constexpr uint32_t kPerWord = 4;
  uint32_t *map;
  uint32_t w0, span;
  __device__ __forceinline__ void add(uint32_t r) const { reinterpret_cast<unsigned char *>(map)[r] = 1; }
  __device__ __forceinline__ uint32_t operator()(uint32_t w) const {
    return reinterpret_cast<const unsigned char *>(map)[min(w - w0, span)];
  }
};
struct TcBits {
  static constexpr uint32_t kPerWord = 32;
  uint32_t *map;
  uint32_t w0, span;
  __device__ __forceinline__ void add(uint32_t r) const { atomicOr(map + (r >> 5), 1u << (r & 31)); }
  __device__ __forceinline__ uint32_t operator()(uint32_t w) const {
    const uint32_t r = min(w - w0, span);
    return (map[r >> 5] >> (r & 31)) & 1u;
  }
};

// Persistent CTAs take chunks of N-(v) in turn, the next one's number fetched
// while one is counted.  Ranks past the map take further passes over N-(v).
// RMAT 2^22 / 2^26 draws (7.2e9 lookups): bytes 7.2 ms, mid bits 2.1 ms, the
// hash sets 1.0 ms; bits in 16 KB for every v took 13.3 ms, issue-bound (70
// instructions for 32 lookups, 4-byte list loads), and leaving every v of a short
// N- to the hash sets 4.7 ms.  At RMAT 2^20 the byte maps run at 63% of the issue
// slots and 61% of L1 (1.7 conflicts a shared load), 24% of L2.
template <class Set, int kBlock>
__global__ void __launch_bounds__(kBlock, 2048 / kBlock) k_tc_map(const uint32_t *__restrict__ nbr,
                                                        const uint64_t *__restrict__ row,
                                                        const uint64_t *__restrict__ in,
                                                        const uint32_t *__restrict__ icnt,
                                                        const uint64_t *__restrict__ units,
                                                        const unsigned long long *__restrict__ nunits, uint32_t words,
                                                        uint32_t sorted_cap, unsigned long long *next,
                                                        unsigned long long *total) {
  extern __shared__ __align__(16) uint32_t map[];
  __shared__ unsigned long long s_unit[2], sm[kBlock / 32 + 1];
  const uint64_t nu = *nunits;
  const uint32_t room = words * Set::kPerWord - 1;  // one entry stays 0
  uint64_t cnt = 0;
  uint32_t have = kSentinel;  // the vertex whose whole map is in shared memory
  if (threadIdx.x == 0) s_unit[0] = atomicAdd(next, 1ull);
  __syncthreads();
  for (int turn = 0;; turn ^= 1) {
    const uint64_t t = s_unit[turn];
    if (t >= nu) break;
    if (threadIdx.x == 0) s_unit[turn ^ 1] = atomicAdd(next, 1ull);
    const uint64_t unit = units[t];
    const uint32_t v = (uint32_t)(unit >> 32);
    const uint64_t own = row[v];
    const uint32_t nout = (uint32_t)own & 0xFFFFFF;
    const uint32_t i0 = (uint32_t)unit * kTcChunk, i1 = min(icnt[v], i0 + kTcChunk);
    const uint32_t *ulist = nbr + in[v];
    for (uint64_t w0 = 0; w0 < v; w0 += room) {
      const uint32_t span = (uint32_t)min(v - w0, (uint64_t)room);
      const Set set{map, (uint32_t)w0, span};
      if (have != v) {
        uint4 *m4 = reinterpret_cast<uint4 *>(map);
        for (uint32_t i = threadIdx.x; i <= span / (4 * Set::kPerWord); i += blockDim.x) m4[i] = make_uint4(0, 0, 0, 0);
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < nout; i += blockDim.x) {
          const uint32_t r = nbr[(own >> 24) + i] - (uint32_t)w0;
          if (r < span) set.add(r);
        }
        have = v <= room ? v : kSentinel;
        __syncthreads();
      }
      cnt += tc_lookups<8, kBlock / 8>(nbr, row, ulist, i0 + (threadIdx.x >> 3), i1, v, sorted_cap, set);
      __syncthreads();
    }
  }
  const unsigned long long tot = block_sum((unsigned long long)cnt, sm);
  if (threadIdx.x == 0 && tot) atomicAdd(total, tot);
}

struct TcHash {
  const uint32_t *t;
  uint32_t mask, shift;
  uint32_t v;
  __device__ __forceinline__ uint32_t operator()(uint32_t x) const {
    if (x >= v) return 0;
    uint32_t h = (x * 0x9E3779B1u) >> shift;
    for (;;) {
      const uint32_t y = t[h];
      if (y == x) return 1;
      if (y == kSentinel) return 0;
      h = (h + 1) & mask;
    }
  }
};

// L lanes to each hashed v (tc_class): N+(v) in an open-addressing hash set of
// the next power of two >= 4 |N+(v)| entries (a miss, most lookups, ends after ~1.2
// probes).  Up to 16 entries half a warp, 8 u's at a time with two lanes to a list
// (the lists of the u's are then as short); more a warp, 4 u's at a time.  Bound by
// instructions and the chain row -> lists -> rows of the u's -> their lists: uniform
// 10^6 vertices of degree 16 492 us with the halves, 665 by warps alone.  Below
// kTcHashSplit ranks a second launch costs what it saves (Chung-Lu 10^4 240 us a count
// with it, 226 without; uniform 10^5 346 with, 360 without).
template <int L>
__global__ void __launch_bounds__(256) k_tc_hash(const uint32_t *__restrict__ nbr, const uint64_t *__restrict__ row,
                                                 const uint64_t *__restrict__ in, const uint32_t *__restrict__ icnt,
                                                 uint32_t n2, uint32_t few, uint32_t sorted_cap,
                                                 unsigned long long *total) {
  constexpr uint32_t kTable = L == 32 ? kTcHash : 4 * kTcHashFew;
  constexpr int G = L == 32 ? 8 : 2;
  __shared__ uint32_t tabs[256 / L][kTable];
  __shared__ unsigned long long sm[9];
  const unsigned lane = threadIdx.x % L, mask = L == 32 ? kFull : ((1u << (L & 31)) - 1) << (lane_id() & ~(L - 1));
  uint32_t *tab = tabs[threadIdx.x / L];
  const uint64_t g0 = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / L;
  const uint64_t ng = ((uint64_t)gridDim.x * blockDim.x) / L;
  uint64_t cnt = 0;
  uint64_t own = g0 < n2 ? row[g0] : 0;  // loaded ahead: most v's are passed over
  uint32_t ni = g0 < n2 ? icnt[g0] : 0;
  for (uint64_t t = g0; t < n2; t += ng) {
    const uint64_t own1 = t + ng < n2 ? row[t + ng] : 0;
    const uint32_t ni1 = t + ng < n2 ? icnt[t + ng] : 0, nout = (uint32_t)own & 0xFFFFFF;
    if (tc_class((uint32_t)t, nout, ni) == kTcHashed && (nout <= few) == (L < 32)) {
      const uint32_t lg = max(6, 32 - __clz((int)(4 * nout - 1))), size = 1u << lg;
      for (uint32_t i = lane; i < size; i += L) tab[i] = kSentinel;
      __syncwarp(mask);
      for (uint32_t i = lane; i < nout; i += L) {
        const uint32_t x = nbr[(own >> 24) + i];
        uint32_t h = (x * 0x9E3779B1u) >> (32 - lg);
        while (atomicCAS(tab + h, kSentinel, x) != kSentinel) h = (h + 1) & (size - 1);
      }
      __syncwarp(mask);
      const TcHash set{tab, size - 1, 32 - lg, (uint32_t)t};
      cnt += tc_lookups<G, L / G>(nbr, row, nbr + in[t], lane / G, ni, (uint32_t)t, sorted_cap, set);
      __syncwarp(mask);
    }
    own = own1;
    ni = ni1;
  }
  const unsigned long long tot = block_sum((unsigned long long)cnt, sm);
  if (threadIdx.x == 0 && tot) atomicAdd(total, tot);
}

}  // namespace

int tc_run(byo_graph *g, uint64_t *count) {
  byo_ctx *ctx = g->ctx;
  const uint64_t n = g->n;
  *count = 0;
  if (n == 0) return BYO_OK;
  uint64_t *keys = nullptr, *sorted = nullptr, *h = nullptr;
  uint32_t *rank = nullptr;
  unsigned long long *d = nullptr;  // [0] triangles, [1..3] next units, [4..5] ranks of
                                    // degree >= 2, > kTcRowMax, [6..8] units, [9] whether
                                    // N- differs from N+
  BYO_TRY(ws(g, WS_TC_OFF, 2 * n + 2, &keys));
  BYO_TRY(ws(g, WS_TC_RANK, n, &rank));
  BYO_TRY(ws(g, WS_MISC, 20, (uint32_t **)&d));
  BYO_TRY(pinned(ctx, 4096, (void **)&h));
  BYO_CU(ctx, cudaMemsetAsync(d, 0, 80, ctx->stream));
  launch(ctx, k_tc_rank_keys, dim3(grid_for(ctx, n, 256)), dim3(256), 0, (const uint32_t *)g->d_deg, n, keys);
  const uint64_t id_mask = sig_mask_for(n + 1) & 0xFFFFFFFFull;  // degrees are at most n
  BYO_TRY(sort_u64(ctx, keys, keys + n + 1, n, (id_mask << 32) | id_mask, &sorted));
  launch(ctx, k_tc_ranks, dim3(grid_for(ctx, n, 256)), dim3(256), 0, (const uint64_t *)sorted, n, rank,
         (uint64_t *)(d + 4));
  BYO_CU(ctx, cudaMemcpyAsync(h, d + 4, 16, cudaMemcpyDeviceToHost, ctx->stream));
  BYO_CU(ctx, cudaStreamSynchronize(ctx->stream));
  const uint32_t n2 = (uint32_t)h[0], nh = (uint32_t)h[1];
  if (n2 < 3) return check_launch(ctx, "triangle_count");
  uint64_t *roff = nullptr, *row = nullptr;
  uint32_t *icnt = nullptr, *nbr = nullptr;
  BYO_TRY(ws(g, WS_SCAN, n2, &roff));
  BYO_TRY(ws(g, WS_TC_CNT, 2 * (uint64_t)n2, &row));
  BYO_TRY(ws(g, WS_BUCKETS, n2, &icnt));
  BYO_TRY(ws(g, WS_TC_NBR, g->m + 7 * (uint64_t)n2, &nbr));
  uint64_t *in = row + n2;
  const uint64_t *tot = nullptr;
  BYO_TRY(scan_apply(ctx, n2, InRowSize{sorted, n}, OutPrefix{roff}, &tot));
  const uint32_t stage = effective_tuning(g).tc_stage;
  const uint32_t cap = std::min(kTcSortCap, stage);
  const uint64_t seed = (uint64_t)std::chrono::steady_clock::now().time_since_epoch().count() * 0x9E3779B97F4A7C15ull;
  TcRows a{g->d_off, g->d_slots, rank, sorted, roff, n, n2, nbr, row, in, icnt, seed, d + 9};
  if (nh) {
    uint32_t p2 = 1;
    while (p2 < cap) p2 <<= 1;
    BYO_CU(ctx, cudaFuncSetAttribute(k_tc_rows_block, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kTcSortCap * 4));
    launch(ctx, k_tc_rows_block, dim3(std::min<uint32_t>(nh, 2 * ctx->num_sms)), dim3(kTcRowBlock), (size_t)p2 * 4, a,
           nh, cap);
  }
  if (n2 > nh) launch(ctx, k_tc_rows, dim3(grid_for(ctx, (uint64_t)(n2 - nh) * 32, 256)), dim3(256), 0, a, nh);
  uint64_t *units = nullptr;
  const uint64_t ucap = (uint64_t)n2 + g->m / kTcChunk;
  BYO_TRY(ws(g, WS_TC_OFF, kTcClasses * ucap, &units));  // `sorted` is done with
  // counts into h
  auto count_all = [&]() -> int {
    launch(ctx, k_tc_units, dim3(grid_for(ctx, n2, 256)), dim3(256), 0, (const uint64_t *)row, (const uint32_t *)icnt, n2,
           units, ucap, d + 6);
    auto count_class = [&](int c, auto kernel, int block, uint32_t bytes) -> int {
      const uint32_t words = std::min(stage, bytes / 4);
      BYO_CU(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
      launch_t(ctx, "tc_intersect", kernel, dim3(2048 / block * ctx->num_sms), dim3(block),
               ((size_t)words * 4 + 15) & ~(size_t)15, (const uint32_t *)nbr, (const uint64_t *)row,
               (const uint64_t *)in, (const uint32_t *)icnt, (const uint64_t *)(units + c * ucap),
               (const unsigned long long *)(d + 6 + c), words, cap, d + 1 + c, d);
      return BYO_OK;
    };
    BYO_TRY(count_class(kTcByte, k_tc_map<TcBytes, 1024>, 1024, kTcMapBytes));
    BYO_TRY(count_class(kTcMid, k_tc_map<TcBits, 256>, 256, kTcMidBytes));
    if (n2 > kTcMidRanks) BYO_TRY(count_class(kTcFar, k_tc_map<TcBits, 1024>, 1024, kTcMapBytes));
    const uint32_t few = n2 < kTcHashSplit ? 0 : kTcHashFew;
    launch_t(ctx, "tc_intersect", k_tc_hash<32>, dim3(grid_for(ctx, (uint64_t)n2 * 32, 256)), dim3(256), 0,
             (const uint32_t *)nbr, (const uint64_t *)row, (const uint64_t *)in, (const uint32_t *)icnt, n2, few, cap, d);
    if (few)
      launch_t(ctx, "tc_intersect", k_tc_hash<16>, dim3(grid_for(ctx, (uint64_t)n2 * 16, 256)), dim3(256), 0,
               (const uint32_t *)nbr, (const uint64_t *)row, (const uint64_t *)in, (const uint32_t *)icnt, n2, few, cap, d);
    BYO_CU(ctx, cudaMemcpyAsync(h, d, 80, cudaMemcpyDeviceToHost, ctx->stream));
    BYO_CU(ctx, cudaStreamSynchronize(ctx->stream));
    return BYO_OK;
  };
  BYO_TRY(count_all());
  if (h[9]) {  // edges stored at one end
    uint32_t *ins = nullptr;
    BYO_TRY(ws(g, WS_MS_LEVELS, (g->m + 1) / 2 + 1, (uint64_t **)&ins));
    const uint64_t base = (uint64_t)(((intptr_t)ins - (intptr_t)nbr) / 4);  // both from cudaMalloc
    const dim3 grid(grid_for(ctx, (uint64_t)n2 * 32, 256));
    BYO_CU(ctx, cudaMemsetAsync(icnt, 0, n2 * 4ull, ctx->stream));
    launch(ctx, k_tc_in<false>, grid, dim3(256), 0, nbr, (const uint64_t *)row, n2, (const uint64_t *)in, icnt);
    BYO_TRY(scan_apply(ctx, n2, InU32{icnt}, OutStart{in, base}, &tot));
    BYO_CU(ctx, cudaMemsetAsync(icnt, 0, n2 * 4ull, ctx->stream));
    launch(ctx, k_tc_in<true>, grid, dim3(256), 0, nbr, (const uint64_t *)row, n2, (const uint64_t *)in, icnt);
    BYO_CU(ctx, cudaMemsetAsync(d, 0, 80, ctx->stream));
    BYO_TRY(count_all());
  }
  *count = h[0];
  return check_launch(ctx, "triangle_count");
}

}  // namespace byo
