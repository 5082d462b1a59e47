// bytepd.cu -- byte-PD compressed neighbour lists, encoded and decoded on the
// GPU.
//
// The format is the reference's bytepd_amortized encoding
// (gbbs/encodings/byte_pd_amortized.h:1100-1155 writes a vertex,
// byte_pd_amortized.cc:7-55 its integers, the reader's iter at
// byte_pd_amortized.h:180-260) in the compressed graph file of
// gbbs/graph_io.h:351-390 (int64 n, m, total bytes; uint64 byte offsets
// [n+1]; uint32 degrees [n]; the bytes).  A vertex of degree d > 0 holds
// uint32 d, uint32 byte offsets (from the vertex start) of blocks 1 .. nb-1
// (nb = 1 + (d-1)/P), and per block uint32 i*P followed by up to P
// neighbours: the first as a signed difference from the source (first byte:
// bit 7 "more bytes", bit 6 sign, six value bits; then 7 bits per byte), the
// rest as differences to the previous neighbour (7 bits per byte, bit 7
// "more").  The reader's P is PARALLEL_DEGREE = 1000 (gbbs/macros.h:83).
//
// GB300 holds a 2^32-edge CSR in 16 GB, so the graph is decoded once into the
// library's CSR / PMA at load time rather than traversed compressed.
//
// Decode: a group of lanes or a warp per block, an aligned word a lane.  A lane
// assembles the integers that end in its word from it and the word before (an
// integer takes at most 5 bytes), ballots count the ends before it, and a scan of
// the lanes' sums of differences gives the neighbour ids.  Encode: every edge's
// byte length is independent (its difference to the source or the previous
// neighbour); a block's are summed, a scan over the blocks places every block and
// header, and the lengths are scanned again to write the bytes: one word a block
// is kept, where a byte and an 8-byte place an edge were.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <vector>

#include "device.cuh"
#include "internal.h"
#include "scan.cuh"

namespace byo {

constexpr uint32_t kBpdDefaultBlock = 1000;

// The word at byte offset p of an aligned buffer whose last word is whole.
__device__ __forceinline__ uint32_t bpd_u32(const uint32_t *__restrict__ words, uint64_t p) {
  const uint32_t lo = words[p >> 2], hi = words[(p + 3) >> 2];
  return __funnelshift_r(lo, hi, 8 * (uint32_t)(p & 3));
}
__device__ __forceinline__ void bpd_put_u32(unsigned char *p, uint32_t x) {
  p[0] = (unsigned char)x;
  p[1] = (unsigned char)(x >> 8);
  p[2] = (unsigned char)(x >> 16);
  p[3] = (unsigned char)(x >> 24);
}
__device__ __forceinline__ uint32_t bpd_blocks(uint32_t d, uint32_t P) { return d ? 1 + (d - 1) / P : 0; }
__device__ __forceinline__ uint32_t varint_bytes(uint32_t a) {  // 7 bits a byte; 0 takes none
  return (uint32_t)(38 - __clz(a)) / 7;
}

// ---------------------------------------------------------------- decode

struct InBlocks {
  const uint32_t *deg;
  uint32_t P;
  __device__ uint64_t operator()(uint64_t v) const { return bpd_blocks(deg[v], P); }
};

// blk_vertex[first block of v + i] = v
__global__ void k_bpd_block_owner(const uint32_t *__restrict__ deg, uint64_t n, uint32_t P,
                                  const uint64_t *__restrict__ bfirst, uint32_t *blk_vertex) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t b0 = bfirst[v], nb = bfirst[v + 1] - b0;
    for (uint64_t i = 0; i < nb; i++) blk_vertex[b0 + i] = (uint32_t)v;
  }
}

// A block's integers: those after the first, k - done of them at byte offsets
// [p, pend), go to out[done ..]; run is the neighbour before them.
struct BpdRun {
  uint64_t p, pend, out;
  uint32_t k, done, run;
};

// Decodes one run in each group of GS lanes, an aligned word a lane, the groups
// of the warp in step.  Ids are sums modulo 2^32: every difference is below 2^32,
// so a sum that wraps, or a zero, shows as an id not above the one before.
template <int GS>
__device__ __forceinline__ bool bpd_decode_runs(BpdRun x, const uint32_t *__restrict__ words, uint32_t *nbrs) {
  const uint32_t gl = lane_id() % GS, shift = lane_id() & ~(uint32_t)(GS - 1);
  const uint32_t gmask = GS == 32 ? kFull : ((1u << (GS & 31)) - 1), below = (1u << gl) - 1;
  uint32_t last = 0, last2 = 0;  // the two words before the window; 0: four ends
  bool wrong = false;
  for (uint64_t at = (x.p & ~3ull) + 4 * gl; __any_sync(kFull, x.done < x.k); at += 4 * GS) {
    if (x.done < x.k && at - 4 * gl >= x.pend) {  // an integer running past the block
      wrong = true;
      x.k = x.done;
    }
    uint32_t w = 0x80808080u, in = 0;  // in: bit 7 of the block's bytes
    if (x.done < x.k && at < x.pend) {
      w = words[at >> 2];
      in = 0x80808080u;
      if (at + 4 > x.pend) in >>= 8 * (uint32_t)(at + 4 - x.pend);
      if (at < x.p) {  // bytes before the run count as ends
        const uint32_t skip = 8 * (uint32_t)(x.p - at);
        w = w >> skip << skip;
        in = in >> skip << skip;
      }
    }
    uint32_t q = __shfl_up_sync(kFull, w, 1, GS);
    if (gl == 0) q = last;
    uint32_t before = __shfl_up_sync(kFull, q, 1, GS);
    if (gl == 0) before = last2;
    last2 = __shfl_sync(kFull, w, GS - 2, GS);
    last = __shfl_sync(kFull, w, GS - 1, GS);
    const uint32_t ends = ~w & in, need = x.k - x.done;
    uint32_t rank = 0, total = 0;  // ends in the group's lanes before, in all
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t m = __ballot_sync(kFull, (ends >> (8 * j + 7)) & 1u) >> shift & gmask;
      rank += __popc(m & below);
      total += __popc(m);
    }
    // the bytes that q leaves open: its last ones without an end
    const uint32_t open = (uint32_t)__clz(~q & 0x80808080u) >> 3;  // 4 if there is none
    const uint32_t raw = open ? q >> (32 - 8 * open) : 0;
    uint32_t acc = (raw & 0x7fu) | (raw >> 1 & 0x3f80u) | (raw >> 2 & 0x1fc000u) | (raw >> 3 & 0xfe00000u);
    uint32_t sh = 7 * open, sum = 0, upto[4];
    bool over = open == 4 && (before >> 31);  // the first end here ends more than 5 bytes
    const uint32_t mine = rank < need ? need - rank : 0;
    uint32_t seen = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t c = w >> (8 * j);
      over |= sh > 28 || (sh == 28 && (c & 0x70u));  // a sixth byte, or 2^32 and more
      acc |= sh <= 28 ? (c & 0x7fu) << sh : 0;
      sh += 7;
      if ((ends >> (8 * j + 7)) & 1u) {
        wrong |= over && seen < mine;
        sum += acc;
        seen++;
      }
      if (!(c & 0x80u)) {  // an end, or a byte before the run
        acc = 0;
        sh = 0;
        over = false;
      }
      upto[j] = sum;
    }
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < GS; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, inc, o, GS);
      if (gl >= (uint32_t)o) inc += y;
    }
    uint32_t prev = x.run + inc - sum;
    const uint32_t base = prev;
    uint32_t *to = nbrs + x.out + x.done + rank;
    seen = 0;
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (((ends >> (8 * j + 7)) & 1u) && seen < mine) {
        const uint32_t id = base + upto[j];
        wrong |= id <= prev || id == kSentinel;
        to[seen++] = id;
        prev = id;
      }
    x.run += __shfl_sync(kFull, inc, GS - 1, GS);
    x.done += min(total, need);
  }
  return wrong;
}

// bad: 1 malformed run.  A warp takes kBpdTake blocks a step, a lane group each:
// the group reads the headers and the first integer, and runs of up to kBpdShort
// bytes are decoded side by side, the others by the whole warp in turn.  Bound by
// instructions (70% of issue slots): a warp per block had most lanes idle, for half
// the vertices of RMAT 2^20 (2^24 draws) have five neighbours or fewer.  649 -> 350
// us there, uniform 2^20 of degree 32 / 4 and Chung-Lu of degree 6 570 -> 426,
// 213 -> 142, 175 -> 116 (against a warp per block with the same words a lane
// for the first, 4 blocks a step for the others).  4 / 8 / 16 blocks a step: 354 /
// 318 / 315 at 64 bytes; 64 / 96 / 128 bytes at 8 blocks: 318 / 350 / 368, and 561 /
// 426 / 404 on the uniform graph of degree 32.
constexpr int kBpdTake = 8;
constexpr uint64_t kBpdShort = 96;
__global__ void __launch_bounds__(256) k_bpd_decode(const uint32_t *__restrict__ words,
                                                    const uint64_t *__restrict__ bo,
                                                    const uint32_t *__restrict__ deg,
                                                    const uint64_t *__restrict__ off,
                                                    const uint64_t *__restrict__ bfirst,
                                                    const uint32_t *__restrict__ blk_vertex, uint64_t nblocks,
                                                    uint32_t P, uint32_t *nbrs, unsigned int *bad) {
  constexpr int GS = 32 / kBpdTake;
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t group = lane_id() / GS;
  bool wrong = false;
  // blocks in strides: neighbouring ones are as heavy as each other
  for (uint64_t g0 = gw; g0 < nblocks; g0 += kBpdTake * nw) {
    const uint64_t g = g0 + group * nw;
    BpdRun x{0, 0, 0, 0, 0, 0};
    if (g < nblocks) {
      const uint32_t v = blk_vertex[g], d = deg[v], i = (uint32_t)(g - bfirst[v]), nbk = bpd_blocks(d, P);
      const uint64_t vb = bo[v], vlen = bo[v + 1] - vb, hdr = 4ull * nbk;
      bool ok = vlen >= hdr + 4 && bpd_u32(words, vb) == d;
      uint64_t pb = 0, pe = 0, e0 = 0, e1 = 0;
      if (ok) {
        pb = i == 0 ? hdr : bpd_u32(words, vb + 4ull * i);
        pe = i + 1 == nbk ? vlen : bpd_u32(words, vb + 4 + 4ull * i);
        ok = pb + 4 <= pe && pe <= vlen && (i + 1 == nbk || pe + 4 <= vlen);
      }
      if (ok) {
        e0 = bpd_u32(words, vb + pb);
        e1 = i + 1 == nbk ? d : bpd_u32(words, vb + pe);
        ok = e0 <= e1 && e1 <= d;
      }
      if (ok && e1 > e0) {  // the first neighbour: signed, from the source
        x = BpdRun{vb + pb + 4, vb + pe, off[v] + e0, (uint32_t)(e1 - e0), 1, 0};
        const unsigned char *bytes = reinterpret_cast<const unsigned char *>(words);
        uint32_t c = x.p < x.pend ? bytes[x.p++] : 0x80u, sh = 6;
        uint64_t far = c & 0x3fu;
        const bool neg = c & 0x40u;
        while ((c & 0x80u) && x.p < x.pend && sh < 34) {
          c = bytes[x.p++];
          far |= (uint64_t)(c & 0x7fu) << sh;
          sh += 7;
        }
        const int64_t id = neg ? (int64_t)v - (int64_t)far : (int64_t)v + (int64_t)far;
        ok = !(c & 0x80u) && id >= 0 && id < (int64_t)kSentinel;
        x.run = (uint32_t)id;
        if (ok && lane_id() % GS == 0) nbrs[x.out] = x.run;
      }
      if (!ok) {
        wrong = true;
        x.k = x.done = 0;
      }
    }
    const bool wide = x.k > x.done && x.pend - x.p > kBpdShort;
    BpdRun narrow = x;
    if (wide) narrow.k = narrow.done;
    wrong |= bpd_decode_runs<GS>(narrow, words, nbrs);
    for (uint32_t m = __ballot_sync(kFull, wide && lane_id() % GS == 0); m; m &= m - 1) {
      const int o = __ffs(m) - 1;
      const BpdRun y{__shfl_sync(kFull, x.p, o),  __shfl_sync(kFull, x.pend, o), __shfl_sync(kFull, x.out, o),
                     __shfl_sync(kFull, x.k, o), __shfl_sync(kFull, x.done, o), __shfl_sync(kFull, x.run, o)};
      wrong |= bpd_decode_runs<32>(y, words, nbrs);
    }
  }
  if (wrong) atomicOr(bad, 1u);
}

// The blocks of P edges of every vertex: bfirst[v] (its first block, n+1
// entries) and owner[block] = v (both cudaMalloc'd, the caller frees them).
static int block_list(byo_ctx *ctx, uint64_t n, const uint32_t *d_deg, uint32_t P, uint64_t **bfirst_out,
                      uint32_t **owner_out, uint64_t *nblocks) {
  const uint64_t *tot = nullptr;
  uint64_t *bfirst = nullptr;
  uint32_t *owner = nullptr;
  BYO_CU(ctx, cudaMalloc(&bfirst, (n + 1) * 8));
  int rc = scan_apply(ctx, n, InBlocks{d_deg, P}, OutPrefix{bfirst}, &tot);
  uint64_t *h = nullptr;
  if (rc == BYO_OK) rc = pinned(ctx, 4096, (void **)&h);
  if (rc == BYO_OK) {
    cudaMemcpyAsync(bfirst + n, tot, 8, cudaMemcpyDeviceToDevice, ctx->stream);
    cudaMemcpyAsync(h, tot, 8, cudaMemcpyDeviceToHost, ctx->stream);
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) rc = set_error(ctx, BYO_EDEVICE, "byte-PD blocks", e);
  }
  const uint64_t nb = rc == BYO_OK ? h[0] : 0;
  if (rc == BYO_OK) {
    cudaError_t e = cudaMalloc(&owner, (nb ? nb : 1) * 4);
    if (e != cudaSuccess) rc = set_error(ctx, BYO_ENOMEM, "cudaMalloc", e);
  }
  if (rc == BYO_OK)
    launch(ctx, k_bpd_block_owner, dim3(grid_for(ctx, n, 256)), dim3(256), 0, d_deg, n, P, (const uint64_t *)bfirst,
           owner);
  if (rc != BYO_OK) {
    cudaFree(bfirst);
    if (owner) cudaFree(owner);
    return rc;
  }
  *bfirst_out = bfirst;
  *owner_out = owner;
  *nblocks = nb;
  return BYO_OK;
}

int bytepd_decode(byo_ctx *ctx, uint64_t n, const uint64_t *d_bo, const uint32_t *d_deg, const unsigned char *d_bytes,
                  uint32_t P, uint64_t *d_off, uint32_t *d_nbrs) {
  BYO_TRY(scan_u32_to_u64(ctx, d_deg, n, d_off));
  uint64_t *bfirst = nullptr;
  uint32_t *owner = nullptr;
  uint64_t nblocks = 0;
  BYO_TRY(block_list(ctx, n, d_deg, P, &bfirst, &owner, &nblocks));
  unsigned int *bad = nullptr;
  int rc = BYO_OK;
  cudaError_t e0 = cudaMalloc(&bad, 4);
  if (e0 != cudaSuccess) rc = set_error(ctx, BYO_ENOMEM, "cudaMalloc", e0);
  if (rc == BYO_OK) {
    cudaMemsetAsync(bad, 0, 4, ctx->stream);
    launch_t(ctx, "bytepd_decode", k_bpd_decode, dim3(grid_for(ctx, nblocks * 32, 256, 8)), dim3(256), 0,
             reinterpret_cast<const uint32_t *>(d_bytes), d_bo, d_deg, (const uint64_t *)d_off, (const uint64_t *)bfirst, (const uint32_t *)owner, nblocks, P,
             d_nbrs, bad);
    unsigned int hb = 0;
    cudaMemcpyAsync(&hb, bad, 4, cudaMemcpyDeviceToHost, ctx->stream);
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) rc = set_error(ctx, BYO_EDEVICE, "byte-PD decode", e);
    else if (hb) rc = set_error(ctx, BYO_EINVAL, "malformed byte-PD data");
  }
  if (owner) cudaFree(owner);
  if (bad) cudaFree(bad);
  cudaFree(bfirst);
  return rc;
}

// ---------------------------------------------------------------- encode

// The edges [x0, x1) of a block of v; started: v has edges before them.
struct BpdBlock {
  uint64_t x0, x1;
  uint32_t v;
  bool started;
};

// GS of a block's edges from x - lane up: a lane's bytes (0 past the block), and
// what goes into them.  `before` is the neighbour before the GS, of the same list.
struct BpdEdge {
  uint32_t bytes, mag, nbr;  // mag: the difference, for a block's first edge its size
  bool neg, rising;
};
template <int GS>
__device__ __forceinline__ BpdEdge bpd_edge(const BpdBlock &k, const uint32_t *__restrict__ nbrs, uint64_t x,
                                            uint32_t before) {
  BpdEdge r;
  r.nbr = x < k.x1 ? nbrs[x] : 0;
  uint32_t prev = __shfl_up_sync(kFull, r.nbr, 1, GS);
  if (lane_id() % GS == 0) prev = before;
  r.rising = x >= k.x1 || r.nbr > prev || (x == k.x0 && !k.started);
  r.neg = false;
  r.mag = 0;
  r.bytes = 0;
  if (x < k.x1) {
    if (x == k.x0) {
      r.neg = r.nbr < k.v;
      r.mag = r.neg ? k.v - r.nbr : r.nbr - k.v;
      r.bytes = 1 + varint_bytes(r.mag >> 6);
    } else {
      r.mag = r.nbr - prev;
      r.bytes = varint_bytes(r.mag);
    }
  }
  return r;
}

// A block in each group of GS lanes, the groups of the warp in step: its integers'
// bytes (in the group's first lane), and whether its neighbours increase.
template <int GS>
__device__ __forceinline__ uint64_t bpd_size_runs(const BpdBlock &k, const uint32_t *__restrict__ nbrs, bool &rising) {
  uint32_t before = k.started && k.x0 < k.x1 ? nbrs[k.x0 - 1] : 0;
  uint64_t mine = 0;
  for (uint64_t xb = k.x0; __any_sync(kFull, xb < k.x1); xb += GS) {
    const BpdEdge r = bpd_edge<GS>(k, nbrs, xb + lane_id() % GS, before);
    before = __shfl_sync(kFull, r.nbr, GS - 1, GS);
    mine += r.bytes;
    rising = rising && r.rising;
  }
#pragma unroll
  for (int o = GS / 2; o > 0; o >>= 1) mine += __shfl_down_sync(kFull, mine, o, GS);
  return mine;
}
// The same for writing: the integers of a block go to bytes[at ..].
template <int GS>
__device__ __forceinline__ void bpd_write_runs(const BpdBlock &k, const uint32_t *__restrict__ nbrs, uint64_t at,
                                               unsigned char *bytes) {
  const uint32_t gl = lane_id() % GS;
  unsigned char *to = bytes + at;
  uint32_t before = 0;
  for (uint64_t xb = k.x0; __any_sync(kFull, xb < k.x1); xb += GS) {
    const BpdEdge r = bpd_edge<GS>(k, nbrs, xb + gl, before);
    before = __shfl_sync(kFull, r.nbr, GS - 1, GS);
    uint32_t inc = r.bytes;
#pragma unroll
    for (int o = 1; o < GS; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, inc, o, GS);
      if (gl >= (uint32_t)o) inc += y;
    }
    unsigned char *w = to + (inc - r.bytes);
    uint32_t a = r.mag, left = r.bytes;
    if (xb + gl == k.x0 && left) {
      *w++ = (unsigned char)((a & 0x3f) | (r.neg ? 0x40 : 0) | (left > 1 ? 0x80 : 0));
      a >>= 6;
      left--;
    }
#pragma unroll
    for (uint32_t j = 0; j < 5; j++)
      if (j < left) w[j] = (unsigned char)((a >> (7 * j) & 0x7f) | (j + 1 < left ? 0x80 : 0));
    to += __shfl_sync(kFull, inc, GS - 1, GS);
  }
}

// Blocks of up to kBpdFew edges are encoded side by side, kBpdTake to a warp, as
// k_bpd_decode's short runs are; the others by the whole warp in turn.  RMAT 2^20
// (2^24 draws): sizes 213 -> 179 us, writing 344 -> 296; the uniform graph of degree 32
// 250 -> 127 and 406 -> 359.
constexpr uint64_t kBpdFew = 48;
__device__ __forceinline__ BpdBlock bpd_block_from(const BpdBlock &k, int o) {
  return BpdBlock{__shfl_sync(kFull, k.x0, o), __shfl_sync(kFull, k.x1, o), __shfl_sync(kFull, k.v, o),
                  __shfl_sync(kFull, (int)k.started, o) != 0};
}

// Bytes of each block's integers; bad |= 1 for a list that is not strictly
// increasing.
__global__ void __launch_bounds__(256) k_bpd_size(const uint64_t *__restrict__ off, const uint32_t *__restrict__ nbrs,
                                                  uint32_t P, const uint64_t *__restrict__ bfirst,
                                                  const uint32_t *__restrict__ blk_vertex, uint64_t nblocks,
                                                  uint64_t *size, unsigned int *bad) {
  constexpr int GS = 32 / kBpdTake;
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  bool rising = true;
  for (uint64_t g0 = gw; g0 < nblocks; g0 += kBpdTake * nw) {
    const uint64_t g = g0 + lane_id() / GS * nw;
    BpdBlock k{0, 0, 0, false};
    if (g < nblocks) {
      k.v = blk_vertex[g];
      const uint64_t b = off[k.v], e = off[k.v + 1];
      k.x0 = b + (g - bfirst[k.v]) * P;
      k.x1 = k.x0 + P < e ? k.x0 + P : e;
      k.started = k.x0 > b;
    }
    const bool wide = k.x1 - k.x0 > kBpdFew;
    BpdBlock few = k;
    if (wide) few.x1 = few.x0;
    const uint64_t bytes = bpd_size_runs<GS>(few, nbrs, rising);
    if (lane_id() % GS == 0 && g < nblocks && !wide) size[g] = bytes;
    for (uint32_t m = __ballot_sync(kFull, wide && lane_id() % GS == 0); m; m &= m - 1) {
      const int o = __ffs(m) - 1;
      const uint64_t all = bpd_size_runs<32>(bpd_block_from(k, o), nbrs, rising);
      if (lane_id() == 0) size[g0 + o / GS * nw] = all;
    }
  }
  if (!rising) atomicOr(bad, 1u);
}

// bytes of vertex v: headers plus its blocks' bytes (bpos is their prefix)
struct InVertexBytes {
  const uint64_t *off, *bfirst, *bpos;
  uint32_t P;
  __device__ uint64_t operator()(uint64_t v) const {
    const uint64_t d = off[v + 1] - off[v];
    if (!d) return 0;
    const uint32_t nb = bpd_blocks((uint32_t)d, P);
    return 4 + 4ull * (nb - 1) + 4ull * nb + (bpos[bfirst[v + 1]] - bpos[bfirst[v]]);
  }
};

// Every block's header (and, for block 0, the vertex's degree) and its edges'
// bytes, placed by a scan of their lengths.
__global__ void __launch_bounds__(256) k_bpd_write(const uint64_t *__restrict__ off, const uint32_t *__restrict__ nbrs,
                                                   uint32_t P, const uint64_t *__restrict__ bfirst,
                                                   const uint32_t *__restrict__ blk_vertex, uint64_t nblocks,
                                                   const uint64_t *__restrict__ bpos, const uint64_t *__restrict__ bo,
                                                   unsigned char *bytes) {
  constexpr int GS = 32 / kBpdTake;
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t g0 = gw; g0 < nblocks; g0 += kBpdTake * nw) {
    const uint64_t g = g0 + lane_id() / GS * nw;
    BpdBlock k{0, 0, 0, false};
    uint64_t at = 0;  // the block's first edge byte
    if (g < nblocks) {
      k.v = blk_vertex[g];
      const uint64_t b = off[k.v], e = off[k.v + 1], blk = g - bfirst[k.v];
      const uint32_t nb = bpd_blocks((uint32_t)(e - b), P);
      const uint64_t base = bo[k.v], q0 = 4ull * nb + 4 * (blk + 1) + (bpos[g] - bpos[g - blk]);
      k.x0 = b + blk * P;
      k.x1 = k.x0 + P < e ? k.x0 + P : e;
      at = base + q0;
      if (lane_id() % GS == 0) {
        if (blk == 0) bpd_put_u32(bytes + base, (uint32_t)(e - b));
        else bpd_put_u32(bytes + base + 4 * blk, (uint32_t)(q0 - 4));
        bpd_put_u32(bytes + at - 4, (uint32_t)(blk * P));
      }
    }
    const bool wide = k.x1 - k.x0 > kBpdFew;
    BpdBlock few = k;
    if (wide) few.x1 = few.x0;
    bpd_write_runs<GS>(few, nbrs, at, bytes);
    for (uint32_t m = __ballot_sync(kFull, wide && lane_id() % GS == 0); m; m &= m - 1) {
      const int o = __ffs(m) - 1;
      bpd_write_runs<32>(bpd_block_from(k, o), nbrs, __shfl_sync(kFull, at, o), bytes);
    }
  }
}

// Encodes the device CSR of g (its snapshot for a PMA); the device byte
// offsets bo[n+1] and bytes are returned in *d_bo / *d_bytes (cudaMalloc'd,
// the caller frees them).
int bytepd_encode(byo_graph *g, uint32_t P, uint64_t **d_bo_out, unsigned char **d_bytes_out, uint64_t *nbytes) {
  byo_ctx *ctx = g->ctx;
  byo_graph *t = nullptr;
  BYO_TRY(traversal_view(g, &t));
  const uint64_t n = t->n;
  *d_bo_out = nullptr;
  *d_bytes_out = nullptr;
  uint64_t *size = nullptr, *bo = nullptr;
  unsigned char *bytes = nullptr;
  unsigned int *bad = nullptr;
  int rc = BYO_OK;
  cudaError_t e = cudaMalloc(&bo, (n + 1) * 8);
  if (e == cudaSuccess) e = cudaMalloc(&bad, 4);
  if (e != cudaSuccess) rc = set_error(ctx, BYO_ENOMEM, "cudaMalloc", e);
  uint64_t *h = nullptr;
  if (rc == BYO_OK) rc = pinned(ctx, 4096, (void **)&h);
  uint64_t *bfirst = nullptr;
  uint32_t *owner = nullptr;
  uint64_t nblocks = 0;
  if (rc == BYO_OK) rc = block_list(ctx, n, t->d_deg, P, &bfirst, &owner, &nblocks);
  if (rc == BYO_OK && (e = cudaMalloc(&size, (2 * nblocks + 1) * 8)) != cudaSuccess)
    rc = set_error(ctx, BYO_ENOMEM, "cudaMalloc", e);
  uint64_t *bpos = size + nblocks;
  if (rc == BYO_OK) {
    cudaMemsetAsync(bad, 0, 4, ctx->stream);
    launch(ctx, k_bpd_size, dim3(grid_for(ctx, nblocks * 32, 256, 8)), dim3(256), 0, (const uint64_t *)t->d_off,
           (const uint32_t *)t->d_slots, P, (const uint64_t *)bfirst, (const uint32_t *)owner, nblocks, size, bad);
    const uint64_t *tot = nullptr;
    rc = scan_apply(ctx, nblocks, InU64{size}, OutPrefix{bpos}, &tot);
    if (rc == BYO_OK) {
      cudaMemcpyAsync(bpos + nblocks, tot, 8, cudaMemcpyDeviceToDevice, ctx->stream);
      rc = scan_apply(ctx, n, InVertexBytes{t->d_off, bfirst, bpos, P}, OutPrefix{bo}, &tot);
    }
    if (rc == BYO_OK) {
      cudaMemcpyAsync(bo + n, tot, 8, cudaMemcpyDeviceToDevice, ctx->stream);
      cudaMemcpyAsync(h, tot, 8, cudaMemcpyDeviceToHost, ctx->stream);
      cudaMemcpyAsync(h + 1, bad, 4, cudaMemcpyDeviceToHost, ctx->stream);
      e = cudaStreamSynchronize(ctx->stream);
      if (e != cudaSuccess) rc = set_error(ctx, BYO_EDEVICE, "byte-PD sizes", e);
      else if ((uint32_t)h[1]) rc = set_error(ctx, BYO_EINVAL, "byte-PD: adjacency not strictly increasing");
    }
  }
  const uint64_t total = rc == BYO_OK ? h[0] : 0;
  if (rc == BYO_OK && (e = cudaMalloc(&bytes, total ? total : 1)) != cudaSuccess)
    rc = set_error(ctx, BYO_ENOMEM, "cudaMalloc", e);
  if (rc == BYO_OK) {
    launch_t(ctx, "bytepd_encode", k_bpd_write, dim3(grid_for(ctx, nblocks * 32, 256, 8)), dim3(256), 0,
             (const uint64_t *)t->d_off, (const uint32_t *)t->d_slots, P, (const uint64_t *)bfirst,
             (const uint32_t *)owner, nblocks, (const uint64_t *)bpos, (const uint64_t *)bo, bytes);
    rc = check_launch(ctx, "bytepd_encode");
  }
  if (bfirst) cudaFree(bfirst);
  if (owner) cudaFree(owner);
  if (size) cudaFree(size);
  if (bad) cudaFree(bad);
  if (rc != BYO_OK) {
    if (bo) cudaFree(bo);
    if (bytes) cudaFree(bytes);
    return rc;
  }
  *d_bo_out = bo;
  *d_bytes_out = bytes;
  *nbytes = total;
  return BYO_OK;
}

// ---------------------------------------------------------------- host side

int graph_from_bytepd_host(byo_ctx *ctx, uint64_t n, const uint64_t *h_bo, const uint32_t *h_deg,
                           const unsigned char *h_bytes, uint64_t nbytes, uint32_t P, int container,
                           byo_graph **out) {
  if (n >= 0xFFFFFFFFull) return set_error(ctx, BYO_EINVAL, "n must be < 2^32 - 1");
  if (!h_bo || (n && !h_deg) || (nbytes && !h_bytes)) return set_error(ctx, BYO_EINVAL, "null byte-PD array");
  if (h_bo[0] != 0 || h_bo[n] > nbytes) return set_error(ctx, BYO_EINVAL, "byte-PD offsets outside the bytes");
  uint64_t m = 0;
  bool drops = false;
  for (uint64_t v = 0; v < n; v++) drops |= h_bo[v + 1] < h_bo[v];
  for (uint64_t v = 0; v < n; v++) m += h_deg[v];
  if (drops) return set_error(ctx, BYO_EINVAL, "byte-PD offsets decrease");
  uint64_t *d_bo = nullptr, *d_off = nullptr;
  uint32_t *d_deg = nullptr, *d_nbrs = nullptr;
  unsigned char *d_bytes = nullptr;
  int rc = BYO_OK;
  cudaError_t e = cudaMalloc(&d_bo, (n + 1) * 8);
  if (e == cudaSuccess) e = cudaMalloc(&d_deg, (n ? n : 1) * 4);
  if (e == cudaSuccess) e = cudaMalloc(&d_bytes, (nbytes / 4 + 1) * 4);  // whole words: k_bpd_decode
  if (e == cudaSuccess) e = cudaMalloc(&d_off, (n + 1) * 8);
  if (e == cudaSuccess) e = cudaMalloc(&d_nbrs, (m + 16) * 4);
  if (e != cudaSuccess) rc = set_error(ctx, BYO_ENOMEM, "cudaMalloc", e);
  if (rc == BYO_OK) {
    cudaMemcpyAsync(d_bo, h_bo, (n + 1) * 8, cudaMemcpyHostToDevice, ctx->stream);
    if (n) cudaMemcpyAsync(d_deg, h_deg, n * 4, cudaMemcpyHostToDevice, ctx->stream);
    if (nbytes) cudaMemcpyAsync(d_bytes, h_bytes, nbytes, cudaMemcpyHostToDevice, ctx->stream);
    rc = bytepd_decode(ctx, n, d_bo, d_deg, d_bytes, P, d_off, d_nbrs);
  }
  if (rc == BYO_OK) rc = graph_from_device_csr(ctx, container, n, m, &d_off, &d_nbrs, &d_deg, out);
  for (void *p : {(void *)d_bo, (void *)d_deg, (void *)d_bytes, (void *)d_off, (void *)d_nbrs})
    if (p) cudaFree(p);
  return rc;
}

int bytepd_read_file(byo_ctx *ctx, const char *path, uint32_t P, int container, byo_graph **out) {
  FILE *f = std::fopen(path, "rb");
  if (!f) return set_error(ctx, BYO_EINVAL, "byte-PD file: cannot open");
  int64_t hdr[3];
  int rc = BYO_OK;
  std::vector<uint64_t> bo;
  std::vector<uint32_t> deg;
  std::vector<unsigned char> bytes;
  if (std::fread(hdr, 8, 3, f) != 3 || hdr[0] < 0 || hdr[1] < 0 || hdr[2] < 0) {
    rc = set_error(ctx, BYO_EINVAL, "byte-PD file: short header");
  } else if ((uint64_t)hdr[0] >= 0xFFFFFFFFull) {
    rc = set_error(ctx, BYO_EINVAL, "byte-PD file: n does not fit 32-bit ids");
  } else {
    const uint64_t n = (uint64_t)hdr[0], nbytes = (uint64_t)hdr[2];
    bo.resize(n + 1);
    deg.resize(n ? n : 1);
    bytes.resize(nbytes ? nbytes : 1);
    if (std::fread(bo.data(), 8, n + 1, f) != n + 1 || (n && std::fread(deg.data(), 4, n, f) != n) ||
        (nbytes && std::fread(bytes.data(), 1, nbytes, f) != nbytes))
      rc = set_error(ctx, BYO_EINVAL, "byte-PD file: body shorter than the header says");
  }
  std::fclose(f);
  BYO_TRY(rc);
  const uint64_t n = (uint64_t)hdr[0];
  uint64_t m = 0;
  for (uint64_t v = 0; v < n; v++) m += deg[v];
  if (m != (uint64_t)hdr[1]) return set_error(ctx, BYO_EINVAL, "byte-PD file: degrees do not sum to m");
  return graph_from_bytepd_host(ctx, n, bo.data(), deg.data(), bytes.data(), (uint64_t)hdr[2], P, container, out);
}

int bytepd_write_file(byo_graph *g, const char *path, uint32_t P) {
  byo_ctx *ctx = g->ctx;
  uint64_t *d_bo = nullptr;
  unsigned char *d_bytes = nullptr;
  uint64_t nbytes = 0;
  BYO_TRY(bytepd_encode(g, P, &d_bo, &d_bytes, &nbytes));
  const uint64_t n = g->n;
  std::vector<uint64_t> bo(n + 1);
  std::vector<uint32_t> deg(n ? n : 1);
  std::vector<unsigned char> bytes(nbytes ? nbytes : 1);
  byo_graph *t = nullptr;
  int rc = traversal_view(g, &t);
  if (rc == BYO_OK) {
    cudaMemcpyAsync(bo.data(), d_bo, (n + 1) * 8, cudaMemcpyDeviceToHost, ctx->stream);
    if (n) cudaMemcpyAsync(deg.data(), t->d_deg, n * 4, cudaMemcpyDeviceToHost, ctx->stream);
    if (nbytes) cudaMemcpyAsync(bytes.data(), d_bytes, nbytes, cudaMemcpyDeviceToHost, ctx->stream);
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) rc = set_error(ctx, BYO_EDEVICE, "byte-PD download", e);
  }
  cudaFree(d_bo);
  cudaFree(d_bytes);
  BYO_TRY(rc);
  FILE *f = std::fopen(path, "wb");
  if (!f) return set_error(ctx, BYO_EINVAL, "byte-PD file: cannot create");
  const int64_t hdr[3] = {(int64_t)n, (int64_t)g->m, (int64_t)nbytes};
  bool ok = std::fwrite(hdr, 8, 3, f) == 3 && std::fwrite(bo.data(), 8, n + 1, f) == n + 1 &&
            (n == 0 || std::fwrite(deg.data(), 4, n, f) == n) &&
            (nbytes == 0 || std::fwrite(bytes.data(), 1, nbytes, f) == nbytes);
  ok = (std::fclose(f) == 0) && ok;
  return ok ? BYO_OK : set_error(ctx, BYO_EINVAL, "byte-PD file: write failed");
}

int bytepd_encode_host(byo_graph *g, uint32_t P, uint64_t *h_bo, uint32_t *h_deg, unsigned char *h_bytes,
                       uint64_t *nbytes) {
  byo_ctx *ctx = g->ctx;
  uint64_t *d_bo = nullptr;
  unsigned char *d_bytes = nullptr;
  uint64_t total = 0;
  BYO_TRY(bytepd_encode(g, P, &d_bo, &d_bytes, &total));
  int rc = BYO_OK;
  const uint64_t cap = *nbytes;
  *nbytes = total;
  if (h_bytes && cap < total) rc = set_error(ctx, BYO_EINVAL, "byte-PD: output buffer too small");
  byo_graph *t = nullptr;
  if (rc == BYO_OK) rc = traversal_view(g, &t);
  if (rc == BYO_OK) {
    if (h_bo) cudaMemcpyAsync(h_bo, d_bo, (g->n + 1) * 8, cudaMemcpyDeviceToHost, ctx->stream);
    if (h_deg && g->n) cudaMemcpyAsync(h_deg, t->d_deg, g->n * 4, cudaMemcpyDeviceToHost, ctx->stream);
    if (h_bytes && total) cudaMemcpyAsync(h_bytes, d_bytes, total, cudaMemcpyDeviceToHost, ctx->stream);
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) rc = set_error(ctx, BYO_EDEVICE, "byte-PD download", e);
  }
  cudaFree(d_bo);
  cudaFree(d_bytes);
  return rc;
}

}  // namespace byo
