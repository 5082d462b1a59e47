// seqsum.cuh -- the FP64 sum of a sequence in its order, bit for bit what
// adding the terms one by one gives, computed by a warp or a CTA at a time.
//
// While the sum stays in one binade [2^E, 2^(E+1)) it is a whole number S of
// units u = 2^(E-52), and adding a term x >= 0 adds a whole number: x / u
// rounded to the nearest, a tie to the side that leaves S even.  Without ties
// those increments do not depend on S, so their order does not matter and an
// integer sum replaces the chain of roundings.  A tie depends on the parity of
// S only, so a term is a pair of increments (for an even and an odd S), and
// pairs compose associatively: a scan finds S after every term.  The term
// that takes S to 2^53 or beyond leaves the binade: it is added by __dadd_rn,
// and the rest goes on in the next binade.  Negative terms, -0, infinities,
// NaNs and subnormal sums are added one by one.
//
// An FP64 addition takes 64 cycles before the next of its warp and 19 cycles of
// the SM's FP64 pipe, however many lanes add (measured): a chain of 500 K terms
// takes 17 ms alone, integer units ~0.1.
#pragma once

#include "device.cuh"

namespace byo {

constexpr uint64_t kSeqTop = 1ull << 53;

// 2^-963 <= acc < 2^1023: normal, with a next binade, and so far above the
// subnormals that they add nothing.
__device__ __forceinline__ bool seq_normal(double acc) {
  const uint64_t b = (uint64_t)__double_as_longlong(acc);
  return b >= (60ull << 52) && b < (0x7FEull << 52);
}
__device__ __forceinline__ bool seq_plain(double x) {  // +0, subnormal or normal, not negative
  return (uint32_t)__double2hiint(x) < 0x7FF00000u;
}
// 0 of either sign, by its bits: an FP64 comparison would take the FP64 pipe as
// long as an addition does.
__device__ __forceinline__ bool seq_zero(double acc) { return ((uint64_t)__double_as_longlong(acc) << 1) == 0; }
__device__ __forceinline__ uint64_t seq_units(double acc) {
  return ((uint64_t)__double_as_longlong(acc) & ((1ull << 52) - 1)) | (1ull << 52);
}
__device__ __forceinline__ int seq_exp(double acc) { return (int)((uint64_t)__double_as_longlong(acc) >> 52); }
__device__ __forceinline__ double seq_value(int e, uint64_t units) {
  return __longlong_as_double((long long)(((uint64_t)e << 52) | (units & ((1ull << 52) - 1))));
}

// Units of the binade with biased exponent e (>= 60) that x adds, a tie rounded
// up, and whether it is one; `fits`: x is below 2^E and no special value.  +0 and
// subnormals come out as 0.
__device__ __forceinline__ uint64_t seq_inc(double x, int e, bool &tie, bool &fits) {
  const uint32_t hi = (uint32_t)__double2hiint(x);
  fits = hi < (uint32_t)e << 20;
  const int sh = min(max(e - (int)(hi >> 20), 1), 55);  // past 54 nothing is left
  const uint64_t t = ((uint64_t)((hi & 0xFFFFF) | 0x100000) << 32 | (uint32_t)__double2loint(x)) + (1ull << (sh - 1));
  tie = t << (64 - sh) == 0;
  return t >> sh;
}

// The running sum, the same in every lane; `any`: a term was added; `zero`:
// one was added while the sum was 0 (of either sign).
struct SeqSum {
  double acc;
  bool any, zero;
};

__device__ __forceinline__ void seq_compose(uint64_t p0, uint64_t p1, uint64_t &a0, uint64_t &a1) {
  const uint64_t n0 = p0 + (p0 & 1 ? a1 : a0), n1 = p1 + (p1 & 1 ? a0 : a1);
  a0 = n0;
  a1 = n1;
}
__device__ __forceinline__ void seq_scan(uint64_t &a0, uint64_t &a1) {  // inclusive, over a warp
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t p0 = __shfl_up_sync(kFull, a0, o), p1 = __shfl_up_sync(kFull, a1, o);
    if (lane_id() >= (unsigned)o) seq_compose(p0, p1, a0, a1);
  }
}

// The pair of a thread's terms in a row (those that are not there are +0).
template <int R>
__device__ __forceinline__ void seq_pair(const double (&x)[R], int e, uint64_t &a0, uint64_t &a1) {
  a0 = a1 = 0;
#pragma unroll
  for (int r = 0; r < R; r++) {
    bool tie, fits;
    uint64_t q = seq_inc(x[r], e, tie, fits);
    if (!fits) q = kSeqTop;  // leaves the binade whatever S is
    a0 += q;
    a1 += q;
    if (fits && tie) {  // down again where that makes S even
      a0 -= a0 & 1;
      a1 -= ~a1 & 1;
    }
  }
}

// 256 terms, lane l holding terms 8l .. 8l + 7 (bit r of `in`: it has term
// 8l + r; x[r] is +0 otherwise).  A lane composes its terms' pairs, a scan
// composes the lanes'; the terms of a lane that leaves the binade are added one
// by one, and the lanes after it are scanned again.
__device__ __forceinline__ void seq_warp(SeqSum &s, const double (&x)[8], unsigned in) {
  const unsigned lane = lane_id();
  unsigned todo = __ballot_sync(kFull, in != 0);
  if (!todo) return;
  s.any = true;
  bool plain = true;
#pragma unroll
  for (int r = 0; r < 8; r++) plain = plain && seq_plain(x[r]);
  plain = !__ballot_sync(kFull, !plain);
  while (todo) {
    int k = __ffs(todo) - 1;
    if (plain && seq_normal(s.acc)) {
      const int e = seq_exp(s.acc);
      const uint64_t S = seq_units(s.acc);
      uint64_t a0, a1;
      seq_pair(x, e, a0, a1);
      if (!((todo >> lane) & 1u)) a0 = a1 = 0;
      seq_scan(a0, a1);
      const uint64_t end = S + (S & 1 ? a1 : a0);
      const unsigned out = __ballot_sync(kFull, end >= kSeqTop);
      if (!out) {
        s.acc = seq_value(e, __shfl_sync(kFull, end, 31));
        return;
      }
      k = __ffs(out) - 1;
      const uint64_t before = __shfl_sync(kFull, end, k ? k - 1 : 0);
      if (k) s.acc = seq_value(e, before);
    }
    const unsigned has = __shfl_sync(kFull, in, k);
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const double y = __shfl_sync(kFull, x[r], k);
      if ((has >> r) & 1u) {
        s.zero |= seq_zero(s.acc);
        s.acc = __dadd_rn(s.acc, y);
      }
    }
    todo &= ~((2u << k) - 1u);
  }
}

// Where term i lies in a stage that threads read R consecutive terms from
// (R + 1 apart: no bank conflicts for a power of two).
template <int R>
__host__ __device__ constexpr unsigned seq_at(unsigned i) {
  return i + i / R;
}

// The increments of a thread's terms in any order: false where one is a tie or
// leaves the binade (terms that are not there are +0).
template <int R>
__device__ __forceinline__ bool seq_loose(const double (&x)[R], int e, uint64_t &sum) {
  bool ok = true;
  sum = 0;
#pragma unroll
  for (int r = 0; r < R; r++) {
    bool tie, fits;
    sum += seq_inc(x[r], e, tie, fits);
    ok = ok && fits && !tie;
  }
  return ok;
}

// A CTA's batch of R * blockDim terms, term i = r * blockDim + thread in
// `x[r]` (+0 where bit r of `in` is off): the increments of all of them at once
// in whatever order, or, where that cannot be (a tie, the end of a binade),
// staged so that a thread holds R in a row, composed and scanned over the CTA,
// again after every thread that leaves the binade.  `stage` has room for
// R * blockDim terms (seq_at), `mask` a word for 32 of them; `turn` counts the
// calls.
struct SeqBlockMem {
  double *stage;
  uint32_t *mask;
  uint64_t (*sums)[32];
  SeqSum *shared;
};
// terms [i0, i1) of the stage (multiples of R) one by one
template <int R>
__device__ __forceinline__ void seq_serial(SeqSum &s, const SeqBlockMem &m, unsigned i0, unsigned i1) {
  for (unsigned i = i0; i < i1; i += R) {
    const unsigned has = m.mask[i >> 5] >> (i & 31);
    double y[R];
#pragma unroll
    for (int r = 0; r < R; r++) y[r] = m.stage[seq_at<R>(i + r)];
#pragma unroll
    for (int r = 0; r < R; r++)
      if ((has >> r) & 1u) {
        s.zero |= seq_zero(s.acc);
        s.acc = __dadd_rn(s.acc, y[r]);
      }
  }
}
template <int R>
__device__ __noinline__ SeqSum seq_block_scan(SeqSum s, const SeqBlockMem m) {
  const unsigned t = threadIdx.x, w = t >> 5, lane = lane_id(), nw = blockDim.x >> 5, n = blockDim.x;
  double x[R];
  const unsigned in = (m.mask[R * t >> 5] >> (R * t & 31)) & ((1u << R) - 1u);
  bool plain = true;
#pragma unroll
  for (int r = 0; r < R; r++) {
    x[r] = m.stage[seq_at<R>(R * t + r)];
    plain = plain && seq_plain(x[r]);
  }
  s.any = __syncthreads_or(in != 0) || s.any;
  if (__syncthreads_or(!plain) || !seq_plain(s.acc)) {
    if (t == 0) {
      seq_serial<R>(s, m, 0, R * n);
      *m.shared = s;
    }
    __syncthreads();
    return *m.shared;
  }
  for (unsigned pos = 0; pos < n;) {  // threads below pos are done
    if (!seq_normal(s.acc)) {         // the sum's first terms
      const unsigned to = min(pos + 32 / R, n);
      if (t == 0) {
        seq_serial<R>(s, m, R * pos, R * to);
        *m.shared = s;
      }
      pos = to;
    } else {
      const int e = seq_exp(s.acc);
      const uint64_t S = seq_units(s.acc);
      uint64_t a0, a1;
      seq_pair(x, e, a0, a1);
      if (t < pos) a0 = a1 = 0;
      seq_scan(a0, a1);
      // past 2^53 only the size counts; sums of 32 stay below 2^64
      if (lane == 31) {
        m.sums[0][w] = min(a0, 2 * kSeqTop);
        m.sums[1][w] = min(a1, 2 * kSeqTop);
      }
      __syncthreads();
      uint64_t b0 = lane < nw ? m.sums[0][lane] : 0, b1 = lane < nw ? m.sums[1][lane] : 0;
      seq_scan(b0, b1);
      const uint64_t p0 = w ? __shfl_sync(kFull, b0, w - 1) : 0, p1 = w ? __shfl_sync(kFull, b1, w - 1) : 0;
      seq_compose(p0, p1, a0, a1);
      const uint64_t end = S + (S & 1 ? a1 : a0), up = __shfl_up_sync(kFull, end, 1);
      const unsigned ok = (unsigned)__syncthreads_count(end < kSeqTop);
      if (t == min(ok, n - 1)) {
        if (ok == n) {
          s.acc = seq_value(e, end);
        } else {
          s.acc = seq_value(e, lane ? up : S + (S & 1 ? p1 : p0));
          seq_serial<R>(s, m, R * t, R * t + R);
        }
        *m.shared = s;
      }
      pos = ok + 1;
    }
    __syncthreads();
    s = *m.shared;
    __syncthreads();
  }
  return s;
}
template <int R>
__device__ __forceinline__ void seq_block(SeqSum &s, const double (&x)[R], unsigned in, const SeqBlockMem &m,
                                          unsigned turn) {
  const unsigned w = threadIdx.x >> 5, lane = lane_id(), nw = blockDim.x >> 5;
  const bool normal = seq_normal(s.acc);
  const int e = seq_exp(s.acc);
  uint64_t sum = 0;
  const bool ok = normal && seq_loose(x, e, sum);
  sum = min(warp_sum(sum), kSeqTop);  // the CTA's total stays below 2^64
  const unsigned some = __ballot_sync(kFull, in != 0);
  if (lane == 0) m.sums[turn & 1][w] = sum | (some ? 1ull << 63 : 0);
  if (!__syncthreads_or(ok ? 0 : 1)) {
    const uint64_t part = lane < nw ? m.sums[turn & 1][lane] : 0;
    if (!__ballot_sync(kFull, part >> 63)) return;
    sum = warp_sum(part & ~(1ull << 63)) + seq_units(s.acc);
    if (sum < kSeqTop) {
      s.any = true;
      s.acc = seq_value(e, sum);
      return;
    }
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    const unsigned word = __ballot_sync(kFull, (in >> r) & 1u);
    m.stage[seq_at<R>(r * blockDim.x + threadIdx.x)] = x[r];
    if (lane == 0) m.mask[r * nw + w] = word;
  }
  __syncthreads();
  s = seq_block_scan<R>(s, m);
  __syncthreads();
}

}  // namespace byo
