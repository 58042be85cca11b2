// kmer.cuh — the per-candidate filter tests shared by the filter (filter.cu)
// and the serving kernels (serve.cu): residue codes, the composition sum and
// the short-word (k-mer) count against a representative's k-mer bitset.
#pragma once
#include <stdint.h>

#include "common.cuh"

namespace ngia {

// Residue code of net position q of a record's planes.
template <int P>
__device__ __forceinline__ uint32_t code_at(const uint32_t *planes, int q) {
  const uint32_t *b = planes + (q >> 5) * P;
  uint32_t c = 0;
#pragma unroll
  for (int p = 0; p < P; p++) c |= ((b[p] >> (q & 31)) & 1u) << p;
  return c;
}

// ---- short-word count of one candidate (kernel_wordFilter job body) ----------
template <int P>
__device__ int word_count(const uint32_t *__restrict__ planes, int net2, int w, const uint32_t *list) {
  constexpr int bits = P == 2 ? 2 : 5;
  const uint32_t mask = (1u << (w * bits)) - 1u;
  uint32_t word = 0;
  int sum = 0;
  for (int i = 0; i < net2; i += 32) {
    uint32_t pl[P];
#pragma unroll
    for (int p = 0; p < P; p++) pl[p] = __ldg(planes + (i >> 5) * P + p);
    const int lim = min(32, net2 - i);
    for (int j = 0; j < lim; j++) {
      uint32_t c = 0;
#pragma unroll
      for (int p = 0; p < P; p++) c |= ((pl[p] >> j) & 1u) << p;
      word = ((word << bits) | c) & mask;
      if (i + j >= w - 1) sum += (list[word >> 5] >> (word & 31)) & 1u;
    }
  }
  return sum;
}

struct KmerBits {
  const uint32_t *w;
  __device__ __forceinline__ uint32_t operator[](uint32_t k) const { return (w[k >> 5] >> (k & 31)) & 1u; }
};

// Bit i of x (i < 16) to bit 2i.
__device__ __forceinline__ uint32_t spread16(uint32_t x) {
  x &= 0xFFFFu;
  x = (x | (x << 8)) & 0x00FF00FFu;
  x = (x | (x << 4)) & 0x0F0F0F0Fu;
  x = (x | (x << 2)) & 0x33333333u;
  x = (x | (x << 1)) & 0x55555555u;
  return x;
}

// ---- fast short-word count -------------------------------------------------------
// tab[word] = 1 if the representative holds the word: a byte table expanded
// in shared memory from the k-mer bitset (filter.cu), or the bitset itself
// (KmerBits: the round filter, whose table changes every few hundred pairs).  Positions q < w-1 have no full word (func.cu:376-396 counts from
// position w-1): the loops below count every position with a zero-filled
// history and then subtract those first w-1 lookups, recomputed the same way.

// 2-bit code stream of one 32-residue DNA block as a 64-bit value (hi:lo),
// earliest residue in the highest bits: residue j's code at bits 2(31-j)
// (plane 0) and 2(31-j)+1 (plane 1).  With the previous block's low word
// above it, the word ending at residue j is the low 2w bits of
// (prev_lo:hi:lo) >> 2(31-j): one funnel shift and one mask.
__device__ __forceinline__ void dna_stream(uint32_t p0, uint32_t p1, uint32_t &hi, uint32_t &lo) {
  const uint32_t r0 = __brev(p0), r1 = __brev(p1);
  hi = spread16(r0 >> 16) | (spread16(r1 >> 16) << 1);
  lo = spread16(r0 & 0xFFFFu) | (spread16(r1 & 0xFFFFu) << 1);
}

// Occurrences of DNA block words in the table: all 32 positions (full) or
// the first lim positions.
template <class Tab>
__device__ __forceinline__ int dna_block_full(uint32_t prev, uint32_t hi, uint32_t lo, uint32_t mask,
                                              const Tab &tab) {
  int sum = 0;
#pragma unroll
  for (int j = 0; j < 16; j++) sum += tab[__funnelshift_r(hi, prev, 30 - 2 * j) & mask];
#pragma unroll
  for (int j = 16; j < 32; j++) sum += tab[__funnelshift_r(lo, hi, 62 - 2 * j) & mask];
  return sum;
}

__device__ __forceinline__ uint32_t dna_word_at(uint32_t prev, uint32_t hi, uint32_t lo, int j) {
  const int sh = 62 - 2 * j;
  return sh >= 32 ? __funnelshift_r(hi, prev, sh - 32) : __funnelshift_r(lo, hi, sh);
}

template <class Tab>
__device__ __forceinline__ int dna_block_part(uint32_t prev, uint32_t hi, uint32_t lo, int lim, uint32_t mask,
                                              const Tab &tab) {
  int sum = 0;
  for (int j = 0; j < lim; j++) sum += tab[dna_word_at(prev, hi, lo, j) & mask];
  return sum;
}

// First w-1 positions of DNA block 0 (zero-filled history), to subtract.
template <class Tab>
__device__ __forceinline__ int dna_head(const uint32_t *planes, int net2, int w, uint32_t mask, const Tab &tab) {
  const int head = min(w - 1, net2);
  if (head <= 0) return 0;
  uint32_t hi, lo;
  dna_stream(__ldg(planes), __ldg(planes + 1), hi, lo);
  int sum = 0;
  for (int j = 0; j < head; j++) sum += tab[dna_word_at(0u, hi, lo, j) & mask];
  return sum;
}

// Code of residue j of a block (P planes).
template <int P>
__device__ __forceinline__ uint32_t code_of(const uint32_t (&pl)[P], int j) {
  uint32_t c = 0;
#pragma unroll
  for (int p = 0; p < P; p++) c |= ((pl[p] >> j) & 1u) << p;
  return c;
}

// Protein: rolling word over the residues of one block.
template <int P, class Tab>
__device__ __forceinline__ int roll_block(const uint32_t (&pl)[P], int lim, uint32_t &word, uint32_t mask,
                                          const Tab &tab) {
  constexpr int bits = P == 2 ? 2 : 5;
  int sum = 0;
  if (lim == 32) {
#pragma unroll
    for (int j = 0; j < 32; j++) {
      word = ((word << bits) | code_of<P>(pl, j)) & mask;
      sum += tab[word];
    }
  } else {
    for (int j = 0; j < lim; j++) {
      word = ((word << bits) | code_of<P>(pl, j)) & mask;
      sum += tab[word];
    }
  }
  return sum;
}

template <int P, class Tab>
__device__ __forceinline__ int roll_head(const uint32_t *planes, int net2, int w, uint32_t mask, const Tab &tab) {
  constexpr int bits = P == 2 ? 2 : 5;
  const int head = min(w - 1, net2);
  if (head <= 0) return 0;
  uint32_t pl[P];
#pragma unroll
  for (int p = 0; p < P; p++) pl[p] = __ldg(planes + p);
  uint32_t word = 0;
  int sum = 0;
  for (int j = 0; j < head; j++) {
    word = ((word << bits) | code_of<P>(pl, j)) & mask;
    sum += tab[word];
  }
  return sum;
}

// Short-word count of one candidate by one thread.
template <int P, class Tab>
__device__ int word_count_fast(const uint32_t *__restrict__ planes, int net2, int w, const Tab &tab) {
  constexpr int bits = P == 2 ? 2 : 5;
  const uint32_t mask = (1u << (w * bits)) - 1u;
  const int nfull = net2 >> 5, rest = net2 & 31;
  int sum = 0;
  if (P == 2) {
    uint32_t prev = 0, hi, lo;
    for (int b = 0; b < nfull; b++) {
      dna_stream(__ldg(planes + 2 * b), __ldg(planes + 2 * b + 1), hi, lo);
      sum += dna_block_full(prev, hi, lo, mask, tab);
      prev = lo;
    }
    if (rest) {
      dna_stream(__ldg(planes + 2 * nfull), __ldg(planes + 2 * nfull + 1), hi, lo);
      sum += dna_block_part(prev, hi, lo, rest, mask, tab);
    }
    return sum - dna_head(planes, net2, w, mask, tab);
  } else {
    uint32_t word = 0;
    for (int b = 0; b <= nfull; b++) {
      const int lim = b < nfull ? 32 : rest;
      if (!lim) break;
      uint32_t pl[P];
#pragma unroll
      for (int p = 0; p < P; p++) pl[p] = __ldg(planes + b * P + p);
      sum += roll_block<P>(pl, lim, word, mask, tab);
    }
    return sum - roll_head<P>(planes, net2, w, mask, tab);
  }
}

// ---- protein short-word count on the residue-code stream (k_codes) -----------
// The w-mer ending at residue j of a block: the 5w bits ending 5(j+1) bits
// below the top of the block's stream words st[], the previous block's last
// word above them (prev; 0 before the first block).  One funnel shift.
__device__ __forceinline__ uint32_t codes_word(const uint32_t (&st)[5], uint32_t prev, int j) {
  const int e = 5 * (j + 1), k = (e - 1) >> 5;
  return __funnelshift_r(st[k], k ? st[k - 1] : prev, 32 * (k + 1) - e);
}

// Lookups of the first lim (<= 32) positions of one block.
template <class Tab>
__device__ __forceinline__ int codes_block(const uint32_t *__restrict__ blk, uint32_t prev, int lim, uint32_t mask,
                                           const Tab &tab, uint32_t &last) {
  uint32_t st[5];
#pragma unroll
  for (int k = 0; k < 5; k++) st[k] = __ldg(blk + k);
  int sum = 0;
  if (lim == 32) {
#pragma unroll
    for (int j = 0; j < 32; j++) sum += tab[codes_word(st, prev, j) & mask];
  } else {
#pragma unroll
    for (int j = 0; j < 32; j++)
      if (j < lim) sum += tab[codes_word(st, prev, j) & mask];
  }
  last = st[4];
  return sum;
}

// The first w-1 positions (zero history), counted by the loops and subtracted.
template <class Tab>
__device__ __forceinline__ int codes_head(const uint32_t *__restrict__ codes, int net2, int w, uint32_t mask,
                                          const Tab &tab) {
  const int head = min(w - 1, net2);
  if (head <= 0) return 0;
  uint32_t st[5];
#pragma unroll
  for (int k = 0; k < 5; k++) st[k] = __ldg(codes + k);
  int sum = 0;
#pragma unroll
  for (int j = 0; j < 7; j++)
    if (j < head) sum += tab[codes_word(st, 0u, j) & mask];
  return sum;
}

// Short-word count of one protein candidate by one thread.
template <class Tab>
__device__ int word_count_codes(const uint32_t *__restrict__ codes, int net2, int w, const Tab &tab) {
  const uint32_t mask = (1u << (5 * w)) - 1u;
  const int nb = (net2 + 31) >> 5;
  uint32_t prev = 0;
  int sum = 0;
  for (int b = 0; b < nb; b++) sum += codes_block(codes + 5 * b, prev, min(32, net2 - 32 * b), mask, tab, prev);
  return sum - codes_head(codes, net2, w, mask, tab);
}

// The same by the whole warp: lane l takes blocks l, l+32, ..., the previous
// block's last stream word from the lane below.  All 32 lanes call it with
// the same arguments.
template <class Tab>
__device__ int word_count_codes_warp(const uint32_t *__restrict__ codes, int net2, int w, const Tab &tab) {
  const uint32_t mask = (1u << (5 * w)) - 1u;
  const int lane = threadIdx.x & 31;
  const int nb = (net2 + 31) >> 5;
  int sum = 0;
  uint32_t carry = 0;  // last stream word of the block below lane 0's
  for (int b0 = 0; b0 < nb; b0 += 32) {
    const int b = b0 + lane;
    const int lim = b < nb ? min(32, net2 - 32 * b) : 0;
    const uint32_t last_mine = b < nb ? __ldg(codes + 5 * b + 4) : 0u;
    uint32_t prev = __shfl_up_sync(kFullMask, last_mine, 1);
    if (lane == 0) prev = carry;
    uint32_t last = 0;
    if (lim > 0) sum += codes_block(codes + 5 * b, prev, lim, mask, tab, last);
    carry = __shfl_sync(kFullMask, last_mine, 31);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(kFullMask, sum, o);
  return sum - codes_head(codes, net2, w, mask, tab);
}

// Short-word count of candidate c by one thread: protein from the code stream
// when the database has one, otherwise from the planes.
template <int P, class Tab>
__device__ __forceinline__ int word_count_cand(const DevDB &db, int c, int net2, int w, const Tab &tab) {
  const int64_t o = __ldg(db.off + c) + db.hw;
  if (P == 5 && db.codes) return word_count_codes(db.codes + o, net2, w, tab);
  return word_count_fast<P>(db.words + o, net2, w, tab);
}

// Short-word count of one candidate by the whole warp against a k-mer
// bitset: lane l takes blocks l, l+32, ...; each block's
// history (the last w-1 residues of the block below) comes from the lane
// below by a shuffle.  Counts positions q >= w-1 (func.cu:376-396).  All 32
// lanes call it with the same arguments.
template <int P>
__device__ int word_count_warp_bits(const uint32_t *__restrict__ planes, int net2, int w, const uint32_t *list) {
  constexpr int bits = P == 2 ? 2 : 5;
  const uint32_t mask = (1u << (w * bits)) - 1u;
  const int lane = threadIdx.x & 31;
  const int nb = (net2 + 31) >> 5;
  int sum = 0;
  uint32_t carry[P];
#pragma unroll
  for (int p = 0; p < P; p++) carry[p] = 0u;
  for (int b0 = 0; b0 < nb; b0 += 32) {
    const int b = b0 + lane;
    const bool have = b < nb;
    const int lim = have ? min(32, net2 - 32 * b) : 0;
    uint32_t pl[P], pv[P];
#pragma unroll
    for (int p = 0; p < P; p++) {
      pl[p] = have ? __ldg(planes + b * P + p) : 0u;
      pv[p] = __shfl_up_sync(kFullMask, pl[p], 1);
      if (lane == 0) pv[p] = carry[p];
    }
    uint32_t word = 0;
    for (int k = 32 - (w - 1); k < 32; k++) {  // history: the block below's last w-1 residues
      uint32_t c = 0;
#pragma unroll
      for (int p = 0; p < P; p++) c |= ((pv[p] >> k) & 1u) << p;
      word = ((word << bits) | c) & mask;
    }
    for (int k = 0; k < lim; k++) {
      uint32_t c = 0;
#pragma unroll
      for (int p = 0; p < P; p++) c |= ((pl[p] >> k) & 1u) << p;
      word = ((word << bits) | c) & mask;
      if (32 * b + k >= w - 1) sum += (list[word >> 5] >> (word & 31)) & 1u;
    }
#pragma unroll
    for (int p = 0; p < P; p++) carry[p] = __shfl_sync(kFullMask, pl[p], 31);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(kFullMask, sum, o);
  return sum;
}

// Composition sum of candidate c against the representative counts rc[].
template <int A>
__device__ __forceinline__ int base_sum(const uint32_t *__restrict__ cnt, int c, const uint32_t *rc) {
  int sum = 0;
  if (A == 4) {
    const uint4 q = __ldg(reinterpret_cast<const uint4 *>(cnt) + c);
    sum = (int)(min(q.x, rc[0]) + min(q.y, rc[1]) + min(q.z, rc[2]) + min(q.w, rc[3]));
  } else {
    const uint4 *q4 = reinterpret_cast<const uint4 *>(cnt + (int64_t)c * 28);
#pragma unroll
    for (int k = 0; k < 7; k++) {
      const uint4 q = __ldg(q4 + k);
      sum += (int)(min(q.x, rc[4 * k]) + min(q.y, rc[4 * k + 1]) + min(q.z, rc[4 * k + 2]) + min(q.w, rc[4 * k + 3]));
    }
  }
  return sum;
}

}  // namespace ngia
