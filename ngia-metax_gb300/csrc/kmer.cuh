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

// ---- short-word test -------------------------------------------------------------
// A candidate passes when at least `need` of its words are in the
// representative's set (word_min).  Only the answer is wanted, so counting
// stops as soon as it is settled: the count has reached `need`, or the words
// left cannot reach it (an unrelated candidate is settled after about
// (1 - need share) / (1 - set share) of its length).
//
// Lookups are of M overlapping words at once: tab[x] is the number of the M
// words inside the w+M-1 residues x that are in the set, so every M-th position
// is looked up.  A table of bytes in shared memory costs a warp 3 to 4 wavefronts
// a lookup whatever M is (random banks), which bounded the test (GB300, 200,000
// DNA of 1,450 residues, w = 5: 136 us with M = 1 and every word counted).
// Positions q < w-1 have no full word (func.cu:376-396 counts from position
// w-1): the loops count every position with a zero-filled history, and the sum
// starts at minus those first lookups.

// Words per lookup: tables of at most 64 KB (DNA: 8 residues; protein: 3), a
// power of two so that a block of 32 positions is whole lookups.
__host__ __device__ constexpr int words_per_lookup(int type, int w) {
  return type == 0 ? (w <= 5 ? 4 : w <= 7 ? 2 : 1) : (w <= 2 ? 2 : 1);
}
__host__ __device__ inline uint32_t list_words_of(int type, int w) {  // words of the set's bitset
  const uint32_t n = (1u << (w * (type == 0 ? 2 : 5))) / 32u;
  return n ? n : 1u;
}
// Bytes of the table for M words per lookup, and of the 2-word table that the
// 4-word one is made from, behind it.
__host__ __device__ inline uint32_t word_table_bytes(int type, int w, int M) {
  const int bits = type == 0 ? 2 : 5;
  return (1u << (bits * (w + M - 1))) + (M == 4 ? 1u << (bits * (w + 1)) : 0u);
}

// The set's table in shared memory; every thread of the CTA calls it, and the
// table can be read on return.  Four entries (a last residue of 4) per step:
// the words that end before the last residue are common to them.  M = 2 from
// the bitset, M = 4 as the sum of two entries of M = 2 (16,384 steps for w = 5:
// below 2 us of a CTA of 512 threads).
template <int P, int M>
__device__ __forceinline__ void build_word_table(uint8_t *tab, const uint32_t *list, int w) {
  constexpr int bits = P == 2 ? 2 : 5;
  constexpr int kBase = M == 1 ? 1 : 2;
  const uint32_t lmask = (1u << (bits * w)) - 1u;
  uint32_t *base = reinterpret_cast<uint32_t *>(M == 4 ? tab + (1u << (bits * (w + M - 1))) : tab);
  const uint32_t nbase = max(1u, (1u << (bits * (w + kBase - 1))) >> 2);
  for (uint32_t y = threadIdx.x; y < nbase; y += blockDim.x) {
    const uint32_t lo = (4u * y) & lmask;
    const uint32_t nib = (list[lo >> 5] >> (lo & 31)) & 0xFu;
    uint32_t v = (nib & 1u) | ((nib & 2u) << 7) | ((nib & 4u) << 14) | ((nib & 8u) << 21);
    if (kBase == 2) v += KmerBits{list}[y >> (bits - 2)] * 0x01010101u;
    base[y] = v;
  }
  __syncthreads();
  if (M == 4) {
    const uint32_t bmask = (1u << (bits * (w + 1))) - 1u;
    const uint8_t *b8 = reinterpret_cast<const uint8_t *>(base);
    uint32_t *t = reinterpret_cast<uint32_t *>(tab);
    for (uint32_t y = threadIdx.x; y < (1u << (bits * (w + 3))) >> 2; y += blockDim.x)
      t[y] = base[((4u * y) & bmask) >> 2] + b8[(4u * y) >> (2 * bits)] * 0x01010101u;
    __syncthreads();
  }
}

// Residue codes of one protein block (five plane words) as a bit stream, five
// words: residue j's code in bits 155-5j .. 159-5j of the 160-bit value.
__device__ __forceinline__ void protein_stream(const uint32_t (&pl)[5], uint32_t (&st)[5]) {
#pragma unroll
  for (int k = 0; k < 5; k++) st[k] = 0u;
#pragma unroll
  for (int j = 0; j < 32; j++) {
    uint32_t cj = 0;
#pragma unroll
    for (int p = 0; p < 5; p++) cj |= ((pl[p] >> j) & 1u) << p;
    const int t = 155 - 5 * j;  // the code's lowest bit in the 160-bit value
    const int k = 4 - (t >> 5), sh = t & 31;
    st[k] |= cj << sh;
    if (sh > 27) st[k - 1] |= cj >> (32 - sh);  // the group crosses into the word above
  }
}

// A block's code stream, first residue in the highest bits, from its plane
// words (DNA: two words, bits 2(31-j) and 2(31-j)+1 of 64 from planes 0 and 1)
// or, `coded`, as the loader stored it (k_codes).
template <int P>
__device__ __forceinline__ void block_stream(const uint32_t (&r)[P], bool coded, uint32_t (&st)[P]) {
  if constexpr (P == 2) {
    const uint32_t r0 = __brev(r[0]), r1 = __brev(r[1]);
    st[0] = spread16(r0 >> 16) | (spread16(r1 >> 16) << 1);
    st[1] = spread16(r0 & 0xFFFFu) | (spread16(r1 & 0xFFFFu) << 1);
  } else if (coded) {
#pragma unroll
    for (int k = 0; k < 5; k++) st[k] = r[k];
  } else {
    protein_stream(r, st);
  }
}

// The codes that end at residue j of a block, residue j lowest; prev is the
// last stream word of the block before (0 before the first).  One funnel shift.
template <int P>
__device__ __forceinline__ uint32_t codes_word(const uint32_t (&st)[P], uint32_t prev, int j) {
  constexpr int bits = P == 2 ? 2 : 5;
  const int e = bits * (j + 1), k = (e - 1) >> 5;
  return __funnelshift_r(st[k], k ? st[k - 1] : prev, 32 * (k + 1) - e);
}

// Words of the first lim (<= 32) positions of one block that are in the set.
template <int P, int M, class Tab>
__device__ __forceinline__ int block_words(const uint32_t (&st)[P], uint32_t prev, int lim, int w, const Tab &tab,
                                           const uint32_t *list) {
  constexpr int bits = P == 2 ? 2 : 5;
  const uint32_t mask = (1u << (bits * (w + M - 1))) - 1u, lmask = (1u << (bits * w)) - 1u;
  int sum = 0;
  if (lim == 32) {
#pragma unroll
    for (int j = M - 1; j < 32; j += M) sum += tab[codes_word<P>(st, prev, j) & mask];
  } else {
#pragma unroll
    for (int j = 0; j < 32; j++)
      if (j < lim) sum += KmerBits{list}[codes_word<P>(st, prev, j) & lmask];
  }
  return sum;
}

// Lookups of the first w-1 positions of a record (zero history).
template <int P>
__device__ __forceinline__ int head_words(const uint32_t (&st)[P], int net2, int w, const uint32_t *list) {
  constexpr int bits = P == 2 ? 2 : 5;
  const uint32_t lmask = (1u << (bits * w)) - 1u;
  const int head = min(w - 1, net2);
  int sum = 0;
#pragma unroll
  for (int j = 0; j < 7; j++)
    if (j < head) sum += KmerBits{list}[codes_word<P>(st, 0u, j) & lmask];
  return sum;
}

// The short-word test of candidate c by one thread.  G blocks per step, the
// next G loaded while these are counted (a warp's lanes read 32 records: the
// step takes the whole 32-byte sectors they lie in).
template <int P, int M, class Tab>
__device__ __forceinline__ bool words_reach(const DevDB &db, int c, int net2, int w, int need, const Tab &tab,
                                            const uint32_t *list) {
  constexpr int G = P == 2 ? 4 : 2;
  const bool coded = P == 5 && db.codes;
  const uint32_t *rec = (coded ? db.codes : db.words) + __ldg(db.off + c) + db.hw;
  const int nb = (net2 + 31) >> 5;
  uint32_t nx[G][P];
  auto fetch = [&](int b0) {
#pragma unroll
    for (int g = 0; g < G; g++)
#pragma unroll
      for (int p = 0; p < P; p++) nx[g][p] = b0 + g < nb ? __ldg(rec + (b0 + g) * P + p) : 0u;
  };
  fetch(0);
  int sum = 0, left = net2;
  uint32_t prev = 0;
  for (int b0 = 0;; b0 += G) {
    uint32_t cur[G][P];
#pragma unroll
    for (int g = 0; g < G; g++)
#pragma unroll
      for (int p = 0; p < P; p++) cur[g][p] = nx[g][p];
    fetch(b0 + G);
#pragma unroll
    for (int g = 0; g < G; g++) {
      if (left > 0) {
        uint32_t st[P];
        block_stream<P>(cur[g], coded, st);
        if (g == 0 && b0 == 0) sum = -head_words<P>(st, net2, w, list);
        sum += block_words<P, M>(st, prev, min(32, left), w, tab, list);
        left -= min(32, left);
        prev = st[P - 1];
      }
    }
    if (sum >= need) return true;
    if (sum + left < need) return false;
  }
}

// The same by the whole warp: lane l takes blocks l, l+32, ..., a block's
// history from the lane below.  All 32 lanes call it with the same arguments.
template <int P, int M, class Tab>
__device__ __forceinline__ bool words_reach_warp(const DevDB &db, int c, int net2, int w, int need, const Tab &tab,
                                                 const uint32_t *list) {
  const bool coded = P == 5 && db.codes;
  const uint32_t *rec = (coded ? db.codes : db.words) + __ldg(db.off + c) + db.hw;
  const int lane = threadIdx.x & 31;
  const int nb = (net2 + 31) >> 5;
  int sum = 0;
  uint32_t carry = 0;  // last stream word of the block below lane 0's
  uint32_t nx[P];
#pragma unroll
  for (int p = 0; p < P; p++) nx[p] = lane < nb ? __ldg(rec + lane * P + p) : 0u;
  for (int b0 = 0;; b0 += 32) {
    const int b = b0 + lane;
    uint32_t st[P];
    block_stream<P>(nx, coded, st);
#pragma unroll
    for (int p = 0; p < P; p++) nx[p] = b + 32 < nb ? __ldg(rec + (b + 32) * P + p) : 0u;
    uint32_t prev = __shfl_up_sync(kFullMask, st[P - 1], 1);
    if (lane == 0) prev = carry;
    carry = __shfl_sync(kFullMask, st[P - 1], 31);
    const int lim = min(32, net2 - 32 * b);
    int got = 0;
    if (lim > 0) got = block_words<P, M>(st, prev, lim, w, tab, list);
    if (b == 0) got -= head_words<P>(st, net2, w, list);
    sum += __reduce_add_sync(kFullMask, got);
    if (sum >= need) return true;
    if (sum + max(0, net2 - 32 * (b0 + 32)) < need) return false;
  }
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
