// wave.cuh — the banded bit-parallel LCS of one pair by a group of 32 or 128
// threads, for launches whose pairs are too few to give every thread its own.
//
// The band is a grid of 32 x 32 blocks (query block i, rep block j).  A chunk
// of W rep blocks belongs to one thread of the group, chunk q to thread
// q mod GS, its W row words in registers; the columns of a query block are
// taken in units of 16.  Thread g works on unit u = t - q of its chunk at
// step t, so that the carries chunk q-1 put out at unit u reach it one step
// later: a systolic wavefront with one shuffle per step (and one shared word
// per warp for groups of 128), instead of a vote over all lanes per column.
// A thread whose chunk has left the band banks its zeros and opens chunk
// q + GS.  Units the thread's chunk does not take part in run with masked
// match words and no carry in, which leaves the rows as they are and puts no
// carry out.
//
// Match words come from a table of the representative in shared memory, one
// row of words per residue code, so that the 32 lanes (consecutive rep
// blocks, any codes) hit 32 banks; the query's codes from a ring of bytes the
// group fills 32 blocks at a time.
//
// What bounds it: a lone warp per scheduler issues its instructions one
// after the other, about three cycles each: nine per column and 80 per step
// of 16 columns; a pair takes 2 nq + nb1 / W steps.  GB300: a 6,600-residue
// protein pair 375 -> 195 us against a form that resolved every column's
// carries over the lanes with two votes, 500 DNA pairs of 1,450 residues
// 100-275 -> 65 us.  Tried: planes in registers instead of the table (370
// us), the columns rolled by four (250), the carry as a value instead of the
// carry flag (231), two row words per thread where one is enough (292), the
// next step's codes loaded ahead (12 mixed jobs 5% slower).  Once every
// scheduler has a warp the instructions count, (80 + 16 (5 + 4 W)) a step for
// 32 W rows of a warp: then a warp per pair with more words (wave_few).
#pragma once
#include <stdint.h>

#include "common.cuh"
#include "dp_asm.cuh"

namespace ngia {

constexpr int kWaveCols = 16, kWaveUnits = 2;  // columns per unit, units per query block
constexpr int kWaveRing = 128;                 // query blocks of codes a group keeps
constexpr int kWaveRingWords = kWaveRing * 8;  // one byte per residue

__host__ __device__ constexpr int wave_codes(int P) { return 1 << P; }               // residue codes the planes can hold
// Words of a match table of max_nb blocks (rows of whole 32-block lines, so
// that the last chunk's missing blocks read zeros).
__host__ __device__ constexpr int wave_stride(int nb) { return (nb + 31) & ~31; }
__host__ __device__ constexpr int wave_table_words(int P, int nb) { return wave_codes(P) * wave_stride(nb); }
// Place of block j's word in its row: 16-byte units of a 128-byte line swapped
// by the line, so that eight lanes reading one unit each of chunks of 8 or 16
// words (32 or 64 bytes apart) find it in eight different bank groups.
__host__ __device__ constexpr int wave_place(int j) { return j ^ (((j >> 5) & 3) << 2); }

// Widest band (blocks a query block covers) a group of GS threads can take
// with W row words per thread when chunks are reused: a thread must have left
// chunk q - 1 + GS alone until its neighbour is through with chunk q.
__host__ __device__ constexpr int wave_cap(int GS, int W) { return W * (GS - 2) + GS / kWaveUnits + 1; }

// Pairs up to which a CTA per pair is faster than a warp per pair, when a group
// per pair is up to `pairs` (56 per SM for a job that has the GPU to itself:
// here one pair per SM, a warp for each scheduler).  GB300, 12 mixed jobs of
// records up to 10,000 residues 47.5 ms with a CTA always; 30.6, 30.4, 30.3,
// 29.7 ms from 4, 2, 1 and 1/2 pairs per SM on; 30,000 proteins at s = 0.5 10.5
// ms, and 9.4, 9.4, 9.2, 9.8.
__host__ __device__ constexpr int wave_few(int pairs) { return pairs / 56; }

// Band of one pair in blocks below and above the diagonal.  With a cutoff,
// only the diagonals a chain of that many matches can touch; false when no
// chain can reach it.
__device__ __forceinline__ bool wave_band(int B, int net1, int net2, int cut, int &lo, int &hi) {
  lo = hi = B;
  if (cut == kNoCut) return true;
  if (net1 < cut || net2 < cut) return false;
  lo = min(B, 1 + ((net2 - cut) >> 5));
  hi = min(B, 1 + ((net1 - cut) >> 5));
  return true;
}

// Builds the match table of a representative (planes rp, nb1 blocks, vlast
// the valid rows of the last) at tab with `threads` threads, t of them;
// the caller synchronises.
template <int P>
__device__ __forceinline__ void wave_table(const uint32_t *rp, int nb1, uint32_t vlast, uint32_t *tab, int t,
                                           int threads) {
  const int stride = wave_stride(nb1);
  for (int j = t; j < stride; j += threads) {
    uint32_t pl[P];
#pragma unroll
    for (int p = 0; p < P; p++) pl[p] = j < nb1 ? rp[j * P + p] : 0u;
    const uint32_t valid = j < nb1 - 1 ? 0xFFFFFFFFu : j == nb1 - 1 ? vlast : 0u;
#pragma unroll
    for (int a = 0; a < wave_codes(P); a++) {
      uint32_t m = valid;
#pragma unroll
      for (int p = 0; p < P; p++) m &= (a >> p) & 1 ? pl[p] : ~pl[p];
      tab[a * stride + wave_place(j)] = m;
    }
  }
}

// The residue codes of one query block (planes pl) as 32 bytes.
template <int P>
__device__ __forceinline__ void wave_unpack(const uint32_t (&pl)[P], uint4 *out) {
  uint32_t v[8];
#pragma unroll
  for (int x = 0; x < 8; x++) {
    v[x] = 0;
#pragma unroll
    for (int c = 0; c < 4; c++)
#pragma unroll
      for (int p = 0; p < P; p++) v[x] |= ((pl[p] >> (4 * x + c)) & 1u) << (8 * c + p);
  }
  out[0] = make_uint4(v[0], v[1], v[2], v[3]);
  out[1] = make_uint4(v[4], v[5], v[6], v[7]);
}

// The W match words of a chunk at row a of the table: off[k] is the byte offset
// of its k-th unit of four words (of its first word, W < 4).
template <int W, int U>
__device__ __forceinline__ void wave_load(uint32_t (&e)[W], const char *tab, uint32_t a, const uint32_t (&off)[U]) {
  if constexpr (W == 1) {
    e[0] = *reinterpret_cast<const uint32_t *>(tab + (a + off[0]));
  } else if constexpr (W == 2) {
    const uint2 v = *reinterpret_cast<const uint2 *>(tab + (a + off[0]));
    e[0] = v.x;
    e[1] = v.y;
  } else {
#pragma unroll
    for (int k = 0; k < U; k++) {
      const uint4 v = *reinterpret_cast<const uint4 *>(tab + (a + off[k]));
      e[4 * k] = v.x;
      e[4 * k + 1] = v.y;
      e[4 * k + 2] = v.z;
      e[4 * k + 3] = v.w;
    }
  }
}

// Zero count of the pair over its band, the same in every thread of the
// group, or -1 once it cannot reach `cut`.  All GS = 32 NW threads call it
// with the same arguments (NW > 1: the whole CTA, xch = 4 NW shared words).
// tab: the representative's match table, ring: the group's code ring (both
// shared, 16-byte aligned), qp: query planes.  B >= 0, nb1 > 0 and nq > 0.
template <int P, int W, int NW>
__device__ __forceinline__ int wave_pair(const uint32_t *tab, int nb1, const uint32_t *qp, int nq, int net2, int lo,
                                         int hi, int cut, uint32_t *ring, uint32_t *xch, unsigned long long &n_done) {
  constexpr int GS = 32 * NW, C = kWaveCols, S = kWaveUnits;
  const int lane = threadIdx.x & 31, warp = NW > 1 ? (int)(threadIdx.x >> 5) : 0;
  const int g = warp * 32 + lane;
  const int q_last = min(nb1 - 1, nq - 1 + hi) / W;
  const uint32_t row_bytes = 4u * (uint32_t)wave_stride(nb1);
  constexpr int U = W > 4 ? W / 4 : 1;
  uint32_t row[W], off[U];
  const char *tabc = reinterpret_cast<const char *>(tab);
  int q = g, u0 = 0, u1 = 0, acc = 0;
  auto open = [&]() {  // chunk q: rows all-ones
    const bool used = q <= q_last;
    u0 = used ? S * max(0, q * W - hi) : 0;
    u1 = used ? min(S * nq, S * (q * W + W + lo)) : 0;
#pragma unroll
    for (int k = 0; k < U; k++) off[k] = used ? 4u * (uint32_t)wave_place(q * W + 4 * k) : 0u;
#pragma unroll
    for (int w = 0; w < W; w++) row[w] = 0xFFFFFFFFu;
  };
  open();
  uint32_t cout = 0, cells = 0;
  int low = 0, low_end = S * (W + lo), filled = 0;  // lowest active chunk, the step it ends at; blocks of codes fetched
  const int steps = S * nq + q_last;
  if constexpr (NW == 1) __syncwarp();  // the group is through with the last pair's ring
  for (int t = 0; t < steps; t++) {
    // The lowest chunk still in the band is furthest along the query, the
    // GS chunks from it at most GS / 2 blocks behind: the next 32 blocks'
    // codes are fetched when it reaches them, over blocks no thread needs.
    if (t >= low_end) {
      low++;
      low_end += S * W + 1;
    }
    if (((t - low) >> 1) >= filled && filled < nq) {
      const int b = filled + g;
      if (g < 32 && b < nq) {
        uint32_t pl[P];
#pragma unroll
        for (int p = 0; p < P; p++) pl[p] = __ldg(qp + b * P + p);
        wave_unpack<P>(pl, reinterpret_cast<uint4 *>(ring) + 2 * (b & (kWaveRing - 1)));
      }
      filled += 32;
      if constexpr (NW == 1) __syncwarp();
    }
    // carries of the chunk below at this unit
    uint32_t cin = __shfl_sync(kFullMask, cout, (lane + 31) & 31);
    if constexpr (NW > 1) {
      if (lane == 31) xch[(t & 1) * NW + warp] = cout;
      if ((t & 7) == 7 && cut != kNoCut) {
        int z = acc;
#pragma unroll
        for (int w = 0; w < W; w++) z += __popc(~row[w]);
        z = __reduce_add_sync(kFullMask, z);
        if (lane == 0) xch[2 * NW + ((t >> 3) & 1) * NW + warp] = (uint32_t)z;
      }
      __syncthreads();
      if (lane == 0) cin = xch[(t & 1) * NW + (warp + NW - 1) % NW];
    }
    if (cut != kNoCut && (t & 7) == 7) {
      // Every row's zeros up to its own unit of the last step bound the
      // longest chain that ends at the top row reached so far, and each
      // column after that row's unit adds at most one.
      int z = 0;
      if constexpr (NW > 1) {
#pragma unroll
        for (int k = 0; k < NW; k++) z += (int)xch[2 * NW + ((t >> 3) & 1) * NW + k];
      } else {
        z = acc;
#pragma unroll
        for (int w = 0; w < W; w++) z += __popc(~row[w]);
        z = __reduce_add_sync(kFullMask, z);
      }
      int top = (t - 1 + S * hi) / (S * W + 1);
      if (top * W <= hi) top = min(t - 1, hi / W);
      top = min(top, q_last);
      if (z + max(0, net2 - C * (t - top)) < cut) {  // the group decides alike
        n_done += cells;
        return -1;
      }
    }
    const int u = t - q, i = u >> 1;
    const bool active = u >= u0 && u < u1;
    const int ncol = active ? max(0, min(C, net2 - C * u)) : 0;
    uint32_t act[W];
    int rows = 0;
#pragma unroll
    for (int w = 0; w < W; w++) {
      const int j = q * W + w;
      const bool in = active && (W == 1 || (j >= i - lo && j <= i + hi));
      act[w] = in ? 0xFFFFFFFFu : 0u;
      rows += in ? 1 : 0;
    }
    cells += (uint32_t)(rows * ncol);
    // idle threads take code 0: the ring's other bytes may be from nowhere
    uint4 codes = make_uint4(0u, 0u, 0u, 0u);
    if (active) codes = reinterpret_cast<const uint4 *>(ring)[2 * (i & (kWaveRing - 1)) + (u & 1)];
    const uint32_t code[4] = {codes.x, codes.y, codes.z, codes.w};
    uint32_t cw = ncol > 0 && q > 0 ? cin << (32 - ncol) : 0u, ncw = 0;
    auto column = [&](uint32_t c) {  // one column of residue code c
      uint32_t e[W];
      wave_load<W, U>(e, tabc, c * row_bytes, off);
      dp_wave<W>(row, e, act, cw, ncw);
    };
    if (t < S * nq - 2 || __all_sync(kFullMask, !active || ncol == C)) {
#pragma unroll(W <= 2 ? C : 4)
      for (int k = 0; k < C; k++) column(__byte_perm(code[k >> 2], 0, 0x4440 | (k & 3)));
    } else {  // the query's last columns
#pragma unroll 1
      for (int k = 0; k < ncol; k++) {
        const uint32_t w = k < 4 ? code[0] : k < 8 ? code[1] : k < 12 ? code[2] : code[3];
        column((w >> (8 * (k & 3))) & 0xFFu);
      }
    }
    cout = ncw;
    if (u >= 0 && u + 1 >= u1 && q <= q_last) {  // the chunk has left the band
#pragma unroll
      for (int w = 0; w < W; w++) acc += __popc(~row[w]);
      q += GS;
      open();
    }
  }
  n_done += cells;
  int sum = __reduce_add_sync(kFullMask, acc);
  if constexpr (NW > 1) {
    __syncthreads();
    if (lane == 0) xch[warp] = (uint32_t)sum;
    __syncthreads();
    sum = 0;
#pragma unroll
    for (int k = 0; k < NW; k++) sum += (int)xch[k];
    __syncthreads();
  }
  return sum;
}

// Whether a group of GS threads with up to W row words each can hold the band.
__host__ __device__ constexpr bool wave_holds(int GS, int W, int lo, int hi, int nb1) {
  return lo + hi + 1 <= wave_cap(GS, W) || nb1 <= GS * W;
}

// The same with the fewest row words per thread (up to WMAX) the band allows;
// a group that holds every rep block at once takes any band.  The caller
// makes sure that WMAX words do.
template <int P, int NW, int WMAX>
__device__ __forceinline__ int wave_any(const uint32_t *tab, int nb1, const uint32_t *qp, int nq, int net2, int lo,
                                        int hi, int cut, uint32_t *ring, uint32_t *xch, unsigned long long &n_done) {
#define NGIA_WAVE(W)                                          \
  if constexpr (W <= WMAX)                                    \
    if (W == WMAX || wave_holds(32 * NW, W, lo, hi, nb1))     \
      return wave_pair<P, W, NW>(tab, nb1, qp, nq, net2, lo, hi, cut, ring, xch, n_done);
  NGIA_WAVE(1) NGIA_WAVE(2) NGIA_WAVE(4) NGIA_WAVE(8) NGIA_WAVE(16)
#undef NGIA_WAVE
  return -1;
}

// ---- several pairs per warp -----------------------------------------------------
// The same wavefront with GS = 8 threads per pair, four pairs per warp, once
// there are more pairs than schedulers: for the windows of common records (up
// to some 50 blocks) a warp per pair has one row word per thread, and 14
// instructions per column and word instead of 5; here W = 8 words per thread
// (4 and 16 for narrower and wider bands) and 2 nq + nb1 / 8 steps.
constexpr int kSubGroup = 8, kSubs = 32 / kSubGroup;
constexpr int kSubRing = 32, kSubFetch = 16;  // query blocks of codes a group keeps, and fetches at a time
constexpr int kSubRingWords = kSubRing * 8;
static_assert(kSubs * kSubRingWords == kWaveRingWords, "the kernels with both forms share the rings");

// Each group's zero count (in all of its threads) or -1 once it cannot reach
// `cut`.  All 32 lanes call it; arguments but tab, nb1 and cut differ by
// group, nq = 0 for a group without a pair; ring: the group's.
template <int P, int W>
__device__ __forceinline__ int wave_sub(const uint32_t *tab, int nb1, const uint32_t *qp, int nq, int net2, int lo,
                                        int hi, int cut, uint32_t *ring, unsigned long long &n_done) {
  constexpr int GS = kSubGroup, C = kWaveCols, S = kWaveUnits, U = W > 4 ? W / 4 : 1;
  const int lane = threadIdx.x & 31, g = lane & (GS - 1);
  const int below = (lane & ~(GS - 1)) | ((g + GS - 1) & (GS - 1));
  const uint32_t row_bytes = 4u * (uint32_t)wave_stride(nb1);
  const char *tabc = reinterpret_cast<const char *>(tab);
  int q_last = nq > 0 ? min(nb1 - 1, nq - 1 + hi) / W : -1;
  uint32_t row[W], off[U];
  int q = g, u0 = 0, u1 = 0, acc = 0;
  auto open = [&]() {  // chunk q: rows all-ones
    const bool used = q <= q_last;
    u0 = used ? S * max(0, q * W - hi) : 0;
    u1 = used ? min(S * nq, S * (q * W + W + lo)) : 0;
#pragma unroll
    for (int k = 0; k < U; k++) off[k] = used ? 4u * (uint32_t)wave_place(q * W + 4 * k) : 0u;
#pragma unroll
    for (int w = 0; w < W; w++) row[w] = 0xFFFFFFFFu;
  };
  open();
  uint32_t cout = 0, cells = 0;
  int low = 0, low_end = S * (W + lo), filled = 0;  // as in wave_pair; the other chunks are at most 4 blocks behind
  bool dead = false;
  const int steps = (int)__reduce_max_sync(kFullMask, (unsigned)(nq > 0 ? S * nq + q_last : 0));
  __syncwarp();  // the warp is through with the last pairs' rings
  for (int t = 0; t < steps; t++) {
    if (t >= low_end) {
      low++;
      low_end += S * W + 1;
    }
    const bool fetch = ((t - low) >> 1) >= filled && filled < nq;
    if (__any_sync(kFullMask, fetch)) {
      if (fetch) {
        for (int b = filled + g; b < min(nq, filled + kSubFetch); b += GS) {
          uint32_t pl[P];
#pragma unroll
          for (int p = 0; p < P; p++) pl[p] = __ldg(qp + b * P + p);
          wave_unpack<P>(pl, reinterpret_cast<uint4 *>(ring) + 2 * (b & (kSubRing - 1)));
        }
        filled += kSubFetch;
      }
      __syncwarp();
    }
    const uint32_t cin = __shfl_sync(kFullMask, cout, below);
    if (cut != kNoCut && (t & 7) == 7) {  // wave_pair's bound, group by group
      int z = acc;
#pragma unroll
      for (int w = 0; w < W; w++) z += __popc(~row[w]);
#pragma unroll
      for (int o = GS / 2; o; o >>= 1) z += __shfl_xor_sync(kFullMask, z, o);
      int top = (t - 1 + S * hi) / (S * W + 1);
      if (top * W <= hi) top = min(t - 1, hi / W);
      top = min(top, q_last);
      dead = dead || nq == 0 || z + max(0, net2 - C * (t - top)) < cut;
      if (__all_sync(kFullMask, dead)) break;
    }
    const int u = t - q, i = u >> 1;
    const bool active = !dead && u >= u0 && u < u1;
    const int ncol = active ? max(0, min(C, net2 - C * u)) : 0;
    uint32_t act[W];
    int rows = 0;
#pragma unroll
    for (int w = 0; w < W; w++) {
      const int j = q * W + w;
      const bool in = active && j >= i - lo && j <= i + hi;
      act[w] = in ? 0xFFFFFFFFu : 0u;
      rows += in ? 1 : 0;
    }
    cells += (uint32_t)(rows * ncol);
    uint4 codes = make_uint4(0u, 0u, 0u, 0u);  // idle threads take code 0
    if (active) codes = reinterpret_cast<const uint4 *>(ring)[2 * (i & (kSubRing - 1)) + (u & 1)];
    const uint32_t code[4] = {codes.x, codes.y, codes.z, codes.w};
    uint32_t cw = ncol > 0 && q > 0 ? cin << (32 - ncol) : 0u, ncw = 0;
    auto column = [&](uint32_t c) {
      uint32_t e[W];
      wave_load<W, U>(e, tabc, c * row_bytes, off);
      dp_wave<W>(row, e, act, cw, ncw);
    };
    if (__all_sync(kFullMask, !active || ncol == C)) {
#pragma unroll 4
      for (int k = 0; k < C; k++) column(__byte_perm(code[k >> 2], 0, 0x4440 | (k & 3)));
    } else {  // some pair's last columns
#pragma unroll 1
      for (int k = 0; k < ncol; k++) {
        const uint32_t w = k < 4 ? code[0] : k < 8 ? code[1] : k < 12 ? code[2] : code[3];
        column((w >> (8 * (k & 3))) & 0xFFu);
      }
    }
    cout = ncw;
    if (u >= 0 && u + 1 >= u1 && q <= q_last) {  // the chunk has left the band
#pragma unroll
      for (int w = 0; w < W; w++) acc += __popc(~row[w]);
      q += GS;
      open();
    }
  }
  n_done += cells;
  int sum = acc;
#pragma unroll
  for (int o = GS / 2; o; o >>= 1) sum += __shfl_xor_sync(kFullMask, sum, o);
  return dead ? -1 : sum;
}

// Pairs above which a warp takes four, when a group per pair is up to `pairs`
// (56 per SM).  other: words of row per thread in the form it replaces: 1 (a
// warp per pair, bands of one word per thread), 4 (a warp, wider), 0 (a CTA).
// GB300, score calls, us with the other form and with 8 threads per pair: DNA
// 1,450 residues 73 and 84 for 1,000 pairs, 93 and 87 for 1,500, 168 and 112 for
// 4,096; protein 380 residues 57 and 58 for 2,500, 71 and 57 for 4,096; DNA 2,600
// residues, a CTA per pair, 142 and 131 for 400, 947 and 243 for 4,096.  Against
// a warp with four words a pair takes three times as long, and 1.4 times fewer
// instructions: a serving batch with 500 to 1,500 such pairs per round 1.42 ms,
// 1.49 with 8 threads.  Proteins with a cut-off stay with a warp: most pairs
// are out after a fifth of their length, and a warp of four runs as long as its
// longest (100,000 proteins, s = 0.9, 8.4 ms, 9.3 with four).
__host__ __device__ constexpr int sub_from(int P, int other, int pairs) {
  return (int)((long long)pairs * (other == 0 ? 3 : other == 4 || P == 5 ? 20 : 9) / 56);
}

// Bands that 8 threads with 16 row words each can hold.
__host__ __device__ constexpr bool sub_holds(int lo, int hi, int nb1) { return wave_holds(kSubGroup, 16, lo, hi, nb1); }

// The same with the fewest row words per thread that hold every group's band;
// the caller makes sure that 16 do.
template <int P>
__device__ __forceinline__ int sub_any(const uint32_t *tab, int nb1, const uint32_t *qp, int nq, int net2, int lo,
                                       int hi, int cut, uint32_t *ring, unsigned long long &n_done) {
  const int n = (int)__reduce_max_sync(kFullMask, (unsigned)(nq > 0 ? lo + hi + 1 : 0));
  if (n <= wave_cap(kSubGroup, 4) || nb1 <= kSubGroup * 4)
    return wave_sub<P, 4>(tab, nb1, qp, nq, net2, lo, hi, cut, ring, n_done);
  if (n <= wave_cap(kSubGroup, 8) || nb1 <= kSubGroup * 8)
    return wave_sub<P, 8>(tab, nb1, qp, nq, net2, lo, hi, cut, ring, n_done);
  return wave_sub<P, 16>(tab, nb1, qp, nq, net2, lo, hi, cut, ring, n_done);
}

// ---- the query's blocks as rows -------------------------------------------------
// Short queries against a long representative: GS = 16 threads per pair, two
// pairs per warp, one query block per thread as its row word, the
// representative's residues as columns.  The band and the recurrence are
// symmetric in the two sequences, so the count is the same; a pair takes
// 2 nb1 + nq steps of two lanes' groups instead of 2 nq + nb1 / W of 128
// threads.  No early rejection: while the representative is long, every
// query residue can still find its match.
// rep_codes: the representative's residue codes, 32 bytes per block (shared
// by the CTA); tab: the warp's match table, one word per code and lane.
// Lanes of a group without a pair pass nq = 0.  Returns the zero count to
// every lane of the pair's group.
constexpr int kQueryGroup = 16;
static_assert(kQueryRows <= kQueryGroup, "a query block per thread");

template <int P>
__device__ __forceinline__ int wave_query(const uint32_t *rep_codes, int nb1, int net1, const uint32_t *qp, int nq,
                                          int net2, int lo, int hi, uint32_t *tab, unsigned long long &n_done) {
  constexpr int C = kWaveCols, S = kWaveUnits;
  const int lane = threadIdx.x & 31, g = lane & (kQueryGroup - 1);
  // row word g: the query's block g; its match words by code
  uint32_t pl[P];
  const bool used = g < nq;
#pragma unroll
  for (int p = 0; p < P; p++) pl[p] = used ? __ldg(qp + g * P + p) : 0u;
  const uint32_t valid = !used ? 0u : g == nq - 1 && (net2 & 31) ? (1u << (net2 & 31)) - 1u : 0xFFFFFFFFu;
  __syncwarp();  // the last pair's table is read
#pragma unroll
  for (int a = 0; a < wave_codes(P); a++) {
    uint32_t m = valid;
#pragma unroll
    for (int p = 0; p < P; p++) m &= (a >> p) & 1 ? pl[p] : ~pl[p];
    tab[32 * a + lane] = m;
  }
  __syncwarp();
  // units of the rep this row takes part in (row block g, rep block i:
  // -lo <= i - g <= hi), and the steps the warp needs
  const int u0 = used ? S * max(0, g - lo) : 0, u1 = used ? min(S * nb1, S * (g + 1 + hi)) : 0;
  const int steps = (int)__reduce_max_sync(kFullMask, (unsigned)(u1 > u0 ? u1 + g : 0));
  uint32_t row[1] = {0xFFFFFFFFu}, cout = 0, cells = 0;
  const char *base = reinterpret_cast<const char *>(tab + lane);
  for (int t = 0; t < steps; t++) {
    const uint32_t cin = __shfl_sync(kFullMask, cout, (lane + 31) & 31);
    const int u = t - g;
    const bool active = u >= u0 && u < u1;
    const int ncol = active ? max(0, min(C, net1 - C * u)) : 0;
    const uint32_t act[1] = {active ? 0xFFFFFFFFu : 0u};
    cells += (uint32_t)ncol;
    uint4 codes = make_uint4(0u, 0u, 0u, 0u);
    if (active) codes = reinterpret_cast<const uint4 *>(rep_codes)[u];
    const uint32_t code[4] = {codes.x, codes.y, codes.z, codes.w};
    uint32_t cw = ncol > 0 && g > 0 ? cin << (32 - ncol) : 0u, ncw = 0;
    auto column = [&](uint32_t c) {
      uint32_t e[1];
      e[0] = *reinterpret_cast<const uint32_t *>(base + c * 128u);
      dp_wave<1>(row, e, act, cw, ncw);
    };
    if (__all_sync(kFullMask, !active || ncol == C)) {
#pragma unroll
      for (int k = 0; k < C; k++) column(__byte_perm(code[k >> 2], 0, 0x4440 | (k & 3)));
    } else {  // the representative's last columns
#pragma unroll 1
      for (int k = 0; k < ncol; k++) {
        const uint32_t w = k < 4 ? code[0] : k < 8 ? code[1] : k < 12 ? code[2] : code[3];
        column((w >> (8 * (k & 3))) & 0xFFu);
      }
    }
    cout = ncw;
  }
  n_done += cells;
  int sum = __popc(~row[0]);
#pragma unroll
  for (int o = kQueryGroup / 2; o; o >>= 1) sum += __shfl_xor_sync(kFullMask, sum, o);
  return sum;
}

}  // namespace ngia
