// tile.cuh — the register-tile update of the banded bit-parallel LCS shared
// by the alignment kernels (align.cu) and the serving kernels (serve.cu):
// band-row rings, one tile of rep blocks over the columns of a query block,
// and the build-time tuning of the tiled kernel.
#pragma once
#include <stdint.h>

#include "common.cuh"
#include "dp_asm.cuh"
#include "kmer.cuh"

// Build-time tuning of the DNA alignment kernels (swept on GB300, 1M DNA):
//  NGIA_TILED_MAIN_DNA / NGIA_TILED_BLOCKS_DNA  main tile width and resident
//    CTAs per SM of the tiled kernel.
//  NGIA_EQ_PF_MAIN  load the next column's match words during the current
//    column in the main tiles of the clustering kernel.
//  NGIA_SERVE_PF  the same in the kernel that takes the representative per
//    pair: off (60.2k against 64.3k queries/s).
//  Settled before the window followed the pair (band_advance), on windows of
//  49 blocks: match words from the representative's table instead of plane
//  registers +16%; columns unrolled 2/4/8 times 0.92x/0.64x/0.41x
//  (instruction cache); code, address and carry bookkeeping as multiply-adds
//  by run-time constants (FMA pipe) +2.9%; adds as IMAD.X 0.97x; straight
//  tiles +3%.
#ifndef NGIA_TILED_MAIN_DNA
#define NGIA_TILED_MAIN_DNA 16
#endif
#ifndef NGIA_TILED_BLOCKS_DNA
#define NGIA_TILED_BLOCKS_DNA 4
#endif
#ifndef NGIA_EQ_PF_MAIN
#define NGIA_EQ_PF_MAIN 1
#endif
#ifndef NGIA_SERVE_PF
#define NGIA_SERVE_PF 0
#endif
// Remainder tiles: rounded up to a multiple of this many slots.  Two: windows
// that follow their pair end at any width, and half as many tile bodies miss
// less in the instruction cache (20,000 DNA to the end 286 -> 250 ms, four
// 258 ms; 400k DNA, 12 iterations 27.3 -> 24.4, four 25.4).
#ifndef NGIA_REM_ROUND
#define NGIA_REM_ROUND 2
#endif

namespace ngia {

constexpr int kAlignThreads = 128;  // threads per CTA of every alignment kernel

// Band rows of one lane's pair, indexed by absolute rep block j.  Windows of
// up to RING blocks keep them in shared memory (row j of thread t at
// (j mod RING) * threads + t: the 32 lanes of a warp hit 32 banks); wider
// windows keep them in global scratch with the same layout over all lanes
// of the grid (a warp's accesses to one row are one 128-byte line).
template <int RING>
struct SmemRing {
  static constexpr int kSize = RING;
  uint32_t *base;  // ring + threadIdx.x
  __device__ __forceinline__ uint32_t &operator[](int j) const { return base[(j & (RING - 1)) * kAlignThreads]; }
  __device__ __forceinline__ uint32_t *at(int j) const { return base + (j & (RING - 1)) * kAlignThreads; }
};
struct GlobalRing {
  static constexpr int kSize = 0;  // no straight-tile path
  __device__ __forceinline__ uint32_t *at(int) const { return nullptr; }
  uint32_t *base;  // scratch + global lane index
  uint32_t mask;   // ring size - 1 (a power of two >= the widest window)
  int64_t stride;  // lanes of the grid
  __device__ __forceinline__ uint32_t &operator[](int j) const { return base[(int64_t)(j & mask) * stride]; }
};
template <int RING>
struct RingOf {
  using T = SmemRing<RING>;
};
template <>
struct RingOf<0> {
  using T = GlobalRing;
};

// One tile: band rows base .. base+TW-1 (rows above je are padding) through
// the `cols` columns of the current query block, whose P plane words are
// cur[]; s_pl points at the representative's planes (shared or global
// memory).  cw holds the column carries into the tile (column k at bit
// 31-k after the shift below), ncw collects the carries out.  Returns the
// change of the zero count over the tile's rows.
template <int P, int TW, class Ring>
__device__ __forceinline__ int tiled_tile(const Ring &ring, const uint32_t *s_pl, int base, int je, int cols,
                                          const uint32_t (&cur)[P], uint32_t &cw, uint32_t &ncw) {
  uint32_t row[TW], pl[P][TW];
  int zold = 0;
#pragma unroll
  for (int m = 0; m < TW; m++) {
    const int j = base + m;
    const bool in = j <= je;
    row[m] = in ? ring[j] : 0u;
    zold += in ? __popc(~row[m]) : 0;
#pragma unroll
    for (int p = 0; p < P; p++) pl[p][m] = in ? s_pl[j * P + p] : 0u;
  }
  uint32_t rv[P];
#pragma unroll
  for (int p = 0; p < P; p++) rv[p] = __brev(cur[p]);
#pragma unroll 2
  for (int k = 0; k < cols; k++) {
    uint32_t mk[P];
#pragma unroll
    for (int p = 0; p < P; p++) {
      mk[p] = (uint32_t)((int)rv[p] >> 31);
      rv[p] <<= 1;
    }
    dp_tile<P, TW>(row, pl, mk, cw, ncw);
  }
  int znew = 0;
#pragma unroll
  for (int m = 0; m < TW; m++) {
    const int j = base + m;
    if (j <= je) {
      ring[j] = row[m];
      znew += __popc(~row[m]);
    }
  }
  return znew - zold;
}

// DNA match table: for every rep block j its four match words, word 4j + c =
// the rows of block j whose residue is c (c = plane-0 bit | plane-1 bit << 1),
// i.e. ~(p0 ^ m0) & ~(p1 ^ m1) for the masks of residue c — the same words
// the plane form builds per column.  kEqPad zero blocks follow the last rep
// block, so a tile's padding slots (rows above je, whose row words are 0 and
// mask whatever they read) stay inside the table.
constexpr int kEqPad = 32;
__host__ __device__ constexpr int eq_words(int max_nb) { return 4 * (max_nb + kEqPad); }
// Word offset of the match table in the tiled kernel's dynamic shared memory:
// after the planes, the k-mer bitset and the row ring (ring = 0: global ring).
__host__ __device__ constexpr int tiled_eq_off(int P, int max_nb, int ring) {
  return ((max_nb * P + 3) & ~3) + kListWords + ring * kAlignThreads;
}

// Builds the match table of the representative whose planes are staged at
// s_pl (nb1 blocks) with all threads of the CTA; the caller synchronises.
__device__ __forceinline__ void build_eq(const uint32_t *s_pl, int nb1, uint32_t *s_eq) {
  for (int j = threadIdx.x; j < nb1 + kEqPad; j += blockDim.x) {
    const bool real = j < nb1;
    const uint32_t p0 = real ? s_pl[2 * j] : 0u, p1 = real ? s_pl[2 * j + 1] : 0u;
    uint4 e;
    e.x = real ? ~p0 & ~p1 : 0u;
    e.y = p0 & ~p1;
    e.z = ~p0 & p1;
    e.w = p0 & p1;
    *reinterpret_cast<uint4 *>(s_eq + 4 * j) = e;
  }
}

// ---- match-table tiles with the per-column bookkeeping on the FMA pipe -------
// Run-time constants 1 and 4: ptxas cannot fold a multiply by them into a
// shift or an add, so the multiply-adds below stay IMADs (FMA pipe).
struct FmaK {
  uint32_t one, four;
};

// Column codes of one 32-residue query block, first column on top: w[h]
// holds columns 16h..16h+15, two bits each (plane-1 bit above plane-0 bit),
// column 16h in bits 31..30.
__device__ __forceinline__ void eq_codes_top(const uint32_t (&cur)[2], uint32_t (&w)[2]) {
  const uint32_t r0 = __brev(cur[0]), r1 = __brev(cur[1]);
  w[0] = spread16(r0 >> 16) | (spread16(r1 >> 16) << 1);
  w[1] = spread16(r0) | (spread16(r1) << 1);
}

// Shared-memory address of the next column's match words: code = w >> 30,
// w <<= 2, address = eb + 4 code — three multiply-adds.
__device__ __forceinline__ uint32_t eq_next_addr(uint32_t &w, uint32_t eb, const FmaK &k) {
  uint32_t c, a;
  asm("mul.hi.u32 %0, %1, %2;" : "=r"(c) : "r"(w), "r"(k.four));
  asm("mul.lo.u32 %0, %0, %1;" : "+r"(w) : "r"(k.four));
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(a) : "r"(c), "r"(k.four), "r"(eb));
  return a;
}

// Match words of TW slots at shared address a (slot m at a + 16 m; the
// offsets are immediates of the loads).
template <int M, int TW>
struct EqLoad {
  static __device__ __forceinline__ void run(uint32_t (&e)[TW], uint32_t a) {
    EqLoad<M - 1, TW>::run(e, a);
    asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(e[M - 1]) : "r"(a), "n"(16 * (M - 1)));
  }
};
template <int TW>
struct EqLoad<0, TW> {
  static __device__ __forceinline__ void run(uint32_t (&)[TW], uint32_t) {}
};
template <int TW>
__device__ __forceinline__ void eq_load_s(uint32_t (&e)[TW], uint32_t a) {
  EqLoad<TW, TW>::run(e, a);
}

// eq_columns with the codes on top of w[] and the FMA-pipe bookkeeping.
template <int TW, bool PF>
__device__ __forceinline__ void eq_columns_f(uint32_t (&row)[TW], uint32_t eb, const uint32_t (&wc)[2], int cols,
                                             uint32_t &cw, uint32_t &ncw, const FmaK &k) {
#pragma unroll 1
  for (int h = 0; h < 2; h++) {
    const int n = min(16, cols - 16 * h);
    if (n <= 0) break;
    uint32_t w = wc[h];
    if constexpr (PF) {
      uint32_t ea[TW], eo[TW];
      eq_load_s<TW>(ea, eq_next_addr(w, eb, k));
      int c = 0;
#pragma unroll 1
      for (; c + 2 <= n; c += 2) {
        eq_load_s<TW>(eo, eq_next_addr(w, eb, k));
        dp_tile_eqf<TW>(row, ea, cw, ncw, k.one);
        eq_load_s<TW>(ea, eq_next_addr(w, eb, k));  // past the last column: code 0, in bounds
        dp_tile_eqf<TW>(row, eo, cw, ncw, k.one);
      }
      if (c < n) dp_tile_eqf<TW>(row, ea, cw, ncw, k.one);
    } else {
#pragma unroll 1
      for (int c = 0; c < n; c++) {
        uint32_t ev[TW];
        eq_load_s<TW>(ev, eq_next_addr(w, eb, k));
        dp_tile_eqf<TW>(row, ev, cw, ncw, k.one);
      }
    }
  }
}

// Straight tile: rows base .. base+TW-1 all inside the lane's window
// (<= je) and contiguous in the shared-memory ring (no wrap).  Its rows are
// then at rp + m * threads, immediate offsets from one address.
template <int TW, class Ring>
__device__ __forceinline__ bool tile_straight(const Ring &ring, int base, int je, uint32_t *&rp) {
  if constexpr (Ring::kSize >= TW) {
    rp = ring.at(base);
    return base + TW - 1 <= je && (base & (Ring::kSize - 1)) + TW <= Ring::kSize;
  } else {
    rp = nullptr;
    return false;
  }
}
template <int TW>
__device__ __forceinline__ void tile_load_straight(uint32_t (&row)[TW], const uint32_t *rp) {
#pragma unroll
  for (int m = 0; m < TW; m++) row[m] = rp[m * kAlignThreads];
}
// Stores a straight tile's rows; returns their zero count.
template <int TW>
__device__ __forceinline__ int tile_store_straight(const uint32_t (&row)[TW], uint32_t *rp) {
#pragma unroll
  for (int m = 0; m < TW; m++) rp[m * kAlignThreads] = row[m];
  int ones = 0;
#pragma unroll
  for (int m = 0; m < TW; m++) ones += __popc(row[m]);
  return 32 * TW - ones;
}

// One tile of band rows base .. base+TW-1 (rows above je are padding) through
// the block's columns, with the match table at shared address s_eq_s; returns
// the zero count of the tile's rows after the block.
template <int TW, bool PF, class Ring>
__device__ __forceinline__ int tiled_tile_eqf(const Ring &ring, uint32_t s_eq_s, int base, int je, int nb1, int cols,
                                              const uint32_t (&wc)[2], uint32_t &cw, uint32_t &ncw, const FmaK &k) {
  uint32_t row[TW];
  uint32_t *rp = nullptr;
  const bool straight = tile_straight<TW>(ring, base, je, rp);
  if (straight) {
    tile_load_straight<TW>(row, rp);
  } else {
#pragma unroll
    for (int m = 0; m < TW; m++) {
      const int j = base + m;
      row[m] = j <= je ? ring[j] : 0u;
    }
  }
  // A tile past the rep's last block (a lane with a narrower window than its
  // warp's widest) is all padding: it reads the zero blocks after nb1.
  eq_columns_f<TW, PF>(row, s_eq_s + 16u * (uint32_t)min(base, nb1), wc, cols, cw, ncw, k);
  if (straight) return tile_store_straight<TW>(row, rp);
  int z = 0;
#pragma unroll
  for (int m = 0; m < TW; m++) {
    const int j = base + m;
    if (j <= je) {
      ring[j] = row[m];
      z += __popc(~row[m]);
    }
  }
  return z;
}

// Remainder tile widths 1 .. 16, rounded up to a multiple of NGIA_REM_ROUND
// (extra slots are padding).
#define NGIA_REM_CASES(X) \
  X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16)

template <class Ring>
__device__ __forceinline__ int tiled_rem_eqf(int rem, const Ring &ring, uint32_t s_eq_s, int base, int je, int nb1,
                                             int cols, const uint32_t (&wc)[2], uint32_t &cw, uint32_t &ncw,
                                             const FmaK &k) {
  constexpr int R = NGIA_REM_ROUND;
  switch ((rem + R - 1) / R * R) {
#define NGIA_REM(W) \
  case W:           \
    if (W % R == 0) return tiled_tile_eqf<W % R == 0 ? W : 1, false, Ring>(ring, s_eq_s, base, je, nb1, cols, wc, cw, ncw, k); \
    return 0;
    NGIA_REM_CASES(NGIA_REM)
#undef NGIA_REM
    default:
      return 0;
  }
}

// The last tile of a block row, exactly `rem` (1..MT-1, warp-uniform) slots wide.
template <int P, class Ring, int MT>
__device__ __forceinline__ int tiled_rem(int rem, const Ring &ring, const uint32_t *s_pl, int base, int je, int cols,
                                         const uint32_t (&cur)[P], uint32_t &cw, uint32_t &ncw) {
  switch (rem) {
#define NGIA_REM(W) \
  case W:           \
    if (W < MT) return tiled_tile<P, (W < MT ? W : 1), Ring>(ring, s_pl, base, je, cols, cur, cw, ncw); \
    return 0;
    NGIA_REM_CASES(NGIA_REM)
#undef NGIA_REM
    default:
      return 0;
  }
}

// Rep block a pair's window reaches in its first query block: blocks whose
// first row could still end at `cut` zeros after 32 columns.
__device__ __forceinline__ int band_first_top(int B, int nb1, int net1, int cut) {
  return min(min(B, nb1 - 1), max(0, (32 + net1 - cut) >> 5));
}

// Moves a pair's window [js, je] from query block i-1 to query block i of its
// band and drops the rows that no score of at least `cut` can use.
//
// Write F(j) for the zeros counted in rows below j (the longest chain of
// matches that ends there), left for the query residues still to come.  A
// chain that stops below row j now can gain at most `left` more matches, and
// one that continues above row j at most net1 - j.  So
//   * block js is out for good when F(its end) + left < cut: it is banked
//     (frozen), as a block that leaves the reference's band is;
//   * the pair is out when F(start of js) + (rows above it) < cut;
//   * block je is idle during block i when F(its start) + 32 + (rows from
//     it) < cut (F grows by at most one per column): its state is dropped,
//     and it enters all-ones again once the rule lets it back in, so the
//     chains it held, which cannot reach cut, are gone.
// What remains is the recurrence over a smaller staircase of the same band,
// which keeps every chain that reaches cut: accepted scores are the
// reference's, and a pair that stays below cut stays below it.  The limits
// move by at most one block per query block, so one entering block is enough.
// cut = kNoCut disables the rules (every score is wanted).
//
// DNA s=0.85, rep 1,990 against 1,450 residues: windows of 22 blocks on
// average instead of 49, half of the cells.  GB300: 12 iterations over 1M DNA
// 97.5 -> 64.4 ms, a 20,000-sequence job to the end 487 -> 320 ms, 16 query
// batches against 6,000 representatives 51.4 -> 31.8 ms.
constexpr int kNoCut = -(1 << 30);
enum { kBandGo = 0, kBandDone = 1, kBandReject = 2 };

template <class Ring>
__device__ __forceinline__ int band_advance(const Ring &ring, int i, int B, int nb1, int net1, uint32_t vlast,
                                            int left, int cut, int &js, int &je, int &frozen, int &zw) {
  while (js <= je) {
    const uint32_t r = ~ring[js];
    const int z = __popc(js == nb1 - 1 ? r & vlast : r);
    if (js >= i - B && frozen + z + left >= cut) break;
    frozen += z;
    zw -= __popc(r);
    js++;
  }
  if (frozen + zw + left < cut || frozen + max(net1 - 32 * js, 0) < cut) return kBandReject;
  while (je > js) {
    const int z = __popc(~ring[je]);
    if (frozen + zw - z + 32 + net1 - 32 * je >= cut) break;
    zw -= z;
    je--;
  }
  if (je < min(i + B, nb1 - 1) && frozen + zw + net1 - 32 * je >= cut) {
    je++;
    ring[je] = 0xFFFFFFFFu;
  }
  return js > je ? kBandDone : kBandGo;
}

// Main tile width of the tiled kernel (16 slots; NGIA_TILED_MAIN_DNA for DNA).
__host__ __device__ constexpr int tiled_main(int P) { return P == 2 ? NGIA_TILED_MAIN_DNA : 16; }
__host__ __device__ constexpr int tiled_min_blocks(int P) { return P == 2 ? NGIA_TILED_BLOCKS_DNA : 2; }

}  // namespace ngia
