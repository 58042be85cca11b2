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
//  Swept with windows that follow their pair (20,000 DNA to the end | 400k
//  DNA, 12 iterations, ms): 16 slots, 4 CTAs, prefetch 233 | 22.7; without
//  prefetch 234 | 24.6; 5 CTAs 236 | 23.1; 12 slots 252 | 25.6 (5 CTAs); 8
//  slots 260 | 27 (6, 7 CTAs); remainder tiles of even width 238 | 23.3.
//  Columns unrolled, adds as IMAD.X and the like lost 3-60% earlier (the
//  kernels are sensitive to their instruction footprint).
#ifndef NGIA_TILED_MAIN_DNA
#define NGIA_TILED_MAIN_DNA 16
#endif
#ifndef NGIA_TILED_BLOCKS_DNA
#define NGIA_TILED_BLOCKS_DNA 4
#endif
#ifndef NGIA_EQ_PF_MAIN
#define NGIA_EQ_PF_MAIN 1
#endif
namespace ngia {

constexpr int kAlignThreads = 128;  // threads per CTA of every alignment kernel

// Band rows of one lane's pair, indexed by absolute rep block j and one after
// the other in memory, so that a tile's rows have immediate offsets from its
// first.  A tile loads and stores all its rows: those above the window's top
// (padding of a lane whose window is narrower than its warp's widest) hold
// anything, and a row is set when it enters the window (band_advance).
//
// SmemRing: CAP rows per lane in shared memory, row j of thread t at
// (j - off) * threads + t (the 32 lanes of a warp hit 32 banks); when a
// window reaches the end its rows move to the start (fit), once in CAP minus
// the warp's widest window query blocks (kSmallWindow, kWideWindow: 16 at
// least).
// GlobalRing: every rep block and the padding (global_rows) in global
// scratch, with the same layout over all lanes of the grid (a warp's access
// to one row is one 128-byte line).
template <int CAP>
struct SmemRing {
  static constexpr int kPitch = kAlignThreads;
  uint32_t *base;  // rows + threadIdx.x
  int off = 0;     // rep block of the first row
  __device__ __forceinline__ void reset() { off = 0; }
  __device__ __forceinline__ uint32_t &operator[](int j) const { return base[(j - off) * kAlignThreads]; }
  __device__ __forceinline__ void fit(int js, int je, int slots) {
    if (js - off + slots < CAP) return;  // and a row for the block that enters next
    for (int j = js; j <= je; j++) base[(j - js) * kAlignThreads] = base[(j - off) * kAlignThreads];
    off = js;
  }
};
struct GlobalRing {
  static constexpr int kPitch = 0;
  uint32_t *base;  // scratch + global lane index
  int64_t stride;  // lanes of the grid
  __device__ __forceinline__ void reset() {}
  __device__ __forceinline__ uint32_t &operator[](int j) const { return base[(int64_t)j * stride]; }
  __device__ __forceinline__ void fit(int, int, int) {}
};
template <int CAP>
struct RingOf {
  using T = SmemRing<CAP>;
};
template <>
struct RingOf<0> {
  using T = GlobalRing;
};

template <int TW, class Ring>
__device__ __forceinline__ void rows_load(const Ring &ring, int base, uint32_t (&row)[TW]) {
  const uint32_t *rp = &ring[base];
  if constexpr (Ring::kPitch > 0) {
#pragma unroll
    for (int m = 0; m < TW; m++) row[m] = rp[m * Ring::kPitch];
  } else {
#pragma unroll
    for (int m = 0; m < TW; m++) row[m] = rp[m * ring.stride];
  }
}
// Stores a tile's rows; returns their zero count.
template <int TW, class Ring>
__device__ __forceinline__ int rows_store(const Ring &ring, int base, const uint32_t (&row)[TW]) {
  uint32_t *rp = &ring[base];
  int ones = 0;
  if constexpr (Ring::kPitch > 0) {
#pragma unroll
    for (int m = 0; m < TW; m++) rp[m * Ring::kPitch] = row[m];
  } else {
#pragma unroll
    for (int m = 0; m < TW; m++) rp[m * ring.stride] = row[m];
  }
#pragma unroll
  for (int m = 0; m < TW; m++) ones += __popc(row[m]);
  return 32 * TW - ones;
}

// One tile from plane registers: rows base .. base+TW-1 through the `cols`
// columns of the current block, whose P plane words are cur[]; planes points
// at the rows' sequence (nbr blocks, shared or global memory).  cw holds the
// column carries into the tile (column 0 at bit 31), ncw collects the
// carries out.  Returns the rows' zero count.
template <int P, int TW, class Ring>
__device__ __forceinline__ int tile_planes(const Ring &ring, const uint32_t *planes, int base, int nbr, int cols,
                                           const uint32_t (&cur)[P], uint32_t &cw, uint32_t &ncw) {
  uint32_t row[TW], pl[P][TW];
  rows_load<TW>(ring, base, row);
#pragma unroll
  for (int m = 0; m < TW; m++) {
    const uint32_t *b = planes + min(base + m, nbr - 1) * P;
#pragma unroll
    for (int p = 0; p < P; p++) pl[p][m] = b[p];
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
  return rows_store<TW>(ring, base, row);
}

// DNA match table: for every rep block j its four match words, word 4j + c =
// the rows of block j whose residue is c (c = plane-0 bit | plane-1 bit << 1),
// i.e. ~(p0 ^ m0) & ~(p1 ^ m1) for the masks of residue c — the same words
// the plane form builds per column.  kEqPad zero blocks follow the last rep
// block, so a tile's padding slots (rows above je) read inside the table.  Their
// rows hold anything: carries only go up, away from the window's rows, and
// tile_block takes their zeros off the count.
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
  uint32_t one, two, four, eight;
  __device__ __forceinline__ explicit FmaK(uint32_t one_rt) : one(one_rt), two(one_rt << 1), four(one_rt << 2), eight(one_rt << 3) {}
};

// Shared-memory address of the next column's match words: the code's two bits
// are on top of the bit-reversed planes w[]; four high and low products by a
// run-time 2 and two multiply-adds, all on the FMA pipe.  (Packing the codes
// first takes half of these and 42 logic instructions per block of columns:
// the same time.)
__device__ __forceinline__ uint32_t eq_next_addr(uint32_t (&w)[2], uint32_t eb, const FmaK &k) {
  uint32_t c0, c1, a;
  asm("mul.hi.u32 %0, %1, %2;" : "=r"(c0) : "r"(w[0]), "r"(k.two));
  asm("mul.hi.u32 %0, %1, %2;" : "=r"(c1) : "r"(w[1]), "r"(k.two));
  asm("mul.lo.u32 %0, %0, %1;" : "+r"(w[0]) : "r"(k.two));
  asm("mul.lo.u32 %0, %0, %1;" : "+r"(w[1]) : "r"(k.two));
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(a) : "r"(c0), "r"(k.four), "r"(eb));
  asm("mad.lo.u32 %0, %1, %2, %0;" : "+r"(a) : "r"(c1), "r"(k.eight));
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

// All `cols` columns of one block through a tile whose match words start at
// shared address eb; the tile takes column carries in cw and hands them out
// in ncw.  PF: the next column's match words are loaded while the current
// column updates (two columns per loop trip).
template <int TW, bool PF>
__device__ __forceinline__ void eq_columns(uint32_t (&row)[TW], uint32_t eb, const uint32_t (&cur)[2], int cols,
                                           uint32_t &cw, uint32_t &ncw, const FmaK &k) {
  uint32_t w[2] = {__brev(cur[0]), __brev(cur[1])};
  if constexpr (PF) {
    uint32_t ea[TW], eo[TW];
    eq_load_s<TW>(ea, eq_next_addr(w, eb, k));
    int c = 0;
#pragma unroll 1
    for (; c + 2 <= cols; c += 2) {
      eq_load_s<TW>(eo, eq_next_addr(w, eb, k));
      dp_tile_eqf<TW>(row, ea, cw, ncw, k.one);
      eq_load_s<TW>(ea, eq_next_addr(w, eb, k));  // past the last column: some code, in bounds
      dp_tile_eqf<TW>(row, eo, cw, ncw, k.one);
    }
    if (c < cols) dp_tile_eqf<TW>(row, ea, cw, ncw, k.one);
  } else {
#pragma unroll 1
    for (int c = 0; c < cols; c++) {
      uint32_t ev[TW];
      eq_load_s<TW>(ev, eq_next_addr(w, eb, k));
      dp_tile_eqf<TW>(row, ev, cw, ncw, k.one);
    }
  }
}

// One DNA tile with the match table at shared address s_eq_s (per column one
// load per slot and three integer instructions per 32 cells: AND, add with
// carry, LOP3).  A tile past the last rep block (a lane with a narrower
// window than its warp's widest) reads the table's zero blocks.
template <int TW, bool PF, class Ring>
__device__ __forceinline__ int tile_eq(const Ring &ring, uint32_t s_eq_s, int base, int nbr, int cols,
                                       const uint32_t (&cur)[2], uint32_t &cw, uint32_t &ncw, const FmaK &k) {
  uint32_t row[TW];
  rows_load<TW>(ring, base, row);
  eq_columns<TW, PF>(row, s_eq_s + 16u * (uint32_t)min(base, nbr), cur, cols, cw, ncw, k);
  return rows_store<TW>(ring, base, row);
}

// Main tile width of the tiled kernels.
__host__ __device__ constexpr int tiled_main(int P) { return P == 2 ? NGIA_TILED_MAIN_DNA : 16; }
__host__ __device__ constexpr int tiled_min_blocks(int P) { return P == 2 ? NGIA_TILED_BLOCKS_DNA : 2; }

// One block of columns (planes cur[], cols of them) over a lane's window
// [js, je] in tiles of `slots` rows altogether (the warp's widest window: the
// lanes stay in step, narrower windows run padding slots).  TABLE: match words from
// s_eq_s, else from the rows' planes.  Returns the window's zero count.
template <int P, bool TABLE, class Ring>
__device__ __forceinline__ int tile_block(Ring &ring, uint32_t s_eq_s, const uint32_t *planes, int js, int je, int nbr,
                                          int slots, int cols, const uint32_t (&cur)[P], const FmaK &fk) {
  constexpr int MT = tiled_main(P);
  ring.fit(js, je, slots);
  uint32_t cw = 0, ncw = 0;
  int z = 0, base = js, left = slots;
  for (; left >= MT; left -= MT, base += MT) {
    if constexpr (TABLE)
      z += tile_eq<MT, NGIA_EQ_PF_MAIN>(ring, s_eq_s, base, nbr, cols, cur, cw, ncw, fk);
    else
      z += tile_planes<P, MT>(ring, planes, base, nbr, cols, cur, cw, ncw);
    cw = ncw << (32 - cols);  // column 0's carry at bit 31
    ncw = 0;
  }
  switch (left) {
#define NGIA_REM(W)                                                                                            \
  case W:                                                                                                      \
    if constexpr (W < MT) {                                                              \
      if constexpr (TABLE)                                                                                     \
        z += tile_eq<W, false>(ring, s_eq_s, base, nbr, cols, cur, cw, ncw, fk);                                \
      else                                                                                                     \
        z += tile_planes<P, W>(ring, planes, base, nbr, cols, cur, cw, ncw);                                   \
    }                                                                                                          \
    break;
    NGIA_REM(1) NGIA_REM(2) NGIA_REM(3) NGIA_REM(4) NGIA_REM(5) NGIA_REM(6) NGIA_REM(7) NGIA_REM(8)
    NGIA_REM(9) NGIA_REM(10) NGIA_REM(11) NGIA_REM(12) NGIA_REM(13) NGIA_REM(14) NGIA_REM(15)
#undef NGIA_REM
    default: break;
  }
  for (int j = je + 1; j < js + slots; j++) z -= __popc(~ring[j]);  // the padding's zeros
  return z;
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

}  // namespace ngia
