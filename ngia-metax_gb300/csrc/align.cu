// align.cu — banded bit-parallel LCS identity kernels (the reference's
// kernel_dynamicGen/Pro, CUDA/signalNode/src/func.cu:450-604).
//
// The reference computes, per (representative, query) pair, a block-banded
// form of the Allison–Dix / Hyyrö bit-vector LCS: the representative's net
// residues are the rows (32 per word, line[j]), the query's net residues the
// columns, processed in 32-column blocks i.  For query block i only rep
// blocks j in [max(i-B,0), min(i+B,nb1-1)] are updated, with
// B = (ceil(fma(-L2,s,L1)) + 31)/32; the carry into the lowest band block is
// 0 and the carry out of the highest is dropped; blocks outside the band keep
// their state.  The score is the number of zero bits of line[] over the net
// length, accepted when >= ceil(L2*s).
//
// Two kernels give the same accepted scores and the same rejections:
//
// k_align_tiled<P,RING>  one thread per pair.  The band rows live in a ring
//   (shared memory for windows up to RING = 64 or 128 blocks, global scratch
//   for any width with RING = 0) and are updated tile by tile in registers:
//   for each query residue a tile of 16 row words is one multi-word addition
//   whose carries ride the hardware carry flag (add.cc/addc.cc).  The match
//   word of a slot comes, for DNA, from the representative's match table in
//   shared memory (four words per rep block, one per residue code; tile.cuh),
//   so a 32-cell word costs one load and three integer instructions (AND,
//   IADD3.X, LOP3); protein builds it from the rep's planes held in registers
//   (one LOP3 per plane).
//
// k_align_wave<P,NW,WMAX>, k_align_query<P>  classes with few queued pairs: 8,
//   32 or 128 threads per pair by their number and the width of their windows;
//   16 threads for a short query against a long representative (wave.cuh).
//
// In clustering both keep only the rows that a score of at least the cutoff
// can use (band_advance in tile.cuh) and stop a pair once it provably cannot
// reach it; accepted pairs are always computed to the end (their score is
// reported).  Pair-score mode computes the whole band.
#include <algorithm>
#include <climits>
#include <cstdlib>
#include <mutex>

#include "ctx.h"
#include "kmer.cuh"
#include "tile.cuh"
#include "wave.cuh"

namespace ngia {

constexpr int kRepPlanesOff = 32;  // planes offset inside rb.rep_rec (filter.cu)

struct AlignHdr {
  int qn, L1, net1, nb1, word_after, rep;
};

// Reads the iteration header and stages the representative's planes (and,
// when the short-word test follows the alignment, its k-mer bitset) into
// shared memory with bulk copies.  Returns false when there is no work.
// groups: pairs a CTA of the group-per-pair kernel works on at a time (it
// takes classes with at most warp_pairs pairs; more once there are more than
// `few`), 0 for the thread-per-pair kernels (classes with more);
// the other kernel of a class returns here, before any staging.
template <int P>
__device__ __forceinline__ bool align_setup(const DevDB &db, const RunBufs &rb, const RunParams &prm, int cls,
                                            int score_mode, int warp_pairs, int groups, int few, int subs, uint32_t *smem,
                                            uint64_t *bar, AlignHdr &h) {
  __shared__ int s_hdr[6];
  RunState *st = rb.st;
  if (threadIdx.x == 0) {
    const bool skip = !score_mode && (st->done || st->iter >= st->iter_limit || st->err);
    const int qn = skip ? 0 : (int)st->qcount[cls];
    const bool mine = groups ? qn <= warp_pairs : qn > warp_pairs;
    const int per = qn > subs ? kAlignThreads / kSubGroup : qn > few ? max(groups, kAlignThreads / 32) : groups;
    const bool idle = (int)blockIdx.x * per >= qn;
    s_hdr[0] = mine && !(groups && idle) ? qn : 0;
    s_hdr[1] = st->rep_len;
    s_hdr[2] = st->rep_net;
    s_hdr[3] = st->rep_nb;
    s_hdr[4] = !score_mode && st->word_active && !st->word_first;
    s_hdr[5] = st->rep;
  }
  __syncthreads();
  h.qn = s_hdr[0];
  if (h.qn == 0) return false;
  h.L1 = s_hdr[1];
  h.net1 = s_hdr[2];
  h.nb1 = s_hdr[3];
  h.word_after = s_hdr[4];
  h.rep = s_hdr[5];
  const uint32_t plane_words = (uint32_t)((h.nb1 * P + 3) & ~3);
  const uint32_t list_words = h.word_after ? (uint32_t)max(4, (int)((1u << (prm.w * (P == 2 ? 2 : 5))) / 32u)) : 0u;
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    const uint32_t bytes = 4u * (plane_words + list_words);
    if (bytes) {
      mbar_expect_tx(bar, bytes);
      if (plane_words) bulk_g2s(smem, rb.rep_rec + kRepPlanesOff, 4u * plane_words, bar);
      if (list_words) bulk_g2s(smem + plane_words, rb.rep_list, 4u * list_words, bar);
    } else {
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
    }
  }
  __syncthreads();
  bool ok = mbar_wait_bounded(bar, 0, prm.wait_polls);
  if (!ok) {
    set_error(st, NGIA_ERR_MBAR_TIMEOUT, 10 + cls);
    mbar_wait_bounded(bar, 0, kWaitPolls);  // let the copy in flight land
  }
  return __syncthreads_and(ok);
}

// Claims the next queue entry for every idle lane with one atomic per warp.
// state: -1 idle, -2 queue exhausted, >= 0 the claimed entry.
__device__ __forceinline__ void claim(RunState *st, int cls, int qn, int lane, int &state) {
  const bool need = state == -1;
  const unsigned nm = __ballot_sync(kFullMask, need);
  if (!nm) return;
  const int leader = __ffs(nm) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(&st->qhead[cls], (uint32_t)__popc(nm));
  base = __shfl_sync(kFullMask, base, leader);
  if (need) {
    const uint32_t idx = base + (uint32_t)__popc(nm & ((1u << lane) - 1u));
    state = idx < (uint32_t)qn ? (int)idx : -2;
  }
}

// Outcome of one pair: membership (or the pair score in score mode).
template <int P>
__device__ __forceinline__ void finish_pair(const DevDB &db, const RunBufs &rb, const RunParams &prm,
                                            const AlignHdr &h, int score_mode, int entry, int cand, int sum,
                                            int cutoff, int L2, int net2, const uint32_t *qpl,
                                            const uint32_t *s_list, unsigned long long &members) {
  if (score_mode) {
    rb.score_out[4 * entry + 2] = sum;
    return;
  }
  bool pass = !(sum < cutoff);
  if (pass && h.word_after && cand == h.rep) {  // every word of its own
    pass = !(max(0, h.net1 - prm.w + 1) < word_min(L2, prm.w, prm.s));
  } else if (pass && h.word_after) {
    // short-word test of func.cu:376-396, evaluated only for aligned members
    int ws = 0;
    {
      constexpr int bits = P == 2 ? 2 : 5;
      const uint32_t mask = (1u << (prm.w * bits)) - 1u;
      uint32_t word = 0;
      for (int i = 0; i < net2; i += 32) {
        uint32_t pl[P];
#pragma unroll
        for (int p = 0; p < P; p++) pl[p] = qpl[(i >> 5) * P + p];
        const int lim = min(32, net2 - i);
        for (int j = 0; j < lim; j++) {
          uint32_t c = 0;
#pragma unroll
          for (int p = 0; p < P; p++) c |= ((pl[p] >> j) & 1u) << p;
          word = ((word << bits) | c) & mask;
          if (i + j >= prm.w - 1) ws += (s_list[word >> 5] >> (word & 31)) & 1u;
        }
      }
    }
    pass = !(ws < word_min(L2, prm.w, prm.s));
  }
  if (pass) {
    rb.cluster[cand] = h.rep;
    rb.ident[cand] = sum;
    atomicAnd(&rb.alive[cand >> 5], ~(1u << (cand & 31)));
    members++;
  }
}

__device__ __forceinline__ void flush_align_stats(RunState *st, int cls, unsigned long long pairs,
                                                  unsigned long long members, unsigned long long cells,
                                                  unsigned long long done, unsigned long long *s_qwords) {
  for (int o = 16; o; o >>= 1) {
    pairs += __shfl_down_sync(kFullMask, pairs, o);
    members += __shfl_down_sync(kFullMask, members, o);
    cells += __shfl_down_sync(kFullMask, cells, o);
    done += __shfl_down_sync(kFullMask, done, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (pairs) atomicAdd(&st->st_align_pairs, pairs);
    if (members) atomicAdd(&st->st_members, members);
    if (cells) atomicAdd(&st->st_band_cells, cells);
    if (done) {
      atomicAdd(&st->st_done_cells, done * 32ull);
      atomicAdd(&st->st_class_done[cls], done * 32ull);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && *s_qwords) atomicAdd(&st->st_class_qwords[cls], *s_qwords);
}

// Tiled window: windows of up to RING rep blocks (any width for RING = 0).
// Each lane keeps its pair's band rows in a ring indexed by absolute rep
// block (SmemRing / GlobalRing above) and runs each query block tile by tile in
// ascending rep-block order, all residues of the block per tile — the
// reference's (i, j, k) loop order at tile granularity.  Full tiles are MT
// slots (tiled_main); the remainder runs as one tile of exactly its width;
// the column carries pass between tiles in one word (one instruction to pop a
// carry, one to push it).  A warp's lanes start their pairs together (see the
// refill below), so their windows are equally wide and padding is rare.
//
template <int P, int RING>
__global__ void __launch_bounds__(kAlignThreads, tiled_min_blocks(P))
    k_align_tiled(DevDB db, RunBufs rb, RunParams prm, int cls, int score_mode, int warp_pairs) {
  extern __shared__ __align__(16) uint32_t smem[];
  __shared__ uint64_t bar;
  AlignHdr h;
  __shared__ unsigned long long s_qw;  // query plane words of the pairs taken (algorithmic bytes / 4)
  if (threadIdx.x == 0) s_qw = 0;
  if (!align_setup<P>(db, rb, prm, cls, score_mode, warp_pairs, 0, 0, 0, smem, &bar, h)) return;
  const uint32_t *s_pl = smem;
  const uint32_t *s_list = smem + ((h.nb1 * P + 3) & ~3);
  RunState *st = rb.st;
  constexpr bool kEq = P == 2;
  uint32_t *s_eq = smem + tiled_eq_off(P, db.max_nb, RING);
  if constexpr (kEq) {
    build_eq(s_pl, h.nb1, s_eq);  // the representative's match table (tile.cuh)
    __syncthreads();
  }
  const uint32_t s_eq_s = smem_u32(s_eq);
  // powers of two as values ptxas cannot fold (nb1 is read from shared memory)
  const uint32_t one_rt = 1u + (uint32_t)(h.nb1 < 0);
  const FmaK fk(one_rt);
  (void)s_eq_s;
  (void)fk;
  typename RingOf<RING>::T ring;
  if constexpr (RING > 0) {
    ring.base = smem + (((db.max_nb * P + 3) & ~3) + kListWords) + threadIdx.x;
  } else {
    const int64_t TL = (int64_t)gridDim.x * blockDim.x;
    if ((int64_t)rb.ring_rows * TL > rb.scratch_words) {
      if (threadIdx.x == 0) set_error(st, NGIA_ERR_SCRATCH, 20);
      return;
    }
    ring.base = rb.scratch + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    ring.stride = TL;
  }
  const int lane = threadIdx.x & 31;
  const float s = prm.s;
  const int nb1 = h.nb1;
  const uint32_t vlast = (h.net1 & 31) ? ((1u << (h.net1 & 31)) - 1u) : 0xFFFFFFFFu;

  int state = -1, entry = 0, cand = 0;
  int i = 0, nq = 0, B = 0, js = 0, je = -1, net2 = 0, L2 = 0, cutoff = 0, lastcols = 32, frozen = 0, zw = 0;
  int cut = 0;  // the band rules' cutoff (none in pair-score mode)
  bool active = false;
  const uint32_t *qpl = nullptr;
  uint32_t cur[P], nxt[P];
  unsigned long long n_pairs = 0, n_members = 0, n_cells = 0, n_done = 0;
  for (;;) {
    // A warp refills once prm.refill of its lanes are idle (or none is busy).
    // Queue entries next to each other are candidates of similar length, so
    // lanes that start together keep equal band windows block after block.
    {
      const unsigned idle = __ballot_sync(kFullMask, state == -1);
      const bool any_busy = __any_sync(kFullMask, state >= 0);  // every lane votes
      if (__popc(idle) >= prm.refill || !any_busy) claim(st, cls, h.qn, lane, state);
    }
    if (__all_sync(kFullMask, state == -2)) break;
    // No lane leaves the loop body early: the warp-wide reductions below are
    // executed by all 32 lanes (lanes without a pair contribute neutral values).
    bool busy = state >= 0;
    if (busy && !active) {
      entry = rb.queue[cls][state];
      cand = score_mode ? rb.score_cands[entry] : entry;
      L2 = __ldg(db.len + cand);
      net2 = __ldg(db.net + cand);
      nq = (net2 + 31) >> 5;
      lastcols = (net2 & 31) ? (net2 & 31) : 32;
      B = band_blocks(h.L1, L2, s);
      cutoff = cutoff_of(L2, s);
      qpl = db.words + __ldg(db.off + cand) + db.hw;
      cut = score_mode ? kNoCut : cutoff;
      i = 0;
      js = 0;
      je = band_first_top(B, nb1, h.net1, cut);
      frozen = 0;
      zw = 0;
      if (!score_mode) {
        n_pairs++;
        n_cells += (unsigned long long)band_cells(B, nb1, net2);
        atomicAdd(&s_qw, (unsigned long long)(nq * P));
      }
      // a sequence against itself: the band holds the diagonal, so the count
      // is its net length (the reference's job list holds the representative)
      const bool self = cand == h.rep && !score_mode;
      if (B < 0 || je < 0 || nq == 0 || self) {
        finish_pair<P>(db, rb, prm, h, score_mode, entry, cand, self ? h.net1 : 0, cutoff, L2, net2, qpl, s_list, n_members);
        state = -1;
        busy = false;
      } else {
        ring.reset();
        for (int j = 0; j <= je; j++) ring[j] = 0xFFFFFFFFu;
#pragma unroll
        for (int p = 0; p < P; p++) cur[p] = __ldg(qpl + p);
        active = true;
      }
    }
    // The lanes run the tiles of the warp's widest window in step (padding
    // slots instead of different branches).
    const int n = busy ? je - js + 1 : 0;
    const int slots = (int)__reduce_max_sync(kFullMask, (unsigned)n);
    if (!busy) continue;
    const int cols = (i == nq - 1) ? lastcols : 32;
    n_done += (unsigned long long)n * cols;
    if (i + 1 < nq) {
#pragma unroll
      for (int p = 0; p < P; p++) nxt[p] = __ldg(qpl + (i + 1) * P + p);
    }
    zw = tile_block<P, kEq>(ring, s_eq_s, s_pl, js, je, nb1, slots, cols, cur, fk);
    i++;
    bool finished = i >= nq;
    if (!finished) {
      const int step = band_advance(ring, i, B, nb1, h.net1, vlast, net2 - 32 * i, cut, js, je, frozen, zw);
      if (step == kBandReject) {
        active = false;
        state = -1;
        continue;
      }
      finished = step == kBandDone;
    }
    if (finished) {
      int sum = frozen;
      for (int j = js; j <= je; j++)
        sum += __popc(~ring[j] & (j == nb1 - 1 ? vlast : 0xFFFFFFFFu));
      finish_pair<P>(db, rb, prm, h, score_mode, entry, cand, sum, cutoff, L2, net2, qpl, s_list, n_members);
      active = false;
      state = -1;
      continue;
    }
#pragma unroll
    for (int p = 0; p < P; p++) cur[p] = nxt[p];
  }
  flush_align_stats(st, cls, n_pairs, n_members, n_cells, n_done, &s_qw);
}


// Word offset of the group kernels' match table: after the planes and the
// k-mer bitset.
__host__ __device__ constexpr int wave_table_off(int P, int max_nb) { return ((max_nb * P + 3) & ~3) + kListWords; }

// ---- a group of threads per pair (wave.cuh) ------------------------------------------
// For classes with few queued pairs the latency of one pair on one thread
// bounds the iteration.  Windows up to 48 blocks: a warp per pair.  Wider ones:
// the CTA per pair for up to `few` pairs, one row word per thread for windows
// up to 112 blocks, up to 16 for any; beyond, when every scheduler has a warp,
// a warp per pair with up to 8 or 16 words, which takes half the instructions:
// a step has 80 beside the columns' (5 + 4 W) each, and 2 nq + nb1 / W steps
// are taken by one warp instead of four.  Classes of windows up to 112 blocks
// go to four pairs per warp above `subs` pairs.
struct WaveCounts {
  unsigned long long pairs = 0, members = 0, cells = 0, done = 0;
};

// This CTA's share of the class's pairs, `per` neighbouring entries at a time.
// MINE: -1 all, 1 the bands that a warp can hold, 0 the others, 2 those that 8
// threads cannot hold.
template <int P, int NW, int WMAX, int MINE>
__device__ __forceinline__ void wave_entries(const DevDB &db, const RunBufs &rb, const RunParams &prm, int cls,
                                             int score_mode, const AlignHdr &h, int per, const uint32_t *s_tab,
                                             uint32_t *s_rings, const uint32_t *s_list, uint32_t *s_xch,
                                             unsigned long long *s_qw, WaveCounts &n) {
  constexpr int kGroups = kAlignThreads / 32 / NW;
  const int group = (int)(threadIdx.x >> 5) / NW;
  const bool lead = threadIdx.x % (32 * NW) == 0;
  const float s = prm.s;
  const int nb1 = h.nb1;
  uint32_t *ring = s_rings + group * kWaveRingWords;
  for (int e0 = blockIdx.x * per; e0 < h.qn; e0 += gridDim.x * per) {
    for (int e = e0 + group; e < min(h.qn, e0 + per); e += kGroups) {
      const int entry = rb.queue[cls][e];
      const int cand = score_mode ? rb.score_cands[entry] : entry;
      const int L2 = __ldg(db.len + cand), net2 = __ldg(db.net + cand);
      const int nq = (net2 + 31) >> 5;
      const int B = band_blocks(h.L1, L2, s);
      const int cutoff = cutoff_of(L2, s), cut = score_mode ? kNoCut : cutoff;
      const uint32_t *qpl = db.words + __ldg(db.off + cand) + db.hw;
      const bool self = cand == h.rep && !score_mode, band = B >= 0 && nb1 > 0 && nq > 0;
      int lo = 0, hi = 0;
      const bool run = !self && band && wave_band(B, h.net1, net2, cut, lo, hi);
      if constexpr (MINE >= 0)
        if ((MINE == 1) == (run && !(MINE == 2 ? sub_holds(lo, hi, nb1) : wave_holds(32, 16, lo, hi, nb1)))) continue;
      if (!score_mode && lead) {
        n.pairs++;
        n.cells += (unsigned long long)band_cells(B, nb1, net2);
        atomicAdd(s_qw, (unsigned long long)(nq * P));
      }
      int sum = self ? h.net1 : 0;  // itself: the band holds the diagonal; no band: score 0
      if (!self && band) {
        if (!run) continue;  // no chain can reach the cutoff
        sum = wave_any<P, NW, WMAX>(s_tab, nb1, qpl, nq, net2, lo, hi, cut, ring, s_xch, n.done);
        if (sum < 0) continue;  // cannot reach the cutoff
      }
      if (score_mode) {
        if (lead) rb.score_out[4 * entry + 2] = sum;
        continue;
      }
      bool pass = !(sum < cutoff);
      if (pass && h.word_after && self) {
        pass = !(max(0, net2 - prm.w + 1) < word_min(L2, prm.w, s));
      } else if (pass && h.word_after && threadIdx.x / 32 == group * NW) {  // short-word test (func.cu:376-396): the group's first warp
        pass = !(word_count_warp_bits<P>(qpl, net2, prm.w, s_list) < word_min(L2, prm.w, s));
      }
      if (lead && pass) {
        rb.cluster[cand] = h.rep;
        rb.ident[cand] = sum;
        atomicAnd(&rb.alive[cand >> 5], ~(1u << (cand & 31)));
        n.members++;
      }
      __syncwarp();
    }
  }
}

// The same, four pairs per warp.
template <int P>
__device__ __forceinline__ void sub_entries(const DevDB &db, const RunBufs &rb, const RunParams &prm, int cls,
                                            int score_mode, const AlignHdr &h, const uint32_t *s_tab, uint32_t *s_rings,
                                            const uint32_t *s_list, unsigned long long *s_qw, WaveCounts &n) {
  constexpr int kGroups = kAlignThreads / kSubGroup;
  const int lane = threadIdx.x & 31, group = threadIdx.x / kSubGroup, first = threadIdx.x / 32 * kSubs;
  const bool lead = lane % kSubGroup == 0;
  const float s = prm.s;
  const int nb1 = h.nb1;
  uint32_t *ring = s_rings + group * kSubRingWords;
  for (int e0 = blockIdx.x * kGroups + first; e0 < h.qn; e0 += gridDim.x * kGroups) {  // warp-uniform
    const int e = e0 + (group - first);
    bool have = e < h.qn, run = false;
    int entry = 0, cand = 0, L2 = 0, net2 = 0, nq = 0, cutoff = 0, lo = 0, hi = 0, sum = 0;
    const uint32_t *qpl = db.words;
    bool self = false;
    if (have) {
      entry = rb.queue[cls][e];
      cand = score_mode ? rb.score_cands[entry] : entry;
      L2 = __ldg(db.len + cand);
      net2 = __ldg(db.net + cand);
      nq = (net2 + 31) >> 5;
      const int B = band_blocks(h.L1, L2, s);
      cutoff = cutoff_of(L2, s);
      qpl = db.words + __ldg(db.off + cand) + db.hw;
      self = cand == h.rep && !score_mode;
      const bool band = !self && B >= 0 && nb1 > 0 && nq > 0;
      run = band && wave_band(B, h.net1, net2, score_mode ? kNoCut : cutoff, lo, hi);
      if (run && !sub_holds(lo, hi, nb1)) have = run = false;  // the next pass takes it
      if (have && !score_mode && lead) {
        n.pairs++;
        n.cells += (unsigned long long)band_cells(B, nb1, net2);
        atomicAdd(s_qw, (unsigned long long)(nq * P));
      }
      if (self) sum = h.net1;
      if (band && !run) have = false;  // no chain can reach the cutoff
    }
    const int got = sub_any<P>(s_tab, nb1, qpl, run ? nq : 0, net2, lo, hi, score_mode ? kNoCut : cutoff, ring, n.done);
    if (run) sum = got;
    if (score_mode) {
      if (have && lead) rb.score_out[4 * entry + 2] = sum;
      continue;
    }
    bool pass = have && !(sum < cutoff) && sum >= 0;
    if (h.word_after) {  // short-word test (func.cu:376-396), a warp per member
      for (int k = 0; k < kSubs; k++) {
        const int src = k * kSubGroup;
        if (!__shfl_sync(kFullMask, (int)pass, src)) continue;
        const uint32_t *q = reinterpret_cast<const uint32_t *>(__shfl_sync(kFullMask, (unsigned long long)qpl, src));
        const int n2 = __shfl_sync(kFullMask, net2, src);
        const int ws = __shfl_sync(kFullMask, (int)self, src) ? max(0, n2 - prm.w + 1)
                                                              : word_count_warp_bits<P>(q, n2, prm.w, s_list);
        if (lane / kSubGroup == k) pass = !(ws < word_min(L2, prm.w, s));
      }
    }
    if (pass && lead) {
      rb.cluster[cand] = h.rep;
      rb.ident[cand] = sum;
      atomicAnd(&rb.alive[cand >> 5], ~(1u << (cand & 31)));
      n.members++;
    }
    __syncwarp();
  }
}

template <int P, int NW, int WMAX>
__global__ void __launch_bounds__(kAlignThreads, WMAX <= 2 ? 5 : 4)
    k_align_wave(DevDB db, RunBufs rb, RunParams prm, int cls, int score_mode, int warp_pairs, int few, int subs) {
  extern __shared__ __align__(16) uint32_t smem[];
  __shared__ uint64_t bar;
  __shared__ uint32_t s_xch[4 * NW];
  AlignHdr h;
  __shared__ unsigned long long s_qw;  // query plane words of the pairs taken (algorithmic bytes / 4)
  if (threadIdx.x == 0) s_qw = 0;
  constexpr int kWarps = kAlignThreads / 32;
  if (!align_setup<P>(db, rb, prm, cls, score_mode, warp_pairs, kWarps / NW, few, subs, smem, &bar, h)) return;
  const uint32_t *s_list = smem + ((h.nb1 * P + 3) & ~3);
  const uint32_t vlast = (h.net1 & 31) ? ((1u << (h.net1 & 31)) - 1u) : 0xFFFFFFFFu;
  uint32_t *s_tab = smem + wave_table_off(P, db.max_nb);
  uint32_t *s_rings = s_tab + wave_table_words(P, db.max_nb);
  wave_table<P>(smem, h.nb1, vlast, s_tab, threadIdx.x, kAlignThreads);
  __syncthreads();
  WaveCounts n;
  if (WMAX <= 2 && h.qn > subs) {
    sub_entries<P>(db, rb, prm, cls, score_mode, h, s_tab, s_rings, s_list, &s_qw, n);
    if (h.nb1 > 16 * kSubGroup) {  // bands too wide for 8 threads
      __syncthreads();
      wave_entries<P, 1, NW == 1 ? WMAX : 8, 2>(db, rb, prm, cls, score_mode, h, kAlignThreads / kSubGroup, s_tab, s_rings,
                                                s_list, s_xch, &s_qw, n);
    }
  } else if (NW == 1 || h.qn <= few) {
    wave_entries<P, NW, WMAX, -1>(db, rb, prm, cls, score_mode, h, kWarps / NW, s_tab, s_rings, s_list, s_xch, &s_qw, n);
  } else if constexpr (NW > 1) {
    constexpr int WW = WMAX == 1 ? 8 : 16;  // one word for each of 128 threads: 8 for 32 hold as much
    wave_entries<P, 1, WW, WMAX == 1 ? -1 : 1>(db, rb, prm, cls, score_mode, h, kWarps, s_tab, s_rings, s_list, s_xch,
                                               &s_qw, n);
    if (WMAX > 1 && h.nb1 > 32 * WW) {  // bands too wide for a warp
      __syncthreads();
      wave_entries<P, NW, WMAX, 0>(db, rb, prm, cls, score_mode, h, kWarps, s_tab, s_rings, s_list, s_xch, &s_qw, n);
    }
  }
  flush_align_stats(rb.st, cls, n.pairs, n.members, n.cells, n.done, &s_qw);
}

// Classes 0 and 1 with few pairs: 16 threads per pair, the query's blocks as
// rows.  Shared memory: rep planes | k-mer bitset | rep codes | a match table
// per warp.
template <int P>
__global__ void __launch_bounds__(kAlignThreads)
    k_align_query(DevDB db, RunBufs rb, RunParams prm, int cls, int score_mode, int warp_pairs) {
  extern __shared__ __align__(16) uint32_t smem[];
  __shared__ uint64_t bar;
  AlignHdr h;
  __shared__ unsigned long long s_qw;  // query plane words of the pairs taken (algorithmic bytes / 4)
  if (threadIdx.x == 0) s_qw = 0;
  constexpr int kGroups = kAlignThreads / kQueryGroup;
  if (!align_setup<P>(db, rb, prm, cls, score_mode, warp_pairs, kGroups, INT_MAX, INT_MAX, smem, &bar, h)) return;
  const uint32_t *s_pl = smem;
  const uint32_t *s_list = smem + ((h.nb1 * P + 3) & ~3);
  const int lane = threadIdx.x & 31, g = lane & (kQueryGroup - 1);
  uint32_t *s_codes = smem + wave_table_off(P, db.max_nb);
  uint32_t *tab = s_codes + 8 * db.max_nb + (threadIdx.x >> 5) * 32 * wave_codes(P);
  const int nb1 = h.nb1;
  for (int b = threadIdx.x; b < nb1; b += kAlignThreads) {
    uint32_t pl[P];
#pragma unroll
    for (int p = 0; p < P; p++) pl[p] = s_pl[b * P + p];
    wave_unpack<P>(pl, reinterpret_cast<uint4 *>(s_codes) + 2 * b);
  }
  __syncthreads();
  RunState *st = rb.st;
  const float s = prm.s;
  unsigned long long n_pairs = 0, n_members = 0, n_cells = 0, n_done = 0;
  const int e0 = (blockIdx.x * kAlignThreads + threadIdx.x) / 32 * 2;  // the warp's first two pairs
  for (int eb = e0; eb < h.qn; eb += (int)gridDim.x * kGroups) {       // warp-uniform
    const int e = eb + lane / kQueryGroup;
    const bool have = e < h.qn;
    int entry = 0, cand = 0, L2 = 0, net2 = 0, nq = 0, B = 0, cutoff = 0, lo = 0, hi = 0, sum = 0;
    const uint32_t *qpl = db.words;
    bool run = false, fails = false;
    if (have) {
      entry = rb.queue[cls][e];
      cand = score_mode ? rb.score_cands[entry] : entry;
      L2 = __ldg(db.len + cand);
      net2 = __ldg(db.net + cand);
      nq = (net2 + 31) >> 5;
      B = band_blocks(h.L1, L2, s);
      cutoff = cutoff_of(L2, s);
      qpl = db.words + __ldg(db.off + cand) + db.hw;
      if (B >= 0 && nb1 > 0 && nq > 0) {
        run = wave_band(B, h.net1, net2, score_mode ? kNoCut : cutoff, lo, hi);
        fails = !run;
      }
      if (!score_mode && g == 0) {
        n_pairs++;
        n_cells += (unsigned long long)band_cells(B, nb1, net2);
        atomicAdd(&s_qw, (unsigned long long)(nq * P));
      }
    }
    const int got = wave_query<P>(s_codes, nb1, h.net1, qpl, run ? nq : 0, net2, lo, hi, tab, n_done);
    if (run) sum = got;
    if (score_mode) {
      if (have && g == 0) rb.score_out[4 * entry + 2] = sum;
      continue;
    }
    bool pass = have && !fails && !(sum < cutoff);
    if (h.word_after) {  // short-word test (func.cu:376-396), a warp per member
      for (int k = 0; k < 2; k++) {
        const int src = k * kQueryGroup;
        if (!__shfl_sync(kFullMask, (int)pass, src)) continue;
        const uint32_t *q = reinterpret_cast<const uint32_t *>(__shfl_sync(kFullMask, (unsigned long long)qpl, src));
        const int n2 = __shfl_sync(kFullMask, net2, src);
        const int ws = word_count_warp_bits<P>(q, n2, prm.w, s_list);
        if (lane / kQueryGroup == k) pass = !(ws < word_min(L2, prm.w, s));
      }
    }
    if (pass && g == 0) {
      rb.cluster[cand] = h.rep;
      rb.ident[cand] = sum;
      atomicAnd(&rb.alive[cand >> 5], ~(1u << (cand & 31)));
      n_members++;
    }
  }
  flush_align_stats(st, cls, n_pairs, n_members, n_cells, n_done, &s_qw);
}

// ---- dispatch ---------------------------------------------------------------------
typedef void (*AlignFn)(DevDB, RunBufs, RunParams, int, int, int);

static const void *wave_fn(int type, int cls) {
  if (is_query_class(cls)) return type == 0 ? (const void *)k_align_query<2> : (const void *)k_align_query<5>;
  const int ring = class_ring(type, cls);
  if (type == 0)
    return ring == 64    ? (const void *)k_align_wave<2, 1, 2>
           : ring == 128 ? (const void *)k_align_wave<2, 4, 1>
                         : (const void *)k_align_wave<2, 4, 16>;
  return ring == 64    ? (const void *)k_align_wave<5, 1, 2>
         : ring == 128 ? (const void *)k_align_wave<5, 4, 1>
                       : (const void *)k_align_wave<5, 4, 16>;
}

// Pairs a CTA of the class's group-per-pair kernel takes at a time.
int wave_pairs_per_cta(int type, int cls) {
  return is_query_class(cls) ? kAlignThreads / kQueryGroup : class_ring(type, cls) == 64 ? kAlignThreads / 32 : 1;
}

static AlignFn align_fn(int type, int cls) {
  const int ring = class_ring(type, cls);
  if (type == 0) return ring == 64 ? k_align_tiled<2, 64> : ring == 128 ? k_align_tiled<2, 128> : k_align_tiled<2, 0>;
  return ring == 64 ? k_align_tiled<5, 64> : ring == 128 ? k_align_tiled<5, 128> : k_align_tiled<5, 0>;
}

// Dynamic shared memory: rep planes | k-mer bitset | row ring | match table
// (the group-per-pair kernels: rep planes | bitset | match table by code |
// code rings, or rep codes | match tables).
static size_t wave_smem(int type, int cls, int max_nb) {
  const int P = type ? 5 : 2;
  size_t words = (size_t)wave_table_off(P, max_nb);
  if (is_query_class(cls))
    words += 8 * (size_t)max_nb + kAlignThreads * wave_codes(P);
  else
    words += (size_t)wave_table_words(P, max_nb) + (size_t)(kAlignThreads / 32) * kWaveRingWords;
  return 4u * words;
}
// Records of up to this many bytes of shared memory per CTA take the
// group-per-pair kernels (proteins up to about 45,000 residues).
constexpr size_t kWaveSmemMost = 226 * 1024;
bool wave_fits(int type, int max_nb) { return wave_smem(type, base_class(type), max_nb) <= kWaveSmemMost; }
static size_t align_smem(int type, int max_nb, int cls) {
  const int P = type ? 5 : 2;
  size_t words = (size_t)tiled_eq_off(P, max_nb, class_ring(type, cls));
  if (P == 2) words += (size_t)eq_words(max_nb);
  return 4u * words;
}

// The dynamic shared memory limit is a property of the kernel on a device, not
// of a context: it only ever grows, so that a context opened on a database of
// shorter records cannot lower it beneath the launches of an open context on
// longer ones.
cudaError_t align_configure(int type, int max_nb) {
  static std::mutex mu;
  static int configured[64][2][2][kNumClasses] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(mu);
  for (int c = 0; c < num_classes(type); c++) {
    if (!class_used(type, c, max_nb)) continue;
    for (int wave = 0; wave < (wave_fits(type, max_nb) ? 2 : 1); wave++) {
      const int want = (int)(wave ? wave_smem(type, c, max_nb) : align_smem(type, max_nb, c));
      int &have = configured[dev][type ? 1 : 0][wave][c];
      if (want <= have) continue;
      e = cudaFuncSetAttribute(wave ? wave_fn(type, c) : (const void *)align_fn(type, c),
                               cudaFuncAttributeMaxDynamicSharedMemorySize, want);
      if (e != cudaSuccess) return e;
      have = want;
    }
  }
  return cudaSuccess;
}

// Resident CTAs per SM of class `cls` (persistent grid = that x SM count);
// wave: of its group-per-pair kernel.
int align_occupancy(int type, int cls, int max_nb, bool wave) {
  int nb = 0;
  const void *fn = wave ? wave_fn(type, cls) : (const void *)align_fn(type, cls);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, kAlignThreads,
                                                    wave ? wave_smem(type, cls, max_nb) : align_smem(type, max_nb, cls)) !=
      cudaSuccess)
    return 1;
  return nb < 1 ? 1 : nb;
}

int align_threads() { return kAlignThreads; }

// Launches class `cls`: the thread-per-pair kernel and the group-per-pair
// kernel; which of the two works is decided on the device from the class's
// queued pair count against the cut-off.  score_mode: 0 in clustering, else
// the pairs of a pair-score call.
cudaError_t launch_align(ngia_ctx *c, int cls, cudaStream_t s, int score_mode) {
  DevDB db = c->db;
  RunBufs rb = c->rb;
  RunParams prm = c->prm;
  // per length bucket (class): its own cut-off and CTA count when the tuner
  // chose them; pair scores go by the context's grids
  const int pairs = score_mode ? c->warp_pairs_default : c->warp_pairs;
  int wp = !score_mode && c->cls_warp_pairs[cls] >= 0 ? c->cls_warp_pairs[cls]
                                                      : group_cut(class_ring(c->db.type, cls), pairs);
  if (!wave_fits(c->db.type, c->cap_nb)) wp = -1;
  int grid = std::max(1, c->grid_align[cls] / std::max(1, c->cls_grid_div[cls]));
  int grid_wave = c->grid_wave[cls];
  if (score_mode) {  // no more CTAs than the call's pairs can use
    grid = std::min(grid, (score_mode + kAlignThreads - 1) / kAlignThreads);
    grid_wave = std::min(grid_wave, score_mode);
  }
  int few = wave_few(std::min(pairs, c->warp_pairs_default));
  const int ring = class_ring(c->db.type, cls);
  // (a batch member's smaller share does not move the four-pairs form: its
  // chain of iterations wants the latency of one pair per warp; 12 mixed jobs
  // 28.0 ms, 48.5 with it from the share on)
  const int share = c->batch_member ? c->warp_pairs_default : std::min(pairs, c->warp_pairs_default);
  int subs = ring && (c->db.P == 2 || score_mode) ? sub_from(c->db.P, ring == 128 ? 4 : 1, share) : INT_MAX;
  void *args[] = {&db, &rb, &prm, &cls, &score_mode, &wp, &few, &subs};
  // a call's pairs are known here: with no more than the cut-off no class can
  // go to the thread-per-pair kernel
  if (!score_mode || score_mode > wp) {
    cudaError_t e = cudaLaunchKernel((const void *)align_fn(c->db.type, cls), dim3(grid), dim3(kAlignThreads), args,
                                     align_smem(c->db.type, c->db.max_nb, cls), s);
    if (e != cudaSuccess) return e;
  }
  if (wp <= 0) return cudaSuccess;  // no class goes to the group kernel
  return cudaLaunchKernel(wave_fn(c->db.type, cls), dim3(grid_wave), dim3(kAlignThreads), args,
                          wave_smem(c->db.type, cls, c->db.max_nb), s);
}

}  // namespace ngia
