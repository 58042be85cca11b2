// assign.cuh — per-pair-representative filter and banded LCS over a set of
// representatives (a RepStore) and a query database, shared by the serving
// loop (serve.cu: resident representatives, first accepting one per query)
// and the speculative greedy rounds (spec.cu: the next K unclustered
// sequences as representatives, every accepting one per query as a bit
// mask).  The per-pair tests are the reference's (composition,
// func.cu:323-354; short words, 357-447; banded LCS, 450-604).
//
// The filters queue the pairs of one representative in groups of 32 entries
// that start at a multiple of 32, the last one padded: a warp of the
// alignment kernel takes a group, so its lanes share the representative and
// its match table lies in shared memory.  (With entries of several
// representatives in a warp the table was read from global memory through
// L1, several cache lines per load.  GB300, 20,000 DNA sequences to the end:
// 313 -> 287 ms, 250 with remainder tiles of even width.)
#pragma once
#include <stdint.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "kmer.cuh"
#include "tile.cuh"
#include "wave.cuh"

namespace ngia {
namespace {

// Pair classes: band windows <= 48 blocks, <= 112, wider, and queries of at
// most kQueryRows blocks with a window above 48 (the query's blocks are the
// rows then).
constexpr int kServeClasses = 4;
constexpr unsigned long long kNoRep = ~0ull;
constexpr int kCtlWords = 16;  // RoundBufs::ctl

// Device view of the resident representatives.
struct RepStore {
  const uint32_t *words;
  const int64_t *off;
  const int32_t *len, *net;
  const uint32_t *cnt;
  const uint32_t *lists;  // n x list_words k-mer bitsets (empty when net < 16)
  int32_t n, list_words;
  uint8_t *first;         // 1: the representative's short-word test goes before the alignment
};

// Buffers of the assignment rounds of one slot.
struct RoundBufs {
  int2 *queue[kServeClasses];  // (representative, query) pairs of a round, query -1 = padding
  uint32_t *ctl;               // [0..3] entries queued per class (groups of 32), [4..7] claimed,
                               // [8..11] pairs queued, [12] queries left, [13] error
  unsigned long long *key;     // per query: rep << 32 | score of the best accepting rep
  uint32_t *todo;              // bitmap of the queries not assigned yet
  unsigned long long *stats;   // [0] pairs aligned, [1] in-band cells computed
  int64_t cap;                 // entries per class queue
  // mask form (speculative rounds): every accepting representative is kept
  const int32_t *list;         // queries are positions in this list of sequences (null: sequences)
  unsigned long long *mask;    // per query: bit r = representative r accepts it
  int32_t *score;              // score of (r, q) at r * score_stride + q, for accepted pairs
  int64_t score_stride;
};
constexpr int kCtlClaimed = 4, kCtlPairs = 8, kCtlLeft = 12, kCtlErr = 13;

__host__ __device__ inline int serve_class(int A) { return A <= kSmallWindow ? 0 : A <= kWideWindow ? 1 : 2; }
__host__ __device__ inline int round_class(int A, int L2) {
  return A > kSmallWindow && L2 <= 32 * kQueryRows ? 3 : serve_class(A);
}
// Whether windows of up to max_nb blocks can put a pair in class c.
__host__ __device__ inline bool serve_class_used(int c, int max_nb, bool rounds) {
  return c == 0 || (max_nb > (c == 2 ? kWideWindow : kSmallWindow) && (c < 3 || rounds));
}

// k-mer presence bitset of every representative (the list of k_prep) and the
// order of its tests.
template <int P>
__global__ void k_rep_lists(RepStore rs, RunParams prm, uint32_t *lists) {
  __shared__ uint32_t s_list[kListWords];
  __shared__ int s_bits;
  const int r = blockIdx.x, w = prm.w;
  const int lw = rs.list_words;
  if (threadIdx.x == 0) s_bits = 0;
  for (int i = threadIdx.x; i < lw; i += blockDim.x) s_list[i] = 0;
  __syncthreads();
  const uint32_t *rec = rs.words + rs.off[r];
  const int net1 = (int)rec[1];
  if (net1 >= 16) {
    constexpr int bits = P == 2 ? 2 : 5;
    const uint32_t mask = (1u << (w * bits)) - 1u;
    const uint32_t *planes = rec + (P == 2 ? 6 : 30);
    for (int p = w - 1 + threadIdx.x; p < net1; p += blockDim.x) {
      uint32_t word = 0;
      for (int t = p - w + 1; t <= p; t++) word = (word << bits) | code_at<P>(planes, t);
      word &= mask;
      atomicOr(&s_list[word >> 5], 1u << (word & 31));
    }
  }
  __syncthreads();
  int bits_set = 0;
  for (int i = threadIdx.x; i < lw; i += blockDim.x) {
    lists[(int64_t)r * lw + i] = s_list[i];
    bits_set += __popc(s_list[i]);
  }
  if (bits_set) atomicAdd(&s_bits, bits_set);
  __syncthreads();
  if (threadIdx.x == 0) rs.first[r] = (uint8_t)word_first_of(P == 2 ? 0 : 1, prm, s_bits);
}

// Queues the survivors of one representative r among n_res tested queries of
// a CTA: s_res[k] = 0 or 1 + class of query q0 + k.  One reservation per class
// (whole groups of 32), then the entries and the padding.  Every thread of the
// CTA calls it after s_res and s_cnt (survivors per class) are complete.
__device__ __forceinline__ void queue_groups(const RoundBufs &rb, int r, int q0, int n_res, const uint8_t *s_res,
                                             const uint32_t *s_cnt, uint32_t *s_base, uint32_t *s_pos) {
  if (threadIdx.x < kServeClasses) {
    const uint32_t cnt = s_cnt[threadIdx.x], padded = (cnt + 31u) & ~31u;
    uint32_t base = 0;
    if (cnt) {
      base = atomicAdd(&rb.ctl[threadIdx.x], padded);
      atomicAdd(&rb.ctl[kCtlPairs + threadIdx.x], cnt);
    }
    s_base[threadIdx.x] = base;
    s_pos[threadIdx.x] = 0;
    for (uint32_t k = cnt; k < padded; k++)
      if ((int64_t)base + k < rb.cap) rb.queue[threadIdx.x][(int64_t)base + k] = make_int2(r, -1);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int k0 = (threadIdx.x >> 5) * 32; k0 < n_res; k0 += blockDim.x) {
    const int k = k0 + lane;
    const int res = k < n_res ? s_res[k] : 0;
    const unsigned pm = __ballot_sync(kFullMask, res != 0);
    if (!res) continue;
    const unsigned peers = __match_any_sync(pm, res);
    const int leader = __ffs(peers) - 1;
    uint32_t b = 0;
    if (lane == leader) b = atomicAdd(&s_pos[res - 1], (uint32_t)__popc(peers));
    b = __shfl_sync(peers, b, leader);
    const int64_t slot = (int64_t)s_base[res - 1] + b + __popc(peers & ((1u << lane) - 1u));
    if (slot < rb.cap) rb.queue[res - 1][slot] = make_int2(r, q0 + k);
  }
}

// One CTA per representative of the chunk and tile of kServeTile queries:
// composition test (and the short-word test in word-first order) for every
// unassigned query.  The outcomes lie in shared memory until they are queued,
// a byte each, so a batch of any size takes the same bounded amount.  (A byte
// per query of the whole batch had to be allowed for by each service's own
// size, and a batch of more than some 220,000 did not fit.)  A tile pads its
// last group of each class; batches of up to 65,536 queries have one tile.
// (Tiles in turn by one CTA cost services of a few queries 3%: 465 -> 478 us for
// five requests of up to three queries against 1,400 representatives.)
constexpr int kServeTile = 1 << 16;
// Entries of one representative and class for `left` queries in `tiles` tiles.
__host__ __device__ constexpr int64_t serve_entries(int64_t left, int64_t tiles) { return (left + 31 * tiles) & ~31ll; }
__host__ __device__ constexpr int64_t serve_tiles(int64_t n) { return (n + kServeTile - 1) / kServeTile; }
// Dynamic shared memory: the k-mer bitset, then a byte per query of a tile.
__host__ __device__ constexpr size_t serve_filter_smem(int list_words, int64_t n) {
  return 4 * (size_t)list_words + (size_t)(n < kServeTile ? (n + 31) & ~31ll : kServeTile);
}
template <int P>
__global__ void __launch_bounds__(256) k_serve_filter(DevDB qdb, RepStore rs, RunParams prm, RoundBufs rb, int r0) {
  extern __shared__ __align__(16) uint32_t s_list[];  // the representative's k-mer bitset, then per query of the tile:
  uint8_t *s_res = reinterpret_cast<uint8_t *>(s_list + rs.list_words);  // 0 = out, 1 + class
  __shared__ uint32_t s_rc[28], s_cnt[kServeClasses], s_base[kServeClasses], s_pos[kServeClasses];
  constexpr int A = P == 2 ? 4 : 28;
  const int r = r0 + blockIdx.x, q0 = blockIdx.y * kServeTile;
  const uint32_t *rec = rs.words + rs.off[r];
  if (threadIdx.x < A) s_rc[threadIdx.x] = rec[2 + threadIdx.x];
  if (threadIdx.x < kServeClasses) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  const int L1 = (int)rec[0], net1 = (int)rec[1], nb1 = (net1 + 31) / 32;
  const float s = prm.s;
  const bool word_here = !prm.precise && net1 >= 16 && rs.first[r];
  if (word_here) {
    for (int t = threadIdx.x; t < rs.list_words; t += blockDim.x) s_list[t] = rs.lists[(int64_t)r * rs.list_words + t];
    __syncthreads();
  }
  const int n = min(kServeTile, qdb.n - q0), nbw = (n + 31) / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int wi = warp; wi < nbw; wi += blockDim.x >> 5) {
    const uint32_t bits = rb.todo[q0 / 32 + wi];
    const int k = wi * 32 + lane, q = q0 + k;
    int res = 0;
    if ((bits >> lane) & 1u) {
      // a smaller representative of this round may already hold q
      const bool open = (rb.key[q] >> 32) > (unsigned long long)r;
      const int L2 = __ldg(qdb.len + q);
      const int cut = cutoff_of(L2, s);
      bool pass = open && !(base_sum<A>(qdb.cnt, q, s_rc) < cut);
      if (pass && word_here) {
        const int net2 = __ldg(qdb.net + q);
        if (net2 >= 16) pass = words_reach<P, 1>(qdb, q, net2, prm.w, word_min(L2, prm.w, s), KmerBits{s_list}, s_list);
      }
      if (pass) res = 1 + serve_class(window_need(L1, L2, cut, band_blocks(L1, L2, s), nb1));
    }
    if (k < n) s_res[k] = (uint8_t)res;
    const unsigned pm = __ballot_sync(kFullMask, res != 0);
    if (res) {
      const unsigned peers = __match_any_sync(pm, res);
      if (lane == __ffs(peers) - 1) atomicAdd(&s_cnt[res - 1], (uint32_t)__popc(peers));
    }
  }
  __syncthreads();
  queue_groups(rb, r, q0, n, s_res, s_cnt, s_base, s_pos);
}

// The filter's dynamic shared memory limit, the largest any service can need:
// it belongs to the kernel on the device, and is set once, so that no service
// changes it under another.
inline cudaError_t serve_filter_configure() {
  static std::mutex mu;
  static bool done[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(mu);
  if (done[dev]) return cudaSuccess;
  constexpr int most = (int)serve_filter_smem(kListWords, kServeTile);
  for (const void *fn : {(const void *)k_serve_filter<2>, (const void *)k_serve_filter<5>}) {
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e != cudaSuccess) return e;
  }
  done[dev] = true;
  return cudaSuccess;
}

// Whether the class's pairs of this round go to the group-per-pair kernel
// (few pairs) or to the thread-per-pair kernel.
__device__ __forceinline__ bool round_wave(const RoundBufs &rb, int cls, int wave_pairs) {
  return rb.ctl[kCtlPairs + cls] <= (uint32_t)wave_pairs;
}

// A pair's score reached its cutoff.  MASK = false: the query's key keeps the
// smallest accepting representative; MASK = true: one bit per representative.
template <bool MASK>
__device__ __forceinline__ void round_accept(const RoundBufs &rb, int r, int q, int sum) {
  if (MASK) {
    rb.score[(int64_t)r * rb.score_stride + q] = sum;
    atomicOr(&rb.mask[q], 1ull << r);
  } else {
    atomicMin(&rb.key[q], ((unsigned long long)r << 32) | (uint32_t)sum);
  }
}

// Representatives of up to this many blocks (8,192 residues) have their DNA
// match table in the warp's shared memory; longer ones are matched from their
// planes (one more operation per word).
constexpr int kRoundTable = 256;
__host__ __device__ constexpr int round_table_blocks(int max_nb) {
  return (max_nb < kRoundTable ? max_nb : kRoundTable) + kEqPad;
}

// Banded LCS of the queued pairs of one class, one thread per pair: the loop
// of k_align_tiled (align.cu) with a warp's 32 entries sharing their
// representative.  Class 3: the query's blocks are the rows and the
// representative's residues the columns (the band is symmetric), always from
// the planes.
template <int P, int RING, bool MASK, bool QROWS>
__global__ void __launch_bounds__(kAlignThreads, tiled_min_blocks(P))
    k_round_align(DevDB qdb, RepStore rs, RunParams prm, RoundBufs rb, int cls, int wave_pairs,
                  uint32_t *scratch, int64_t scratch_words, int ring_rows, int table_blocks) {
  extern __shared__ __align__(16) uint32_t smem[];
  __shared__ uint32_t s_qn;
  if (threadIdx.x == 0) s_qn = round_wave(rb, cls, wave_pairs) ? 0u : (uint32_t)min((int64_t)rb.ctl[cls], rb.cap);
  __syncthreads();
  const uint32_t qn = s_qn;
  if (qn == 0) return;
  using Ring = typename RingOf<RING>::T;
  Ring ring;
  if constexpr (RING > 0) {
    ring.base = smem + threadIdx.x;
  } else {
    const int64_t TL = (int64_t)gridDim.x * blockDim.x;
    if ((int64_t)ring_rows * TL > scratch_words) return;  // the host sizes the grid to the scratch
    ring.base = scratch + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    ring.stride = TL;
  }
  constexpr bool kTable = P == 2 && !QROWS;
  uint32_t *w_eq = smem + RING * kAlignThreads + (threadIdx.x >> 5) * 4 * table_blocks;  // this warp's match table
  const uint32_t w_eq_s = smem_u32(w_eq);
  (void)w_eq_s;
  // powers of two as values ptxas cannot fold (the FMA-pipe bookkeeping of tile.cuh)
  const uint32_t one_rt = 1u + (uint32_t)(qn == 0u);
  const FmaK fk(one_rt);
  (void)fk;
  const int lane = threadIdx.x & 31;
  const float s = prm.s;
  const int hw = qdb.hw;
  unsigned long long n_pairs = 0, n_cells = 0;
  int staged = -1, L1 = 0, net1 = 0, nb1 = 0;  // the warp's representative
  bool word_after = false;  // the short-word test follows the alignment
  const uint32_t *rpl = nullptr;
  bool table = false;
  for (;;) {
    uint32_t e0 = 0;
    if (lane == 0) e0 = atomicAdd(&rb.ctl[kCtlClaimed + cls], 32u);
    e0 = __shfl_sync(kFullMask, e0, 0);
    if (e0 >= qn) break;
    const int2 e = rb.queue[cls][e0 + lane];
    const int r = __shfl_sync(kFullMask, e.x, 0), q = e.y;
    if (r != staged) {
      const uint32_t *rrec = rs.words + rs.off[r];
      L1 = (int)rrec[0];
      net1 = (int)rrec[1];
      nb1 = (net1 + 31) >> 5;
      rpl = rrec + hw;
      word_after = !prm.precise && net1 >= 16 && !rs.first[r];
      staged = r;
      if constexpr (kTable) {
        table = nb1 + kEqPad <= table_blocks;
        if (table) {
          __syncwarp();
          for (int j = lane; j < nb1 + kEqPad; j += 32) {
            const bool real = j < nb1;
            const uint32_t p0 = real ? rpl[2 * j] : 0u, p1 = real ? rpl[2 * j + 1] : 0u;
            *reinterpret_cast<uint4 *>(w_eq + 4 * j) =
                make_uint4(real ? ~p0 & ~p1 : 0u, p0 & ~p1, ~p0 & p1, p0 & p1);
          }
          __syncwarp();
        }
      }
    }
    // rows (their planes rp, blocks nbr, residues nr) and columns (cp, nqc, nc)
    int L2 = 0, net2 = 0, B = 0, cutoff = 0;
    const uint32_t *qpl = nullptr;
    bool active = false;
    if (q >= 0 && (MASK || (rb.key[q] >> 32) > (unsigned long long)r)) {  // else a smaller representative holds q
      const int x = MASK ? rb.list[q] : q;
      L2 = __ldg(qdb.len + x);
      net2 = __ldg(qdb.net + x);
      B = band_blocks(L1, L2, s);
      cutoff = cutoff_of(L2, s);
      qpl = qdb.words + __ldg(qdb.off + x) + hw;
      active = B >= 0 && nb1 > 0 && net2 > 0;
      if (MASK && q == r) {  // a candidate against itself: the band holds the diagonal (align.cu)
        active = false;
        if (!(net1 < cutoff) && !(word_after && net1 - prm.w + 1 < word_min(L2, prm.w, s))) round_accept<MASK>(rb, r, q, net1);
      } else if (!active && !(0 < cutoff)) {
        round_accept<MASK>(rb, r, q, 0);  // no band: score 0
      }
    }
    const uint32_t *rp = QROWS ? qpl : rpl, *cp = QROWS ? rpl : qpl;
    const int nr = QROWS ? net2 : net1, nbr = (nr + 31) >> 5;
    const int nc = QROWS ? net1 : net2, ncb = (nc + 31) >> 5;
    const uint32_t vlast = (nr & 31) ? ((1u << (nr & 31)) - 1u) : 0xFFFFFFFFu;
    int i = 0, js = 0, je = 0, frozen = 0, zw = 0;
    uint32_t cur[P], nxt[P];
    if (active) {
      n_pairs++;
      je = band_first_top(B, nbr, nr, cutoff);
      ring.reset();
      for (int j = 0; j <= je; j++) ring[j] = 0xFFFFFFFFu;
#pragma unroll
      for (int p = 0; p < P; p++) cur[p] = __ldg(cp + p);
    }
    // the group's lanes in step, one column block at a time (at most kMaxBlocks)
    while (__any_sync(kFullMask, active)) {
      const int n = active ? je - js + 1 : 0;
      const int slots = (int)__reduce_max_sync(kFullMask, (unsigned)n);
      if (!active) continue;
      const int cols = min(32, nc - 32 * i);
      n_cells += (unsigned long long)n * cols * 32;
      if (i + 1 < ncb) {
#pragma unroll
        for (int p = 0; p < P; p++) nxt[p] = __ldg(cp + (i + 1) * P + p);
      }
      if constexpr (kTable)
        zw = table ? tile_block<P, true>(ring, w_eq_s, rp, js, je, nbr, slots, cols, cur, fk)
                   : tile_block<P, false>(ring, w_eq_s, rp, js, je, nbr, slots, cols, cur, fk);
      else
        zw = tile_block<P, false>(ring, w_eq_s, rp, js, je, nbr, slots, cols, cur, fk);
      i++;
      bool finished = i >= ncb;
      if (!finished) {
        const int step = band_advance(ring, i, B, nbr, nr, vlast, nc - 32 * i, cutoff, js, je, frozen, zw);
        if (step == kBandReject) {
          active = false;
          continue;
        }
        finished = step == kBandDone;
      }
      if (finished) {
        int sum = frozen;
        for (int j = js; j <= je; j++) sum += __popc(~ring[j] & (j == nbr - 1 ? vlast : 0xFFFFFFFFu));
        bool pass = !(sum < cutoff);
        if (pass && word_after && net2 >= 16)
          pass = !(word_count<P>(qpl, net2, prm.w, rs.lists + (int64_t)r * rs.list_words) < word_min(L2, prm.w, s));
        if (pass) round_accept<MASK>(rb, r, q, sum);
        active = false;
        continue;
      }
#pragma unroll
      for (int p = 0; p < P; p++) cur[p] = nxt[p];
    }
  }
  for (int o = 16; o; o >>= 1) {
    n_pairs += __shfl_down_sync(kFullMask, n_pairs, o);
    n_cells += __shfl_down_sync(kFullMask, n_cells, o);
  }
  if (lane == 0 && n_pairs) {
    atomicAdd(&rb.stats[0], n_pairs);
    atomicAdd(&rb.stats[1], n_cells);
  }
}

// One entry of the round by this thread's group (NW 1 or 4: 32 NW threads,
// rows are the representative's; NW -1: the same with 8 threads; NW 0: 16
// threads, the query's blocks as rows).  MINE: -1 all, 1 the bands that the
// group (a warp, NW -1: 8 threads) can hold, 0 those a warp cannot hold, 2 those
// 8 threads cannot hold.
struct RoundRep {
  int r = -1, L1 = 0, net1 = 0, nb1 = 0;
  bool word_after = false;  // the short-word test follows the alignment
};
template <int P, int NW, int WMAX, bool MASK, int MINE>
__device__ __forceinline__ void round_wave_entry(const DevDB &qdb, const RepStore &rs, const RunParams &prm,
                                                 const RoundBufs &rb, const RoundRep &h, int q, int cap_blocks,
                                                 uint32_t *smem, uint32_t *s_xch, unsigned long long &n_pairs,
                                                 unsigned long long &n_cells) {
  constexpr bool kQ = NW == 0, kSub = NW < 0;
  constexpr int GS = kQ ? kQueryGroup : kSub ? kSubGroup : 32 * NW, kParts = GS < 32 ? 32 / GS : 1;
  const int r = h.r, nb1 = h.nb1, net1 = h.net1, lane = threadIdx.x & 31;
  const bool lead = threadIdx.x % GS == 0;
  const float s = prm.s;
  int L2 = 0, net2 = 0, nq = 0, B = 0, cutoff = 1, lo = 0, hi = 0, sum = 0;
  const uint32_t *qpl = qdb.words;
  // (a key can change while the group's threads look at it: one answer)
  const bool self = MASK && q == r;  // a candidate against itself: the band holds the diagonal (align.cu)
  bool have = q >= 0 && (MASK || (rb.key[q] >> 32) > (unsigned long long)r), run = false;
  if constexpr (!MASK) {
    if constexpr (NW == 4)
      have = __syncthreads_or(have) != 0;
    else
      have = __shfl_sync(kFullMask, (int)have, 0, GS) != 0;
  }
  if (have) {
    const int x = MASK ? rb.list[q] : q;
    L2 = __ldg(qdb.len + x);
    net2 = __ldg(qdb.net + x);
    nq = (net2 + 31) >> 5;
    B = band_blocks(h.L1, L2, s);
    cutoff = cutoff_of(L2, s);
    qpl = qdb.words + __ldg(qdb.off + x) + qdb.hw;
    if (self) {
      sum = net1;
    } else if (B >= 0 && nb1 > 0 && nq > 0) {
      run = wave_band(B, net1, net2, cutoff, lo, hi);
      have = run;
    }
    if constexpr (MINE >= 0)
      if ((MINE == 1) ==
          (run && !(kSub || MINE == 2 ? sub_holds(lo, hi, nb1) : wave_holds(32, 16, lo, hi, nb1))))
        have = run = false;
    if (run && lead) n_pairs++;
  }
  unsigned long long cells = 0;
  if constexpr (kQ) {
    uint32_t *tab = smem + 8 * cap_blocks + (threadIdx.x >> 5) * 32 * wave_codes(P);
    const int got = wave_query<P>(smem, nb1, net1, qpl, run ? nq : 0, net2, lo, hi, tab, cells);
    if (run) sum = got;
  } else if constexpr (kSub) {
    uint32_t *ring = smem + wave_table_words(P, cap_blocks) + (threadIdx.x / GS) * kSubRingWords;
    const int got = sub_any<P>(smem, nb1, qpl, run ? nq : 0, net2, lo, hi, cutoff, ring, cells);
    if (run) sum = got;
  } else if (run) {  // uniform in the group
    uint32_t *ring = smem + wave_table_words(P, cap_blocks) + (threadIdx.x / GS) * kWaveRingWords;
    sum = wave_any<P, NW, WMAX>(smem, nb1, qpl, nq, net2, lo, hi, cutoff, ring, s_xch, cells);
  }
  n_cells += 32 * cells;
  bool pass = have && sum >= 0 && !(sum < cutoff);
  if (h.word_after) {  // short-word test (func.cu:376-396), a warp per member
    const uint32_t *list = rs.lists + (int64_t)r * rs.list_words;
#pragma unroll
    for (int k = 0; k < kParts; k++) {
      const int src = k * GS % 32;
      if (!__shfl_sync(kFullMask, (int)(pass && net2 >= 16), src)) continue;
      const uint32_t *qp = reinterpret_cast<const uint32_t *>(__shfl_sync(kFullMask, (unsigned long long)qpl, src));
      const int n2 = __shfl_sync(kFullMask, net2, src);
      const int ws = word_count_warp_bits<P>(qp, n2, prm.w, list);
      if (kParts == 1 || lane / GS == k) pass = !(ws < word_min(L2, prm.w, s));
    }
  }
  if (pass && lead) round_accept<MASK>(rb, r, q, sum);
}

// The same for classes with few pairs, a group of threads per pair (wave.cuh):
// NW as above; NW 4 is a warp per pair once there are more than `few` (align.cu).
// A CTA takes as many neighbouring entries as it has groups: they share their
// representative.
// Shared memory: match table | code rings, or rep codes | match tables.
template <int P, int NW, int WMAX, bool MASK>
__global__ void __launch_bounds__(kAlignThreads, NW == 0 ? 10 : WMAX <= 2 ? 5 : 4)
    k_round_wave(DevDB qdb, RepStore rs, RunParams prm, RoundBufs rb, int cls, int wave_pairs, int cap_blocks, int few,
                 int subs) {
  extern __shared__ __align__(16) uint32_t smem[];
  constexpr bool kQ = NW == 0;
  constexpr int GS = kQ ? kQueryGroup : 32 * NW, kGroups = kAlignThreads / GS, kWarps = kAlignThreads / 32;
  constexpr int WW = WMAX == 1 ? 8 : 16;
  __shared__ uint32_t s_xch[kQ ? 1 : 4 * NW];
  constexpr bool kSubOk = !kQ && WMAX <= 2;  // windows up to 112 blocks
  __shared__ uint32_t s_qn, s_many, s_subs;
  if (threadIdx.x == 0) {
    s_qn = round_wave(rb, cls, wave_pairs) ? (uint32_t)min((int64_t)rb.ctl[cls], rb.cap) : 0u;
    s_subs = kSubOk && rb.ctl[kCtlPairs + cls] > (uint32_t)subs;
    s_many = NW == 4 && rb.ctl[kCtlPairs + cls] > (uint32_t)few;
  }
  __syncthreads();
  const uint32_t qn = s_qn;
  const bool many = NW == 4 && s_many, sub = kSubOk && s_subs;
  const uint32_t per = sub ? kAlignThreads / kSubGroup : many ? kWarps : kGroups;
  const int hw = qdb.hw, lane = threadIdx.x & 31;
  unsigned long long n_pairs = 0, n_cells = 0;
  RoundRep h;
  for (uint32_t e0 = blockIdx.x * per; e0 < qn; e0 += gridDim.x * per) {
    const int2 first = rb.queue[cls][e0];  // entries of one group: the padding comes last
    if (first.y < 0) continue;             // CTA-uniform
    const int r = first.x;
    if (r != h.r) {
      __syncthreads();  // every group is through with the last representative
      const uint32_t *rrec = rs.words + rs.off[r];
      h.L1 = (int)rrec[0];
      h.net1 = (int)rrec[1];
      h.nb1 = (h.net1 + 31) >> 5;
      h.word_after = !prm.precise && h.net1 >= 16 && !rs.first[r];
      const uint32_t vlast = (h.net1 & 31) ? ((1u << (h.net1 & 31)) - 1u) : 0xFFFFFFFFu;
      if constexpr (kQ) {
        for (int b = threadIdx.x; b < h.nb1; b += kAlignThreads) {
          uint32_t pl[P];
#pragma unroll
          for (int p = 0; p < P; p++) pl[p] = rrec[hw + b * P + p];
          wave_unpack<P>(pl, reinterpret_cast<uint4 *>(smem) + 2 * b);
        }
      } else {
        wave_table<P>(rrec + hw, h.nb1, vlast, smem, threadIdx.x, kAlignThreads);
      }
      __syncthreads();
      h.r = r;
    }
    if constexpr (kSubOk) {
      if (sub) {
        const int q = rb.queue[cls][e0 + threadIdx.x / kSubGroup].y;
        round_wave_entry<P, -1, 16, MASK, 1>(qdb, rs, prm, rb, h, q, cap_blocks, smem, s_xch, n_pairs, n_cells);
        if (h.nb1 > 16 * kSubGroup) {  // bands too wide for 8 threads
          __syncthreads();
          for (int k = threadIdx.x >> 5; k < kAlignThreads / kSubGroup; k += kWarps)
            round_wave_entry<P, 1, NW == 1 ? WMAX : 8, MASK, 2>(qdb, rs, prm, rb, h, rb.queue[cls][e0 + k].y, cap_blocks,
                                                                smem, s_xch, n_pairs, n_cells);
          __syncthreads();
        }
        continue;
      }
    }
    if constexpr (NW == 4) {
      if (many) {
        const int q = rb.queue[cls][e0 + (threadIdx.x >> 5)].y;
        round_wave_entry<P, 1, WW, MASK, WMAX == 1 ? -1 : 1>(qdb, rs, prm, rb, h, q, cap_blocks, smem, s_xch, n_pairs,
                                                             n_cells);
        if (WMAX > 1 && h.nb1 > 32 * WW) {  // bands too wide for a warp
          __syncthreads();
          for (int k = 0; k < kWarps; k++)
            round_wave_entry<P, 4, WMAX, MASK, 0>(qdb, rs, prm, rb, h, rb.queue[cls][e0 + k].y, cap_blocks, smem, s_xch,
                                                  n_pairs, n_cells);
          __syncthreads();
        }
        continue;
      }
    }
    round_wave_entry<P, NW, WMAX, MASK, -1>(qdb, rs, prm, rb, h, rb.queue[cls][e0 + threadIdx.x / GS].y, cap_blocks,
                                            smem, s_xch, n_pairs, n_cells);
  }
  for (int o = 16; o; o >>= 1) {
    n_pairs += __shfl_down_sync(kFullMask, n_pairs, o);
    n_cells += __shfl_down_sync(kFullMask, n_cells, o);
  }
  if (lane == 0 && (n_pairs || n_cells)) {
    atomicAdd(&rb.stats[0], n_pairs);
    atomicAdd(&rb.stats[1], n_cells);
  }
}

// ---- launch ---------------------------------------------------------------------
using RoundAlignFn = void (*)(DevDB, RepStore, RunParams, RoundBufs, int, int, uint32_t *, int64_t, int, int);
using RoundWaveFn = void (*)(DevDB, RepStore, RunParams, RoundBufs, int, int, int, int, int);

template <int P, bool MASK>
RoundAlignFn round_align_fn(int cls) {
  switch (cls) {
    case 0: return k_round_align<P, 64, MASK, false>;
    case 1: return k_round_align<P, 128, MASK, false>;
    case 2: return k_round_align<P, 0, MASK, false>;
    default: return k_round_align<P, 64, MASK, true>;
  }
}
template <int P, bool MASK>
RoundWaveFn round_wave_fn(int cls) {
  switch (cls) {
    case 0: return k_round_wave<P, 1, 2, MASK>;
    case 1: return k_round_wave<P, 4, 1, MASK>;
    case 2: return k_round_wave<P, 4, 16, MASK>;
    default: return k_round_wave<P, 0, 1, MASK>;
  }
}

inline size_t round_align_smem(int type, int cls, int rep_nb) {
  const size_t ring = cls == 2 ? 0 : (size_t)(cls == 1 ? 128 : 64) * kAlignThreads;
  const size_t table = type == 0 && cls != 3 ? (size_t)(kAlignThreads / 32) * 4 * (size_t)round_table_blocks(rep_nb) : 0;
  return 4 * (ring + table);
}
inline size_t round_wave_smem(int type, int cls, int rep_nb) {
  const int P = type ? 5 : 2;
  return 4 * (cls == 3 ? 8 * (size_t)rep_nb + kAlignThreads * wave_codes(P)
                       : (size_t)wave_table_words(P, rep_nb) + (size_t)(kAlignThreads / 32) * kWaveRingWords);
}

// The alignment launches of a round: shapes for representatives of up to
// rep_nb blocks, and per class the pairs up to which a group per pair is
// faster (0: its kernel does not fit).
struct RoundPlan {
  int type = 0, rep_nb = 1;
  int grid[kServeClasses] = {0, 0, 0, 0}, wave_grid[kServeClasses] = {0, 0, 0, 0};
  int wave_pairs[kServeClasses] = {0, 0, 0, 0};
  int few = 0, subs[kServeClasses] = {0, 0, 0, 0};  // k_round_wave's
  uint32_t *scratch = nullptr;  // global ring of class 2
  int64_t scratch_words = 0;
  int ring_rows = 0;
};

template <bool MASK>
const void *round_fn(int type, int cls, bool wave) {
  if (wave) return type == 0 ? (const void *)round_wave_fn<2, MASK>(cls) : (const void *)round_wave_fn<5, MASK>(cls);
  return type == 0 ? (const void *)round_align_fn<2, MASK>(cls) : (const void *)round_align_fn<5, MASK>(cls);
}

// Kernel attributes (the dynamic shared memory limit only grows: launches of
// other open servers or contexts may need more) and grids.  The scratch is the
// caller's to allocate (scratch_words) and free; it has rows for the pairs that
// a round can queue (`pairs` at most), none where their number always takes
// the group-per-pair kernel.
template <bool MASK>
cudaError_t round_plan(RoundPlan &pl, int type, int rep_nb, int num_sms, int64_t pairs) {
  static std::mutex mu;
  static size_t have[64][2][2][kServeClasses] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  pl.type = type;
  pl.rep_nb = rep_nb;
  pl.few = wave_few(56 * num_sms);
  std::lock_guard<std::mutex> lock(mu);
  for (int c = 0; c < kServeClasses; c++)
    for (int wave = 0; wave < 2; wave++) {
      const void *fn = round_fn<MASK>(type, c, wave != 0);
      const size_t bytes = wave ? round_wave_smem(type, c, rep_nb) : round_align_smem(type, c, rep_nb);
      if (wave && bytes > 226 * 1024) continue;  // wave_pairs stays 0: a thread per pair
      size_t &h = have[dev][type ? 1 : 0][wave][c];
      if (bytes > h) {
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return e;
        h = bytes;
      }
      int occ = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kAlignThreads, bytes) != cudaSuccess || occ < 1) occ = 1;
      (wave ? pl.wave_grid : pl.grid)[c] = num_sms * occ;
      // the clustering kernels' cut-off (api.cu)
      if (wave) pl.subs[c] = type == 0 ? sub_from(2, c == 1 ? 4 : 1, 56 * num_sms) : INT_MAX;
      if (wave) pl.wave_pairs[c] = group_cut(c == 2 ? 0 : 64, 56 * num_sms);
    }
  pl.grid[2] = (int)std::min<int64_t>(pl.grid[2], std::max<int64_t>(1, (pairs + kAlignThreads - 1) / kAlignThreads));
  pl.ring_rows = global_rows(rep_nb);
  const bool rows = serve_class_used(2, rep_nb, MASK) && pairs > pl.wave_pairs[2];
  pl.scratch_words = rows ? (int64_t)pl.grid[2] * kAlignThreads * pl.ring_rows : 1;
  return cudaSuccess;
}

// Launches both kernels of every class the representatives' lengths allow;
// the round's pair counts decide on the device which of the two works.
template <bool MASK>
cudaError_t round_launch(const RoundPlan &pl, const DevDB &qdb, const RepStore &rs, const RunParams &prm,
                         const RoundBufs &rb, cudaStream_t st) {
  for (int c = 0; c < kServeClasses; c++) {
    if (!serve_class_used(c, pl.rep_nb, MASK)) continue;
    DevDB db = qdb;
    RepStore r = rs;
    RunParams p = prm;
    RoundBufs b = rb;
    int cls = c, wp = pl.wave_pairs[c], tb = round_table_blocks(pl.rep_nb), cap = pl.rep_nb, few = pl.few, subs = pl.subs[c];
    uint32_t *scr = pl.scratch;
    int64_t sw = pl.scratch_words;
    int rm = pl.ring_rows;
    void *args[] = {&db, &r, &p, &b, &cls, &wp, &scr, &sw, &rm, &tb};
    cudaError_t e = cudaLaunchKernel(round_fn<MASK>(pl.type, c, false), dim3(pl.grid[c]), dim3(kAlignThreads), args,
                                     round_align_smem(pl.type, c, pl.rep_nb), st);
    if (e != cudaSuccess) return e;
    if (wp <= 0) continue;
    void *wargs[] = {&db, &r, &p, &b, &cls, &wp, &cap, &few, &subs};
    e = cudaLaunchKernel(round_fn<MASK>(pl.type, c, true), dim3(pl.wave_grid[c]), dim3(kAlignThreads), wargs,
                         round_wave_smem(pl.type, c, pl.rep_nb), st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace
}  // namespace ngia
