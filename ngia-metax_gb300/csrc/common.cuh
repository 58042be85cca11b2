// common.cuh — device-side definitions shared by the loader, filter,
// alignment and driver kernels: the device database view, the run state,
// the work-queue classes, and the PTX wrappers for bulk (TMA) copies and
// bounded mbarrier waits.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ngia {

constexpr unsigned kFullMask = 0xFFFFFFFFu;
constexpr int kMaxLenDev = 65536;              // makeDB keeps records <= 65,536
constexpr int kMaxBlocks = kMaxLenDev / 32;    // 2048 plane blocks
constexpr int kListWords = 2048;               // rep k-mer presence bitset (65,536 bits)
constexpr int kRefGridThreads = 128 * 128;     // BLOCK*WARP of the reference launch

// Alignment work classes.  Pairs are queued by the width of the band window
// their alignment can need (window_need, in rep blocks): the last three
// classes of a type hold windows of up to 48 or 112 blocks (kSmallWindow,
// kWideWindow) in shared-memory rows, or of any width in global-memory rows.
// Classes 0 and 1 are the pairs of windows of 49 to 112 and of more blocks
// whose query has at most kQueryRows blocks: short queries against a long
// representative, aligned by 16 threads with the query's blocks as rows
// (wave.cuh) while they are few.
// DNA numbers 2 and 3 are unused, so that the last three classes keep their
// numbers.  Tunings and checkpoints saved when classes 0 and 1 (DNA: 0 to 3)
// were the narrowest windows are still taken: a cut-off of theirs then steers the
// short-query classes, and a resumed run's statistics add those up with the
// windows'.  Speed and statistics only.
constexpr int kNumClasses = 7;
constexpr int kQueryRows = 16;
constexpr int kSmallWindow = 48, kWideWindow = 112;
// Global-memory rows per lane: every rep block, and the padding of a lane at
// the last block whose warp's widest window is the whole representative.
__host__ __device__ constexpr int global_rows(int max_nb) { return 2 * max_nb + 16; }
__host__ __device__ inline int num_classes(int type) { return type == 0 ? 7 : 5; }
__host__ __device__ inline int generic_class(int type) { return num_classes(type) - 1; }
__host__ __device__ inline int base_class(int type) { return num_classes(type) - 3; }
// Classes 0 and 1: rows are the query's.
__host__ __device__ inline bool is_query_class(int c) { return c < 2; }
// Shared-memory rows of class c: 64, 128, or 0 (global-memory rows).
__host__ __device__ inline int class_ring(int type, int c) {
  if (is_query_class(c)) return c == 0 ? 128 : 0;
  return c >= generic_class(type) ? 0 : c == generic_class(type) - 1 ? 128 : 64;
}
// Whether a database whose records have up to max_nb blocks can queue pairs
// in class c.
__host__ __device__ inline bool class_used(int type, int c, int max_nb) {
  if (c >= num_classes(type) || (c >= 2 && c < base_class(type))) return false;
  const int ring = class_ring(type, c);
  return ring == 64 || max_nb > (ring == 128 ? kSmallWindow : kWideWindow);
}
// Pairs up to which a class takes its group-per-pair kernel, when those with
// rows in shared memory do up to `pairs` (api.cu): four times as many where
// the other kernel has its rows in global memory.  GB300, ms for 30,000
// proteins at s = 0.5 (two seeds) and 12 mixed jobs: 9.3, 7.4, 30.0 at the
// same, 9.6, 7.4, 30.6 at twice, 5.5, 4.8, 27.7 at four times, 5.4, 4.8, 28.9
// at eight times as many; four times for rows in shared memory too: 28.5, and
// 16 serving batches 28.1 -> 28.7.
__host__ __device__ constexpr int group_cut(int ring, int pairs) {
  return ring == 0 && pairs < (1 << 28) ? 4 * pairs : pairs;
}
// Parallel branch class c runs in: the two classes on the global ring share
// its scratch and run one after the other.
__host__ __device__ inline int class_stream(int type, int c) {
  return class_ring(type, c) == 0 ? generic_class(type) : c;
}
// The class of a pair whose window is A blocks and whose query has L2 (raw)
// residues.
__host__ __device__ inline int class_of(int type, int A, int L2) {
  if (A <= kSmallWindow) return base_class(type);
  if (L2 <= 32 * kQueryRows) return A <= kWideWindow ? 0 : 1;
  return base_class(type) + (A <= kWideWindow ? 1 : 2);
}

// Device copy of the makeDB database plus per-sequence header arrays.
struct DevDB {
  const uint32_t *words;  // records, contiguous (makeDB layout)
  const int64_t *off;     // word offset of record i
  const int32_t *len;     // raw length (record word 0)
  const int32_t *net;     // net length (record word 1)
  const uint32_t *cnt;    // residue counts, 4 (DNA) or 28 (protein) per sequence
  const uint32_t *codes;  // protein: each record's residue codes as a bit stream
                          // (5 words per 32-residue block, at the planes'
                          // offsets); null for DNA
  int32_t long_n;         // records before the first of at most kWarpWordLen residues (filter.cu)
  int32_t n, type;
  int32_t hw, P, A;       // header words, planes, count words
  int32_t max_nb;         // max plane blocks over all records
  int32_t has_short;      // some record has net length < 16
};

// Device-resident run state of the greedy driver.
struct RunState {
  int32_t rep;            // current representative (sorted index)
  int32_t done;           // no unclustered sequence left
  int32_t err;            // device error code (0 = ok)
  int32_t err_where;      // kernel id that set err
  int64_t iter;           // representatives taken so far
  int64_t iter_limit;     // graph loop stops when iter reaches it
  uint32_t qcount[kNumClasses];  // pairs queued per class this iteration
  uint32_t qhead[kNumClasses];   // pairs claimed per class
  uint32_t long_count;    // unused (the run state's layout is that of saved checkpoints)
  int32_t word_first;     // 1: short-word filter before alignment
  int32_t word_active;    // 1: short-word filter applies this iteration
  int32_t rep_nb;         // plane blocks of the representative (net)
  int32_t rep_len, rep_net;
  // statistics (device-accumulated)
  unsigned long long st_candidates, st_base_pass, st_align_pairs, st_members;
  unsigned long long st_band_cells, st_filter_bytes, st_word_checks, st_word_pass;
  unsigned long long st_done_cells;  // in-band cells actually computed
  unsigned long long st_class_pairs[kNumClasses];
  unsigned long long st_class_done[kNumClasses];    // in-band cells computed per class
  unsigned long long st_class_qwords[kNumClasses];  // query plane words of the pairs per class
};

// Polls of an mbarrier wait before a kernel gives up (each poll blocks for a
// hardware-defined interval; a staging copy lands within a few polls).
constexpr uint32_t kWaitPolls = 1u << 20;

// Run parameters (constant during one clustering).
struct RunParams {
  float s;
  int32_t w;
  int32_t precise;
  int32_t word_order;     // 0 auto, 1 word first, 2 alignment first
  int32_t refill;         // tiled alignment: idle lanes a warp waits for before it claims new pairs
  uint32_t wait_polls = kWaitPolls;  // poll limit of the alignment kernels' staging wait
  int32_t word_can = 0;   // auto order: some representative may put the short-word test first (word_can_pay)
};

// Order of the two cheap-to-expensive tests.  Both orders give the same
// members (a candidate joins iff all three tests pass).  A candidate needs
// about L2 (1 - w (1 - s)) of its words in the representative's set
// (word_min); unrelated ones have the set's share of all words.  So the
// short-word test rejects most candidates, and goes first, when that share is
// below what is needed, and hardly any above it.  GB300, 200,000 DNA of 1,450
// residues, w = 5, first representatives (1,950 residues, share 0.85): s =
// 0.95 (0.75 needed) 557 us per iteration with the test first, 450 after the
// alignment; s = 0.99 (0.95 needed) 231 against 317; 60,000 of 600 residues
// (share 0.44), s = 0.93 (0.65 needed) 81 against 130.
__host__ __device__ inline double word_need(const RunParams &prm) { return 1.0 - prm.w * (1.0 - (double)prm.s); }
__host__ __device__ inline double word_space(int type, int w) {  // words over the 4 or 20 residues
  double v = 1.0;
  for (int k = 0; k < w; k++) v *= type == 0 ? 4.0 : 20.0;
  return v;
}
// The representative's set holds `bits` words.
__host__ __device__ inline int word_first_of(int type, const RunParams &prm, int bits) {
  if (prm.word_order == 1) return 1;
  if (prm.word_order == 2) return 0;
  return prm.word_can && bits < word_need(prm) * word_space(type, prm.w);
}

// Device buffers of one clustering run.
struct RunBufs {
  RunState *st;
  int32_t *cluster;       // cluster[i] = representative of i, -1 = none yet
  int32_t *ident;         // banded-LCS score against the representative
  uint32_t *alive;        // bit i = sequence i not yet clustered
  int32_t *queue[kNumClasses];
  uint32_t *rep_rec;      // 16-byte aligned copy of the representative record
  uint32_t *rep_list;     // representative k-mer presence bitset
  // exact short-word path (databases with net length < 16 records)
  uint8_t *flags;         // per-sequence stage flags
  int32_t *pos;           // position of a base survivor in the job list
  int32_t *first_short;   // per reference thread: first job with net < 16
  uint32_t *scan_part;    // scan partials
  uint32_t *scratch;      // per-lane band rows of the widest class (global ring)
  int64_t scratch_words;
  int32_t generic_lanes;
  int32_t ring_rows;      // global-memory rows per lane: every rep block and a tile's padding
  // filter counters, 32 stripes x kFilterStats (one 64-byte line each),
  // added per CTA and folded into the run state by k_next
  unsigned long long *fstats;
  // pair-score mode
  const int32_t *score_cands;
  int32_t *score_out;
};

constexpr int kFilterStats = 8;     // counters per stripe (5 used)
constexpr int kFilterStripes = 32;

#define NGIA_ERR_MBAR_TIMEOUT 1
#define NGIA_ERR_SCRATCH 2
#define NGIA_ERR_RANGE 3

__device__ __forceinline__ void set_error(RunState *st, int code, int where) {
  if (atomicCAS(&st->err, 0, code) == 0) st->err_where = where;
}

// ---- PTX wrappers ---------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
// 1-D bulk copy global -> shared (the TMA unit, non-tensor form).  Both
// addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up after `limit` polls (each poll itself blocks for a
// hardware-defined interval) and returns false.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, uint32_t limit) {
  for (uint32_t i = 0; i < limit; i++)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// Stages `words` uint32 from global `src` (16-byte aligned) into shared `dst`
// with one bulk copy issued by thread 0; every thread waits on the barrier.
// Returns false (after recording an error) if the copy did not land.
__device__ __forceinline__ bool stage_to_smem(uint32_t *dst, const uint32_t *src, uint32_t words,
                                              uint64_t *bar, RunState *st, int where) {
  const uint32_t bytes = (words * 4u + 15u) & ~15u;
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    if (bytes) {
      mbar_expect_tx(bar, bytes);
      bulk_g2s(dst, src, bytes, bar);
    } else {
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
    }
  }
  __syncthreads();
  bool ok = mbar_wait_bounded(bar, 0, 1u << 20);
  if (!ok) {
    set_error(st, NGIA_ERR_MBAR_TIMEOUT, where);
    mbar_wait_bounded(bar, 0, 1u << 20);  // let the copy in flight land
  }
  return __syncthreads_and(ok);
}

// Block-band parameters of one (rep, query) pair, func.cu:469-470: the shift
// is ceil of one fused multiply-add (nvcc contracts (float)L1-(float)L2*s).
__device__ __forceinline__ int band_blocks(int L1, int L2, float s) {
  int shift = (int)ceilf(__fmaf_rn(-(float)L2, s, (float)L1));
  return (shift + 31) / 32;
}
// ceil((float)L2*s), func.cu:334, 515.
__device__ __forceinline__ int cutoff_of(int L2, float s) { return (int)ceilf(__fmul_rn((float)L2, s)); }
// Short-word threshold, func.cu:393-395.
__device__ __forceinline__ int word_min(int L2, int w, float s) {
  int length = (int)ceilf(__fmul_rn((float)L2, __fsub_rn(1.0f, s)));
  return (L2 - w + 1) - length * w;
}

// Window width (rep blocks per query block) of a pair's whole band.
__host__ __device__ __forceinline__ int window_of(int B, int nb1) {
  if (B < 0 || nb1 <= 0) return 0;
  int a = 2 * B + 1;
  return a < nb1 ? a : nb1;
}

// Widest window the alignment of a pair can need when only scores of at
// least `cut` matter: a chain of matches that reaches it leaves at most
// L2 - cut query and L1 - cut rep residues unmatched, so it stays between
// diagonals -(L2 - cut) and L1 - cut (rep position - query position); three
// blocks cover the ends of a 32-column step (band_advance in tile.cuh keeps
// every window within this).  Raw lengths bound the net ones.
__host__ __device__ __forceinline__ int window_need(int L1, int L2, int cut, int B, int nb1) {
  const int a = window_of(B, nb1);
  const int d = L2 > cut ? L2 - cut : 0, u = L1 > cut ? L1 - cut : 0;
  const int need = (d >> 5) + (u >> 5) + 3;
  return a < need ? a : need;
}

// Reference band cells of one pair: sum over query blocks of
// (jend - jstart + 1) * 32 * cols (func.cu:473-484).
__device__ __forceinline__ long long band_cells(int B, int nb1, int net2) {
  const int nq = (net2 + 31) / 32;
  long long c = 0;
  for (int i = 0; i < nq; i++) {
    int js = max(i - B, 0), je = min(i + B, nb1 - 1);
    if (je >= js) {
      int cols = ((i + 1) * 32 > net2) ? (net2 & 31) : 32;
      c += (long long)(je - js + 1) * 32 * cols;
    }
  }
  return c;
}

}  // namespace ngia
