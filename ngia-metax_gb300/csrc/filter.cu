// filter.cu — loader, per-representative preparation, the composition +
// short-word filter with work-queue compaction, and the next-representative
// reduction of the greedy driver.
//
// Reference counterparts (CUDA/signalNode/src/func.cu):
//   k_loader        readData device half (104-154): header arrays per sequence
//   k_prep          updateRepresent rep copy (213-235) + generateListGen/Pro (241-302)
//   k_filter, k_filter_word  kernel_baseFilterGen/Pro (323-354) and
//                   kernel_wordFilterGen/Pro (357-447) fused, survivors compacted on
//                   the device instead of updateJobs (305-320)
//   k_next          updateRepresent assignment/selection (190-215): the next
//                   representative is the first unclustered sequence
#include <algorithm>
#include <climits>
#include <mutex>

#include "../host/host_common.h"
#include "ctx.h"
#include "kmer.cuh"
#include "steps.cuh"

namespace ngia {

// The short-word test of longer candidates takes a warp (k_filter_word).
constexpr int kWarpWordLen = 2048;

// ---- loader ---------------------------------------------------------------
// from_end: n - the first record of at most kWarpWordLen residues.
__global__ void k_loader(const uint32_t *__restrict__ words, const int64_t *__restrict__ off, int64_t n_words,
                         int n, int type, int32_t *len, int32_t *net, uint32_t *cnt, int32_t *max_nb,
                         int32_t *has_short, int32_t *bad, int32_t *from_end) {
  const int A = type ? 28 : 4, hw = type ? 30 : 6, P = type ? 5 : 2;
  int local_max = 0, local_short = 0, local_bad = 0, local_end = 0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
    const int64_t o = off[c];
    if (o < 0 || o + hw > n_words) {
      local_bad = 1;
      len[c] = 0;
      net[c] = 0;
      continue;
    }
    const uint32_t *r = words + o;
    const uint32_t L = r[0], N = r[1];
    const int64_t need = hw + (int64_t)((L + 31) / 32) * P;
    if (L > (uint32_t)kMaxLenDev || N > L || o + need > n_words) {
      local_bad = 1;
      len[c] = 0;
      net[c] = 0;
      continue;
    }
    len[c] = (int32_t)L;
    net[c] = (int32_t)N;
    for (int a = 0; a < A; a++) cnt[(int64_t)c * A + a] = r[2 + a];
    local_max = max(local_max, (int)((N + 31) / 32));
    local_short |= (N < 16);
    if (L <= (uint32_t)kWarpWordLen) local_end = max(local_end, n - c);
  }
  atomicMax(max_nb, local_max);
  if (local_short) atomicOr(has_short, 1);
  if (local_bad) atomicOr(bad, 1);
  atomicMax(from_end, local_end);
}

// Protein residue-code streams, one warp per record (lanes over its
// blocks): each 32-residue block's five plane words become five stream
// words holding the block's residue codes (plane p = bit p of a code) as
// 5-bit groups, residue 0 at the top: residue j's code fills bits 155-5j ..
// 159-5j of the block's 160-bit value, whose bits 159..128 are stream word 0.
// Read across blocks, the stream holds every w-mer of the record in 5w
// contiguous bits with its last residue lowest, as the short-word test's
// rolling word holds it (func.cu:376-396).  Records the loader rejected have
// length 0 and are skipped.
__global__ void k_codes(const uint32_t *__restrict__ words, const int64_t *__restrict__ off,
                        const int32_t *__restrict__ len, int n, int hw, uint32_t *__restrict__ codes) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < n; c += nw) {
    const int nb = (len[c] + 31) >> 5;
    const int64_t base = off[c] + hw;
    for (int b = lane; b < nb; b += 32) {
      uint32_t pl[5], st[5];
#pragma unroll
      for (int p = 0; p < 5; p++) pl[p] = words[base + 5 * b + p];
      protein_stream(pl, st);
#pragma unroll
      for (int k = 0; k < 5; k++) codes[base + 5 * b + k] = st[k];
    }
  }
}

cudaError_t launch_loader(ngia_ctx *c, int32_t *d_maxnb, int32_t *d_short, int32_t *d_bad, int32_t *d_end) {
  int grid = c->num_sms * 4;
  k_loader<<<grid, 256, 0, c->stream>>>(c->d_words, c->d_off, c->n_words, c->db.n, c->db.type, c->d_len,
                                        c->d_net, c->d_cnt, d_maxnb, d_short, d_bad, d_end);
  if (c->db.type != 0 && c->d_codes)
    k_codes<<<grid, 256, 0, c->stream>>>(c->d_words, c->d_off, c->d_len, c->db.n, c->db.hw, c->d_codes);
  return cudaGetLastError();
}

// ---- run initialisation (initBench, func.cu:157-183) ------------------------
__global__ void k_init_run(DevDB db, RunBufs rb, RunParams prm) {
  const int n = db.n;
  const int nw = (n + 31) / 32;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    rb.cluster[i] = -1;
    rb.ident[i] = -1;
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nw; i += gridDim.x * blockDim.x) {
    const int rem = n - i * 32;
    rb.alive[i] = rem >= 32 ? 0xFFFFFFFFu : ((1u << rem) - 1u);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    RunState *st = rb.st;
    st->rep = 0;
    st->done = n == 0;
    st->err = 0;
    st->err_where = 0;
    st->iter = 0;
    st->iter_limit = LLONG_MAX;
    for (int k = 0; k < kNumClasses; k++) st->qcount[k] = st->qhead[k] = 0;
    st->long_count = 0;
    st->word_first = 0;
    st->word_active = 0;
    st->rep_nb = st->rep_len = st->rep_net = 0;
    st->st_candidates = st->st_base_pass = st->st_align_pairs = st->st_members = 0;
    st->st_band_cells = st->st_filter_bytes = st->st_word_checks = st->st_word_pass = 0;
    st->st_done_cells = 0;
    for (int k = 0; k < kFilterStripes * kFilterStats; k++) rb.fstats[k] = 0;
    for (int k = 0; k < kNumClasses; k++) st->st_class_pairs[k] = st->st_class_done[k] = st->st_class_qwords[k] = 0;
  }
}

cudaError_t launch_init_run(ngia_ctx *c) {
  k_init_run<<<c->num_sms * 2, 256, 0, c->stream>>>(c->db, c->rb, c->prm);
  return cudaGetLastError();
}

// ---- representative preparation ----------------------------------------------
// score_rep >= 0: pair-score mode for that representative (no run state
// change); otherwise the representative is st->rep (steps.cuh).
__global__ void k_prep(DevDB db, RunBufs rb, RunParams prm, int score_rep) { prep_body(db, rb, prm, score_rep); }

cudaError_t launch_prep(ngia_ctx *c, int score_rep) {
  k_prep<<<1, 512, 0, c->stream>>>(c->db, c->rb, c->prm, score_rep);
  return cudaGetLastError();
}

// Adds the filter counters of the calling CTA (every thread calls it) to one
// of kFilterStripes counter stripes; k_next folds the stripes into the run
// state.  One warp-level and one CTA-level reduction keep the global atomics
// at five per CTA, spread over 32 cache lines.
__device__ __forceinline__ void flush_stats(const RunBufs &rb, unsigned long long cand, unsigned long long base,
                                            unsigned long long bytes, unsigned long long wchk,
                                            unsigned long long wpass) {
  __shared__ unsigned long long s_acc[5];
  if (threadIdx.x < 5) s_acc[threadIdx.x] = 0;
  __syncthreads();
  for (int o = 16; o; o >>= 1) {
    cand += __shfl_down_sync(kFullMask, cand, o);
    base += __shfl_down_sync(kFullMask, base, o);
    bytes += __shfl_down_sync(kFullMask, bytes, o);
    wchk += __shfl_down_sync(kFullMask, wchk, o);
    wpass += __shfl_down_sync(kFullMask, wpass, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (cand) atomicAdd(&s_acc[0], cand);
    if (base) atomicAdd(&s_acc[1], base);
    if (bytes) atomicAdd(&s_acc[2], bytes);
    if (wchk) atomicAdd(&s_acc[3], wchk);
    if (wpass) atomicAdd(&s_acc[4], wpass);
  }
  __syncthreads();
  if (threadIdx.x < 5 && s_acc[threadIdx.x])
    atomicAdd(&rb.fstats[(blockIdx.x % kFilterStripes) * kFilterStats + threadIdx.x], s_acc[threadIdx.x]);
}

// Composition test over the unclustered set, one tile of 8 x WPW bitmap words
// per CTA pass: each warp takes WPW consecutive words; lanes read the header
// arrays of 32 consecutive sequences (coalesced).  Survivors are compacted
// into the alignment class queues in two levels: warp-aggregated shared-memory
// counters give each survivor its slot inside the tile, then one global atomic
// per class and tile reserves the tile's range, so the global queue counters
// see ~1/1,000 of the candidates.  `exact` = 1 records the survivors instead
// (bitmap in rb.flags) for the exact short-word path.
// Bitmap words per warp and tile pass, swept on GB300 (1M DNA s=0.85): fastest
// with 8 (fewer, fuller CTAs: 20.7 us vs 23.1 us with 4).
// (Issuing every header load of a warp's 8 bitmap words before the first
// use, unpredicated per lane, made the launch slower on GB300: 24.6 vs 18.1 us
// per iteration, 1M DNA s=0.85; predicated on the unclustered bit 24.2 against
// 17.8, 80 registers with spills against 57.)
constexpr int kFilterWords = 8;

// Both filters: whether this launch works, for a representative whose order is
// decided on the device (st->word_first).  turn 0: alignment-first ones only,
// 1: word-first ones only, -1: all.
struct FilterHead {
  int skip, L1, nb1, word;
};
__device__ __forceinline__ FilterHead filter_head(const RunState *st, int exact, int turn) {
  FilterHead h;
  h.word = (!exact && st->word_first && st->word_active) ? 1 : 0;
  h.skip = st->done || st->iter >= st->iter_limit || st->err || (turn >= 0 && turn != h.word);
  h.L1 = st->rep_len;
  h.nb1 = st->rep_nb;
  return h;
}

template <int P, int WPW>
__global__ void __launch_bounds__(256) k_filter(DevDB db, RunBufs rb, RunParams prm, int exact, int turn) {
  RunState *st = rb.st;
  __shared__ uint32_t s_rc[28];
  __shared__ FilterHead h;
  __shared__ uint32_t s_cnt[kNumClasses], s_base[kNumClasses];
  constexpr int A = P == 2 ? 4 : 28;
  if (threadIdx.x == 0) h = filter_head(st, exact, turn);
  if (threadIdx.x < A) s_rc[threadIdx.x] = rb.rep_rec[2 + threadIdx.x];
  __syncthreads();
  if (h.skip) return;
  const int L1 = h.L1, nb1 = h.nb1;
  const float s = prm.s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nbw = (db.n + 31) / 32;
  const int tiles = (nbw + 8 * WPW - 1) / (8 * WPW);
  unsigned long long cand = 0, base = 0, bytes = 0;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    if (threadIdx.x < kNumClasses) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    // The warp's bitmap words first, then every header load of all its
    // words (independent of one another), then the compaction.
    const int w0 = (tile * 8 + warp) * WPW;
    int slot[WPW], cls_of[WPW];
    uint32_t bits_of[WPW];
#pragma unroll
    for (int k = 0; k < WPW; k++) bits_of[k] = w0 + k < nbw ? rb.alive[w0 + k] : 0u;
    unsigned pass_of = 0;  // bit k: this lane's candidate of word k survives
#pragma unroll
    for (int k = 0; k < WPW; k++) {
      cls_of[k] = 0;
      const uint32_t bits = bits_of[k];
      if (!bits) continue;  // warp-uniform
      const int c = (w0 + k) * 32 + lane;
      if ((bits >> lane) & 1u) {
        cand++;
        bytes += 4 * (2 + A);
        const int L2 = __ldg(db.len + c), cut = cutoff_of(L2, s);
        if (!(base_sum<A>(db.cnt, c, s_rc) < cut)) {
          base++;
          pass_of |= 1u << k;
          if (!exact) cls_of[k] = class_of(db.type, window_need(L1, L2, cut, band_blocks(L1, L2, s), nb1), L2);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < WPW; k++) {
      slot[k] = -1;
      if (w0 + k >= nbw) continue;  // warp-uniform
      const bool pass = (pass_of >> k) & 1u;
      const unsigned pm = __ballot_sync(kFullMask, pass);
      if (exact) {
        if (lane == 0) reinterpret_cast<uint32_t *>(rb.flags)[w0 + k] = pm;
        continue;
      }
      if (pass) {
        const int cls = cls_of[k];
        const unsigned peers = __match_any_sync(pm, cls);
        const int leader = __ffs(peers) - 1;
        uint32_t b = 0;
        if (lane == leader) b = atomicAdd(&s_cnt[cls], (uint32_t)__popc(peers));
        b = __shfl_sync(peers, b, leader);
        slot[k] = (int)(b + __popc(peers & ((1u << lane) - 1u)));
      }
    }
    __syncthreads();
    if (threadIdx.x < kNumClasses)
      s_base[threadIdx.x] = s_cnt[threadIdx.x] ? atomicAdd(&st->qcount[threadIdx.x], s_cnt[threadIdx.x]) : 0u;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < WPW; k++)
      if (slot[k] >= 0) rb.queue[cls_of[k]][s_base[cls_of[k]] + (uint32_t)slot[k]] = (w0 + k) * 32 + lane;
  }
  flush_stats(rb, cand, base, bytes, 0, 0);
}

// ---- composition and short-word test -------------------------------------------
// Launches that may put the short-word test first.  The work per candidate
// grows with its length, so warps run independently — each takes every W-th
// bitmap word of the length-sorted database, a CTA's warps words gridDim.x
// apart (a share of every length for each SM) — and queues its survivors with
// one atomic per class and word; no CTA barrier makes a warp wait for the CTA's
// longest candidates.  The records before the first of at most kWarpWordLen
// residues (db.long_n; the longest share the first bitmap words) get a warp
// each, from the grid's last warp on, which has the fewest words to do; a longer
// record further on (a database that is not sorted) gets its lane's warp.  (A
// launch of their own behind this one took 10 us of a 119 us iteration of
// 100,000 proteins.)
//
// GB300, 200,000 DNA of 1,450 residues, w = 5, the whole filter per iteration:
// s = 0.99 42 us (a byte per word and every word counted: 151), s = 0.97 77
// (153); the first iterations of 100,000 proteins of 20 to 6,600 residues,
// w = 3, s = 0.9: 44 us with cold caches (72), the longest candidate of a warp
// and the composition counts; the table of w = 3 allows one word per lookup.
// Two CTAs of 512 threads per SM: one of 1,024 waits for a whole SM when other
// jobs share the GPU (12 mixed jobs 2% slower), 256 threads build the table
// too often (s = 0.97 102 us), 40 registers for three CTAs of 512 spill (90 us).
// kWarpWordLen: 1,024 is no faster, 512 makes the proteins 25% slower.
constexpr int kWordThreads = 512, kWordCtas = 2;

// Shared memory: k-mer bitset | lookup table (word_table_bytes).
template <int P, int M>
__global__ void __launch_bounds__(kWordThreads, kWordCtas)
    k_filter_word(DevDB db, RunBufs rb, RunParams prm, int turn) {
  RunState *st = rb.st;
  extern __shared__ __align__(16) uint32_t s_list[];
  __shared__ uint64_t bar;
  __shared__ uint32_t s_rc[28];
  __shared__ FilterHead h;
  constexpr int A = P == 2 ? 4 : 28;
  if (threadIdx.x == 0) h = filter_head(st, 0, turn);
  if (threadIdx.x < A) s_rc[threadIdx.x] = rb.rep_rec[2 + threadIdx.x];
  __syncthreads();
  if (h.skip) return;
  const int L1 = h.L1, nb1 = h.nb1, word_here = h.word;
  const uint32_t list_words = list_words_of(db.type, prm.w);
  uint8_t *s_tab = reinterpret_cast<uint8_t *>(s_list + list_words);
  if (word_here) {
    if (!stage_to_smem(s_list, rb.rep_list, list_words, &bar, st, 1)) return;
    build_word_table<P, M>(s_tab, s_list, prm.w);
  }
  const float s = prm.s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nbw = (db.n + 31) / 32;
  // 32 bits: a candidate is at most 41 KB (a protein of 65,536 residues), and a
  // thread sees at most 13,800 of the bitmap's words' (2^31 records, 4,864
  // warps) besides its warp's share of the long records, which fit the device
  uint32_t cand = 0, base = 0, bytes = 0, wpass = 0;
  const int W = gridDim.x * (blockDim.x >> 5), gw = warp * gridDim.x + blockIdx.x;
  const int n_long = word_here ? db.long_n : 0;
  for (int c = W - 1 - gw; c < n_long; c += W) {  // a warp per record
    if (!((rb.alive[c >> 5] >> (c & 31)) & 1u)) continue;
    const int L2 = __ldg(db.len + c), net2 = __ldg(db.net + c), cut = cutoff_of(L2, s);
    const bool comp = !(base_sum<A>(db.cnt, c, s_rc) < cut);
    if (lane == 0) {
      cand++;
      base += comp;
      bytes += 4 * (2 + A) + (comp ? 4 * P * ((net2 + 31) / 32) : 0);
    }
    if (!comp) continue;  // warp-uniform
    const bool pass = words_reach_warp<P, M>(db, c, net2, prm.w, word_min(L2, prm.w, s), s_tab, s_list) && lane == 0;
    if (pass) wpass++;
    push_queue(rb, st, pass, pass ? class_of(db.type, window_need(L1, L2, cut, band_blocks(L1, L2, s), nb1), L2) : 0, c);
  }
  for (int wi = gw; wi < nbw; wi += W) {
    const uint32_t bits = rb.alive[wi];
    if (!bits) continue;  // warp-uniform
    const int c = wi * 32 + lane;
    bool pass = false, deferred = false;
    int cls = 0;
    if (((bits >> lane) & 1u) && c >= n_long) {
      cand++;
      bytes += 4 * (2 + A);
      const int L2 = __ldg(db.len + c), cut = cutoff_of(L2, s);
      pass = !(base_sum<A>(db.cnt, c, s_rc) < cut);
      if (pass) {
        base++;
        if (word_here) {
          const int net2 = __ldg(db.net + c);
          bytes += 4 * P * ((net2 + 31) / 32);
          deferred = net2 > kWarpWordLen;
          if (!deferred) {
            pass = words_reach<P, M>(db, c, net2, prm.w, word_min(L2, prm.w, s), s_tab, s_list);
            if (pass) wpass++;
          }
        }
      }
      if (pass) cls = class_of(db.type, window_need(L1, L2, cut, band_blocks(L1, L2, s), nb1), L2);
    }
    for (unsigned dm = __ballot_sync(kFullMask, deferred); dm; dm &= dm - 1) {
      const int src = __ffs(dm) - 1, cc = wi * 32 + src;
      const bool reach = words_reach_warp<P, M>(db, cc, __ldg(db.net + cc), prm.w, word_min(__ldg(db.len + cc), prm.w, s),
                                                s_tab, s_list);
      if (lane == src) {
        pass = reach;
        if (pass) wpass++;
      }
    }
    push_queue(rb, st, pass, cls, c);
  }
  flush_stats(rb, cand, base, bytes, word_here ? base : 0, wpass);
}

// ---- exact short-word path ---------------------------------------------------
// For databases holding records with net length < 16 the reference's word
// kernel returns a whole thread at such a job (func.cu:375, 420), so whether
// a job is tested depends on its position p in the compacted job list and on
// the 16,384-thread map p -> p mod 16384.  These kernels reproduce that: the
// base-survivor bitmap (rb.flags as uint32 words) is prefix-counted to give p,
// first_short[t] is the first position of thread t holding a short query,
// and a job at p >= first_short[p mod 16384] passes untested.
__global__ void k_scan_words(const uint32_t *bm, int nbw, uint32_t *prefix) {
  // single CTA of 1024 threads: exclusive prefix of popcounts
  __shared__ uint32_t s_part[1024];
  const int per = (nbw + 1023) / 1024;
  const int b = threadIdx.x * per, e = min(nbw, b + per);
  uint32_t acc = 0;
  for (int i = b; i < e; i++) acc += __popc(bm[i]);
  s_part[threadIdx.x] = acc;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    uint32_t v = threadIdx.x >= o ? s_part[threadIdx.x - o] : 0;
    __syncthreads();
    s_part[threadIdx.x] += v;
    __syncthreads();
  }
  uint32_t run = threadIdx.x ? s_part[threadIdx.x - 1] : 0;
  for (int i = b; i < e; i++) {
    prefix[i] = run;
    run += __popc(bm[i]);
  }
}

__global__ void k_first_short(DevDB db, RunBufs rb, int reset) {
  const int nbw = (db.n + 31) / 32;
  const uint32_t *bm = reinterpret_cast<const uint32_t *>(rb.flags);
  if (reset) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < kRefGridThreads; t += gridDim.x * blockDim.x)
      rb.first_short[t] = INT_MAX;
    return;
  }
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nbw * 32; c += gridDim.x * blockDim.x) {
    if (c >= db.n) break;
    const uint32_t w = bm[c >> 5];
    if (!((w >> (c & 31)) & 1u)) continue;
    if (db.net[c] >= 16) continue;
    const int p = (int)(rb.scan_part[c >> 5] + __popc(w & ((1u << (c & 31)) - 1u)));
    atomicMin(&rb.first_short[p % kRefGridThreads], p);
  }
}

template <int P>
__global__ void __launch_bounds__(256) k_word_exact(DevDB db, RunBufs rb, RunParams prm) {
  RunState *st = rb.st;
  extern __shared__ __align__(16) uint32_t s_list[];
  __shared__ uint64_t bar;
  __shared__ int s_hdr[3];
  if (threadIdx.x == 0) {
    s_hdr[0] = st->done || st->iter >= st->iter_limit || st->err;
    s_hdr[1] = st->rep_len;
    s_hdr[2] = st->rep_nb;
  }
  __syncthreads();
  if (s_hdr[0]) return;
  const int L1 = s_hdr[1], nb1 = s_hdr[2];
  const int list_words = max(1, (int)((1u << (prm.w * (P == 2 ? 2 : 5))) / 32u));
  if (!stage_to_smem(s_list, rb.rep_list, (uint32_t)list_words, &bar, st, 2)) return;
  const uint32_t *bm = reinterpret_cast<const uint32_t *>(rb.flags);
  const int lane = threadIdx.x & 31;
  const int nbw = (db.n + 31) / 32;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  unsigned long long bytes = 0, wchk = 0, wpass = 0;
  for (int wi = gw; wi < nbw; wi += nwarps) {
    const uint32_t w = bm[wi];
    if (!w) continue;
    const int c = wi * 32 + lane;
    bool pass = (w >> lane) & 1u;
    int cls = 0;
    if (pass) {
      const int p = (int)(rb.scan_part[wi] + __popc(w & ((1u << lane) - 1u)));
      const bool skipped = p >= rb.first_short[p % kRefGridThreads];
      const int L2 = db.len[c];
      if (!skipped) {
        const int net2 = db.net[c];
        const uint32_t *planes = db.words + db.off[c] + db.hw;
        wchk++;
        bytes += 4ull * P * ((net2 + 31) / 32);
        pass = !(word_count<P>(planes, net2, prm.w, s_list) < word_min(L2, prm.w, prm.s));
      }
      if (pass) {
        wpass++;
        cls = class_of(db.type, window_need(L1, L2, cutoff_of(L2, prm.s), band_blocks(L1, L2, prm.s), nb1), L2);
      }
    }
    push_queue(rb, st, pass, cls, c);
  }
  flush_stats(rb, 0, 0, bytes, wchk, wpass);
}

using FilterFn = void (*)(DevDB, RunBufs, RunParams, int, int);
using WordFn = void (*)(DevDB, RunBufs, RunParams, int);
static WordFn word_fn(int type, int M) {
  if (type) return M == 2 ? k_filter_word<5, 2> : k_filter_word<5, 1>;
  return M == 4 ? k_filter_word<2, 4> : M == 2 ? k_filter_word<2, 2> : k_filter_word<2, 1>;
}
static size_t word_smem(int type, int w) {
  return 4 * (size_t)list_words_of(type, w) + word_table_bytes(type, w, words_per_lookup(type, w));
}

cudaError_t filter_configure() {
  constexpr size_t most = 72 * 1024;  // DNA w = 8: 8 KB bitset, 64 KB table
  static std::mutex mu;
  static bool done[64] = {};
  int dev = 0;
  cudaError_t d = cudaGetDevice(&dev);
  if (d != cudaSuccess) return d;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(mu);
  if (done[dev]) return cudaSuccess;
  for (int type = 0; type < 2; type++)
    for (int M = 1; M <= (type ? 2 : 4); M *= 2) {
      cudaError_t e = cudaFuncSetAttribute((const void *)word_fn(type, M), cudaFuncAttributeMaxDynamicSharedMemorySize, most);
      if (e != cudaSuccess) return e;
    }
  done[dev] = true;
  return cudaSuccess;
}

cudaError_t launch_filter(ngia_ctx *c) {
  const int type = c->db.type, P = c->db.P;
  // Exact path only matters when the short-word filter can run and some
  // record is shorter than 16 residues.
  const bool exact = c->db.has_short && !c->prm.precise;
  const int nbw = (c->db.n + 31) / 32;
  const bool small = !exact && c->filter_tile == 1;  // the tuner's choice: one bitmap word per warp and tile
  const int per = 8 * (small ? 1 : kFilterWords);
  const int grid = std::max(1, std::min(c->grid_filter, (nbw + per - 1) / per));
  const FilterFn fn = P == 2 ? (small ? k_filter<2, 1> : k_filter<2, kFilterWords>)
                             : (small ? k_filter<5, 1> : k_filter<5, kFilterWords>);
  if (!exact) {
    // The filter with the short-word test, the one without, or (automatic
    // order, when either may be wanted) both: the representative's order
    // decides on the device which works.
    const bool word = c->prm.word_order == 1 || (c->prm.word_order == 0 && c->prm.word_can);
    const int turn = c->prm.word_order == 0 && c->prm.word_can ? 1 : -1;
    if (word) {
      const int M = words_per_lookup(type, c->prm.w);
      const size_t smem = word_smem(type, c->prm.w);
      const int grid_w = std::max(1, std::min(std::min(c->grid_filter, kWordCtas * c->num_sms), (nbw + 7) / 8));
      word_fn(type, M)<<<grid_w, kWordThreads, smem, c->stream>>>(c->db, c->rb, c->prm, turn);
    }
    if (!word || turn >= 0) fn<<<grid, 256, 0, c->stream>>>(c->db, c->rb, c->prm, 0, turn >= 0 ? 0 : -1);
    return cudaGetLastError();
  }
  const size_t smem = 4 * (size_t)list_words_of(type, c->prm.w);
  fn<<<grid, 256, 0, c->stream>>>(c->db, c->rb, c->prm, 1, -1);
  k_scan_words<<<1, 1024, 0, c->stream>>>(reinterpret_cast<const uint32_t *>(c->rb.flags), nbw, c->rb.scan_part);
  k_first_short<<<64, 256, 0, c->stream>>>(c->db, c->rb, 1);
  k_first_short<<<c->num_sms * 2, 256, 0, c->stream>>>(c->db, c->rb, 0);
  if (P == 2)
    k_word_exact<2><<<c->grid_filter, 256, smem, c->stream>>>(c->db, c->rb, c->prm);
  else
    k_word_exact<5><<<c->grid_filter, 256, smem, c->stream>>>(c->db, c->rb, c->prm);
  return cudaGetLastError();
}

// ---- next representative (steps.cuh) ----------------------------------------
__global__ void k_next(DevDB db, RunBufs rb, unsigned long long cond, int use_cond) {
  next_body(db, rb, cond, use_cond);
}


// Start of a run over a subset of the sequences (the unclustered set was
// loaded into rb.alive): the first member of the subset is the first
// representative; an empty subset is done at once.
__global__ void k_subset_start(DevDB db, RunBufs rb) {
  RunState *st = rb.st;
  __shared__ int s_min[32];
  const int nbw = (db.n + 31) / 32;
  int v = INT_MAX;
  for (int wi = threadIdx.x; wi < nbw; wi += blockDim.x)
    if (rb.alive[wi]) {
      v = wi;
      break;
    }
  for (int o = 16; o; o >>= 1) v = min(v, __shfl_xor_sync(kFullMask, v, o));
  if ((threadIdx.x & 31) == 0) s_min[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    int u = threadIdx.x < (int)(blockDim.x >> 5) ? s_min[threadIdx.x] : INT_MAX;
    for (int o = 16; o; o >>= 1) u = min(u, __shfl_xor_sync(kFullMask, u, o));
    if (threadIdx.x == 0) {
      if (u == INT_MAX) {
        st->done = 1;
      } else {
        st->rep = u * 32 + __ffs(rb.alive[u]) - 1;
        st->done = 0;
      }
    }
  }
}

cudaError_t launch_subset_start(ngia_ctx *c, const uint32_t *d_alive) {
  const int nbw = (c->db.n + 31) / 32;
  cudaError_t e = cudaMemcpyAsync(c->rb.alive, d_alive, sizeof(uint32_t) * (size_t)nbw, cudaMemcpyDeviceToDevice,
                                  c->stream);
  if (e != cudaSuccess) return e;
  k_subset_start<<<1, 1024, 0, c->stream>>>(c->db, c->rb);
  return cudaGetLastError();
}

cudaError_t launch_next(ngia_ctx *c, unsigned long long cond, int use_cond) {
  k_next<<<1, 1024, 0, c->stream>>>(c->db, c->rb, cond, use_cond);
  return cudaGetLastError();
}

// ---- pair-score mode: per-pair composition / word values and queueing ----------
// A warp per candidate: one thread's short-word count of 1,450 residues took
// 58 us of a 32-pair call's 150.
template <int P>
__global__ void __launch_bounds__(256) k_score_classify(DevDB db, RunBufs rb, RunParams prm, int n) {
  RunState *st = rb.st;
  constexpr int A = P == 2 ? 4 : 28;
  __shared__ uint32_t s_rc[28];
  if (threadIdx.x < A) s_rc[threadIdx.x] = rb.rep_rec[2 + threadIdx.x];
  __syncthreads();
  const int L1 = st->rep_len, nb1 = st->rep_nb, net1 = st->rep_net;
  const int warps = gridDim.x * (blockDim.x >> 5);
  for (int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < n; k += warps) {
    const int c = rb.score_cands[k];
    const int L2 = db.len[c], net2 = db.net[c];
    const int ws = net1 < 16 || net2 < 16
                       ? -1
                       : word_count_warp_bits<P>(db.words + db.off[c] + db.hw, net2, prm.w, rb.rep_list);
    if ((threadIdx.x & 31) == 0) {
      const int B = band_blocks(L1, L2, prm.s);
      const int cls = class_of(db.type, window_of(B, nb1), L2);
      rb.score_out[4 * k + 0] = base_sum<A>(db.cnt, c, s_rc);
      rb.score_out[4 * k + 1] = ws;
      rb.score_out[4 * k + 3] = B;
      rb.queue[cls][atomicAdd(&st->qcount[cls], 1u)] = k;
    }
  }
}

cudaError_t launch_score_classify(ngia_ctx *c, int n) {
  const int grid = std::max(1, std::min(c->num_sms * 8, (n + 7) / 8));
  if (c->db.P == 2)
    k_score_classify<2><<<grid, 256, 0, c->stream>>>(c->db, c->rb, c->prm, n);
  else
    k_score_classify<5><<<grid, 256, 0, c->stream>>>(c->db, c->rb, c->prm, n);
  return cudaGetLastError();
}

}  // namespace ngia

namespace ngia {
// ---- the floor under the composition filter's time ---------------------------
// Two kernels with the composition filter's grid and tiles: one that does
// nothing, and one that only reads what the filter reads (each warp's bitmap
// words, then the length and counts of every unclustered sequence of them),
// folding the values so the loads are kept.  Their times on the context's
// stream bound the filter's: launch and one round of dependent loads.
namespace {

__global__ void k_floor_empty(const RunBufs rb) {
  if (threadIdx.x == 0 && blockIdx.x == 0 && rb.st == nullptr) rb.fstats[0] = 1;
}

__global__ void __launch_bounds__(256) k_floor_read(DevDB db, RunBufs rb, unsigned long long *sink) {
  constexpr int kW = kFilterWords, kTileWords = 8 * kW;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nbw = (db.n + 31) / 32;
  const int tiles = (nbw + kTileWords - 1) / kTileWords;
  uint32_t acc = 0;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    uint32_t bits_of[kW];
#pragma unroll
    for (int k = 0; k < kW; k++) {
      const int wi = tile * kTileWords + warp * kW + k;
      bits_of[k] = wi < nbw ? rb.alive[wi] : 0u;
    }
#pragma unroll
    for (int k = 0; k < kW; k++) {
      const int c = (tile * kTileWords + warp * kW + k) * 32 + lane;
      if ((bits_of[k] >> lane) & 1u) {
        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(db.cnt) + c);
        acc += (uint32_t)__ldg(db.len + c) + q.x + q.y + q.z + q.w;
      }
    }
  }
  // A thread sums at most 8 x 5 values below 2^16 (< 2^22), so this never
  // holds; the compiler cannot know that and keeps the loads.
  if (acc == 0xFFFFFFFFu) atomicAdd(sink, 1ull);
}

}  // namespace
}  // namespace ngia

extern "C" int ngia_measure_filter_floor(ngia_ctx *c, double *launch_us, double *read_us) {
  ngia::clear_error();
  if (!c || !launch_us || !read_us) return ngia::fail(NGIA_E_ARG, "ngia_measure_filter_floor: null argument");
  if (!c->begun) return ngia::fail(NGIA_E_STATE, "ngia_measure_filter_floor before ngia_cluster_begin");
  if (c->db.type != 0) return ngia::fail(NGIA_E_ARG, "ngia_measure_filter_floor: DNA databases only");
  const int nbw = (c->db.n + 31) / 32;
  constexpr int kB = ngia::kFilterWords;
  const int grid = std::max(1, std::min(c->grid_filter, (nbw + 8 * kB - 1) / (8 * kB)));
  constexpr int kReps = 20;
  cudaEvent_t e0 = nullptr, e1 = nullptr, e2 = nullptr;
  cudaError_t e = cudaEventCreate(&e0);
  if (e == cudaSuccess) e = cudaEventCreate(&e1);
  if (e == cudaSuccess) e = cudaEventCreate(&e2);
  // the sink (written only in the impossible case above): the last counter
  // of the filter-statistics stripes
  unsigned long long *sink = c->rb.fstats + ngia::kFilterStripes * ngia::kFilterStats - 1;
  if (e == cudaSuccess) {
    ngia::k_floor_empty<<<grid, 256, 0, c->stream>>>(c->rb);  // warm-up
    ngia::k_floor_read<<<grid, 256, 0, c->stream>>>(c->db, c->rb, sink);
    cudaEventRecord(e0, c->stream);
    for (int r = 0; r < kReps; r++) ngia::k_floor_empty<<<grid, 256, 0, c->stream>>>(c->rb);
    cudaEventRecord(e1, c->stream);
    for (int r = 0; r < kReps; r++) ngia::k_floor_read<<<grid, 256, 0, c->stream>>>(c->db, c->rb, sink);
    cudaEventRecord(e2, c->stream);
    e = cudaEventSynchronize(e2);
  }
  float a = 0.f, b = 0.f;
  if (e == cudaSuccess) e = cudaEventElapsedTime(&a, e0, e1);
  if (e == cudaSuccess) e = cudaEventElapsedTime(&b, e1, e2);
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  if (e2) cudaEventDestroy(e2);
  if (e != cudaSuccess) return ngia::fail(NGIA_E_CUDA, "ngia_measure_filter_floor: %s", cudaGetErrorString(e));
  *launch_us = 1e3 * a / kReps;
  *read_us = 1e3 * b / kReps;
  return NGIA_OK;
}
