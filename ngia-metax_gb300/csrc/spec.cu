// spec.cu — speculative rounds of the greedy loop (NGIA_MODE_SPEC).
//
// The greedy loop takes one representative per iteration: the longest
// unclustered sequence, whose members (every unclustered sequence passing
// the composition, short-word and banded-LCS tests against it) leave the set
// (the reference's clustering(), CUDA/signalNode/src/func.cu:607-677).  Once
// the unclustered set is small, an iteration no longer fills the GPU: its
// time is the latency of its slowest pair.  A speculative round takes the
// next K unclustered sequences c_0 < ... < c_{K-1} (sorted order) as
// candidate representatives at once and runs every pair (c_i, x), x an
// unclustered sequence with x >= c_i, through the same three tests; each
// accepted pair sets bit i of x's mask and records its score.  The round then
// replays the greedy order exactly:
//   c_i is a representative  iff  no representative c_j, j < i, accepts it
//     (c_0 always is) — in the greedy loop c_i would have joined that c_j
//     before its own turn, and otherwise it is the longest sequence left
//     when its turn comes, since every c_j, j < i, has been taken or absorbed;
//   x joins the first representative of the round that accepts it, with
//     that pair's score — exactly the representative whose iteration would
//     have absorbed it.
// Sequences accepted by no representative of the round stay unclustered.  The
// per-pair tests are pure functions of the pair, except the reference's
// short-word kernel, whose thread leaves at its first job of net length < 16
// (the job list of one iteration decides which later pairs skip the test):
// with such records, the short-word test on (precise off) and more sequences
// than the reference's 16,384 threads, the driver runs the plain loop
// instead.  K is sized so that a round's pairs stay within
// a budget (a few waves of the alignment kernels); while the unclustered set
// is larger than that budget the plain one-representative iteration runs.
#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>

#include "../host/host_common.h"
#include "assign.cuh"
#include "ctx.h"

using ngia::fail;

namespace ngia {
namespace {

constexpr int kSpecMax = 64;              // candidate representatives per round (one mask bit each)
constexpr int kSpecBudget = 1 << 20;      // pairs per round at most (K x unclustered)
// Rounds start once the unclustered set is this small.  The line is that of an
// earlier round kernel, which took the representative per pair, at half the
// clustering kernels' cell rate; with groups of one representative it lies too
// low.  GB300, ms to the end with rounds from 2^13, 2^14, 2^15 and 2^16
// unclustered sequences on: 60,000 DNA of 600 residues, s = 0.85, 2,350, 1,993,
// 1,380 and 524; 60,000 of 300, s = 0.9, 1,541, 1,307, 896 and 258; 50,000 of
// 1,450 4,984, 4,147, 2,694 and 1,302; 200,000 of 600 from 2^15 to 2^18 10,034,
// 9,039, 7,559 and 6,234 (NGIA_SPEC_MAX_ALIVE).
constexpr int kSpecMaxAlive = 1 << 15;
constexpr int kSpecRecheck = 8;  // graph iterations between looks at the unclustered set
constexpr int64_t kSpecScoreWords = 1ll << 26;  // K x n scores at most (256 MB)

// Pairs of the first round: K starts at this many pairs and doubles while a
// round leaves more than half of the set, so that a representative that takes
// nearly everything (short peptides against a long one) does not cost the
// pairs of all the candidates after it (30,000 proteins, s=0.5: two rounds of 27 ms; with the
// query-row class and the wave kernels 70 -> 14 ms for the job).
constexpr int kSpecFirst = 1 << 16;

struct SpecCtl {
  int32_t k;                // candidates of this round (0: none, or the set is above the budget)
  int32_t alive;            // unclustered sequences at the round's start
  unsigned long long valid;  // bit i: candidate i is a representative
  int32_t left;             // unclustered sequences after the round
  int32_t err;              // 1: an inconsistent mask (never expected)
  int32_t ramp;             // candidates allowed so far (0: first round)
  int32_t reserved;
  uint32_t prev[kCtlWords];  // the previous round's queue counters (RoundBufs ctl)
  unsigned long long stats[2];  // RoundBufs::stats and the run state after the round: the host reads
  RunState st;                  // a round's outcome in one copy
};

struct SpecDev {
  int32_t *list;            // the unclustered sequences in order; the first k are the candidates
  SpecCtl *ctl;
  int64_t *rs_off;          // record offsets of the candidates (the RepStore's off)
  uint32_t *lists;          // k-mer bitsets of the candidates
  uint8_t *first;           // and the order of their tests
};

// Round start (one CTA of 1,024 threads): lists the unclustered set (its
// first list_cap members), sizes K and gathers the candidates' record offsets;
// zeroes the round's queue counters.  Marks the run done when nothing is left.
__global__ void __launch_bounds__(1024) k_spec_pick(DevDB db, RunBufs run, SpecDev sd, RoundBufs rb, int k_max,
                                                    int budget, int max_alive, int list_cap) {
  __shared__ int s_red[32];
  __shared__ int s_k;
  RunState *st = run.st;
  const int nbw = (db.n + 31) / 32;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (tid < kCtlWords) {
    sd.ctl->prev[tid] = rb.ctl[tid];
    rb.ctl[tid] = 0;
  }
  int total = 0;
  for (int base = 0; base < nbw; base += blockDim.x) {
    const int wi = base + tid;
    const uint32_t w = wi < nbw ? run.alive[wi] : 0u;
    const int c = __popc(w);
    int x = c;  // inclusive scan within the warp
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kFullMask, x, o);
      if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) s_red[wid] = x;
    __syncthreads();
    if (wid == 0) {  // inclusive scan of the warp totals
      int v = s_red[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFullMask, v, o);
        if (lane >= o) v += y;
      }
      s_red[lane] = v;
    }
    __syncthreads();
    int r = total + (wid ? s_red[wid - 1] : 0) + x - c;  // rank of this word's first unclustered sequence
    for (uint32_t m = w; m && r < list_cap; m &= m - 1) sd.list[r++] = wi * 32 + __ffs(m) - 1;
    total += s_red[31];
  }
  if (tid == 0) {
    int k = 0;
    const int64_t rem = st->iter_limit - st->iter;
    // at least two candidates per round (one is a plain iteration, which
    // the clustering kernels run faster)
    if (total > 0 && total <= max_alive && (int64_t)total * 2 <= budget && k_max >= 2 && !st->err && rem > 0) {
      int ramp = max(max(sd.ctl->ramp, 2), kSpecFirst / total);
      if (sd.ctl->k > 0 && sd.ctl->ramp > 0 && 2 * total > sd.ctl->alive) ramp = max(ramp, 2 * sd.ctl->ramp);
      ramp = min(ramp, kSpecMax);
      sd.ctl->ramp = ramp;
      k = min(min(k_max, ramp), budget / total);
      k = min(max(k, 2), total);
      if (rem < k) k = (int)rem;
    }
    if (total == 0) st->done = 1;
    sd.ctl->k = k;
    sd.ctl->alive = total;
    sd.ctl->valid = 0;
    sd.ctl->left = 0;
    s_k = k;
  }
  __syncthreads();
  for (int i = tid; i < s_k; i += blockDim.x) sd.rs_off[i] = db.off[sd.list[i]];
  // the plain iteration (and a checkpoint) take the representative from here
  if (tid == 0 && total > 0) st->rep = sd.list[0];
  __syncthreads();
  static_assert(sizeof(RunState) % 4 == 0, "copied by words");
  if (tid < 2) sd.ctl->stats[tid] = rb.stats[tid];
  for (int i = tid; i < (int)(sizeof(RunState) / 4); i += blockDim.x)
    reinterpret_cast<uint32_t *>(&sd.ctl->st)[i] = reinterpret_cast<const uint32_t *>(st)[i];
}

// Filter of a round: candidate blockIdx.y against kSpecTile members of the
// unclustered list from position blockIdx.x * kSpecTile — composition test,
// and the short-word test when it goes first — with the survivors queued by
// class (queue_groups).  The first candidate's CTAs clear the members' masks.
constexpr int kSpecTile = 1024;
template <int P>
__global__ void __launch_bounds__(256) k_spec_filter(DevDB db, SpecDev sd, RoundBufs rb, RunParams prm,
                                                      int list_words) {
  constexpr int A = P == 2 ? 4 : 28;
  extern __shared__ uint32_t s_list[];  // the candidate's k-mer bitset (word-first order)
  __shared__ uint32_t s_rc[A], s_cnt[kServeClasses], s_base[kServeClasses], s_pos[kServeClasses];
  __shared__ uint8_t s_res[kSpecTile];
  const int i = blockIdx.y, alive = sd.ctl->alive, p0 = blockIdx.x * kSpecTile;
  if (i >= sd.ctl->k || p0 >= alive) return;
  const int n = min(kSpecTile, alive - p0);
  const uint32_t *rec = db.words + sd.rs_off[i];
  const int L1 = (int)rec[0], net1 = (int)rec[1], nb1 = (net1 + 31) / 32;
  const bool word_here = !prm.precise && net1 >= 16 && sd.first[i];
  if (threadIdx.x < A) s_rc[threadIdx.x] = rec[2 + threadIdx.x];
  if (threadIdx.x < kServeClasses) s_cnt[threadIdx.x] = 0;
  if (word_here)
    for (int t = threadIdx.x; t < list_words; t += blockDim.x) s_list[t] = sd.lists[(int64_t)i * list_words + t];
  __syncthreads();
  const float s = prm.s;
  const int lane = threadIdx.x & 31;
  for (int k0 = (threadIdx.x >> 5) * 32; k0 < n; k0 += blockDim.x) {
    const int p = p0 + k0 + lane;
    int res = 0;
    if (p < alive) {
      if (i == 0) rb.mask[p] = 0ull;
      if (p >= i) {
        const int x = sd.list[p];
        const int L2 = __ldg(db.len + x), cut = cutoff_of(L2, s);
        bool pass = !(base_sum<A>(db.cnt, x, s_rc) < cut);
        if (pass && word_here) {
          const int net2 = __ldg(db.net + x);
          if (net2 >= 16) pass = words_reach<P, 1>(db, x, net2, prm.w, word_min(L2, prm.w, s), KmerBits{s_list}, s_list);
        }
        if (pass) res = 1 + round_class(window_need(L1, L2, cut, band_blocks(L1, L2, s), nb1), L2);
      }
    }
    s_res[k0 + lane] = (uint8_t)res;
    const unsigned pm = __ballot_sync(kFullMask, res != 0);
    if (res) {
      const unsigned peers = __match_any_sync(pm, res);
      if (lane == __ffs(peers) - 1) atomicAdd(&s_cnt[res - 1], (uint32_t)__popc(peers));
    }
  }
  __syncthreads();
  queue_groups(rb, i, p0, n, s_res, s_cnt, s_base, s_pos);
}

// Applies a round, one thread per member of the list: which candidates are
// representatives (in order: one is iff no earlier representative accepted
// it; every CTA works it out from the candidates' masks), representatives,
// members with their scores, the unclustered set, what is left of it.
__global__ void __launch_bounds__(256) k_spec_assign(RunBufs run, SpecDev sd, RoundBufs rb) {
  __shared__ unsigned long long s_m[kSpecMax], s_v;
  const int k = sd.ctl->k, alive = sd.ctl->alive;
  if (k == 0) return;
  if (threadIdx.x < k) s_m[threadIdx.x] = rb.mask[threadIdx.x];
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long v = 0;
    for (int i = 0; i < k; i++)  // bits of earlier representatives
      if (!(s_m[i] & v)) v |= 1ull << i;
    s_v = v;
    if (blockIdx.x == 0) {
      sd.ctl->valid = v;
      run.st->iter += __popcll(v);
    }
  }
  __syncthreads();
  const unsigned long long v = s_v;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  int left = 0, members = 0, bad = 0;
  if (p < alive) {
    const unsigned long long acc = rb.mask[p];
    const int x = sd.list[p];
    int to = -1, id = -1;
    if (p < k && ((v >> p) & 1ull)) {
      to = x;
      if ((acc >> p) & 1ull) {
        id = rb.score[(int64_t)p * rb.score_stride + p];
        members = 1;
      }
    } else if (acc & v) {
      const int j = __ffsll((long long)(acc & v)) - 1;
      to = sd.list[j];
      id = rb.score[(int64_t)j * rb.score_stride + p];
      members = 1;
    } else if (p < k) {
      bad = 1;  // a candidate that is none has an earlier representative
    }
    if (to >= 0) {
      run.cluster[x] = to;
      run.ident[x] = id;
      atomicAnd(&run.alive[x >> 5], ~(1u << (x & 31)));
    } else {
      left = 1;
    }
  }
  for (int o = 16; o; o >>= 1) {
    left += __shfl_xor_sync(kFullMask, left, o);
    members += __shfl_xor_sync(kFullMask, members, o);
    bad |= __shfl_xor_sync(kFullMask, bad, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (left) atomicAdd(&sd.ctl->left, left);
    if (members) atomicAdd(&run.st->st_members, (unsigned long long)members);
    if (bad) atomicExch(&sd.ctl->err, 1);
  }
}

}  // namespace
}  // namespace ngia

// Per-context state of the speculative driver (allocated on first use).
struct ngia_spec {
  int64_t cap_n = 0;
  int k_max = 0;
  int type = -1;
  ngia::SpecDev d{};
  ngia::RoundBufs rb{};
  ngia::RepStore rs{};
  unsigned char *h_ctl = nullptr;  // the context's: RoundBufs ctl + SpecCtl
  unsigned long long stats[2] = {0, 0};  // pairs and cells of the run's rounds
  DevBlock mem;
  unsigned char *d_ctl = nullptr;
  ngia::RoundPlan plan;
  int budget = ngia::kSpecBudget;  // pairs per round (NGIA_SPEC_BUDGET lowers it)
  int max_alive = ngia::kSpecMaxAlive;  // rounds once this few are unclustered (NGIA_SPEC_MAX_ALIVE)
  bool big = false;           // the unclustered set was above the round budget at the last check
};

namespace ngia {
namespace drv {

namespace {

#define CKP(call)                                                                              \
  do {                                                                                         \
    cudaError_t e_ = (call);                                                                   \
    if (e_ != cudaSuccess) return fail(NGIA_E_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
  } while (0)

constexpr size_t kCtlBytes = kCtlWords * sizeof(uint32_t) + sizeof(SpecCtl);
static_assert(kCtlBytes <= kMirrorCtl, "the mirror in the context");

// The plan and the device arrays (listed in sp->mem, not allocated) for up to
// n sequences of records of up to nb blocks.
int spec_layout(ngia_spec *sp, int type, int64_t n, int nb, int num_sms) {
  sp->cap_n = n;
  sp->type = type;
  sp->k_max = (int)std::max<int64_t>(1, std::min<int64_t>(kSpecMax, kSpecScoreWords / std::max<int64_t>(1, n)));
  const int lw = kListWords;
  const int64_t pairs = std::min<int64_t>(kSpecBudget, n * sp->k_max);
  CKP(round_plan<true>(sp->plan, type, nb, num_sms, pairs));
  // a tile of a candidate pads its last group of each class (64 MB of queues
  // for a small set cost its open and close 0.1 ms)
  const int64_t cap = pairs + 32ll * kSpecMax * ((n + kSpecTile - 1) / kSpecTile);
  DevBlock &m = sp->mem;
  m.add(&sp->d.list, (size_t)n);
  m.add(&sp->d.rs_off, kSpecMax);
  m.add(&sp->d.lists, (size_t)kSpecMax * lw);
  m.add(&sp->d.first, kSpecMax);
  m.add(&sp->d_ctl, kCtlBytes);
  m.add(&sp->rb.mask, (size_t)n);
  m.add(&sp->rb.score, (size_t)sp->k_max * (size_t)n);
  m.add(&sp->rb.stats, 2);
  for (int k = 0; k < kServeClasses; k++)
    if (serve_class_used(k, nb, true)) m.add(&sp->rb.queue[k], (size_t)cap);
  m.add(&sp->plan.scratch, (size_t)sp->plan.scratch_words);
  sp->rb.cap = cap;
  return NGIA_OK;
}

int spec_alloc(ngia_ctx *c) {
  ngia_spec *sp = c->spec;
  const int64_t n = std::max<int64_t>(c->cap_n, c->db.n);
  const int nb = std::max(c->cap_nb, c->db.max_nb);
  if (sp && sp->cap_n >= n && sp->type == c->db.type && sp->plan.rep_nb >= nb) return NGIA_OK;
  spec_free(c);
  sp = new (std::nothrow) ngia_spec();
  if (!sp) return fail(NGIA_E_NOMEM, "spec: out of host memory");
  c->spec = sp;
  int rc = spec_layout(sp, c->db.type, n, nb, c->num_sms);
  if (!rc && sp->mem.take() != cudaSuccess) rc = fail(NGIA_E_NOMEM, "spec: device allocation failed");
  if (rc) {
    spec_free(c);
    return rc;
  }
  sp->h_ctl = c->h_ctl;
  sp->rb.ctl = reinterpret_cast<uint32_t *>(sp->d_ctl);
  sp->d.ctl = reinterpret_cast<SpecCtl *>(sp->d_ctl + kCtlWords * sizeof(uint32_t));
  sp->rb.list = sp->d.list;
  sp->rb.score_stride = n;
  sp->rb.key = nullptr;
  sp->rb.todo = nullptr;
  return NGIA_OK;
}

int spec_pick(ngia_ctx *c) {
  ngia_spec *sp = c->spec;
  k_spec_pick<<<1, 1024, 0, c->stream>>>(c->db, c->rb, sp->d, sp->rb, sp->k_max, sp->budget, sp->max_alive,
                                         (int)std::min<int64_t>(sp->cap_n, sp->max_alive));
  CKP(cudaGetLastError());
  return NGIA_OK;
}

// Launches the round of k candidates and `alive` members that k_spec_pick
// set up: k-mer lists, filter, alignment (mask form), assign; then the next
// round's pick.
int spec_launch_round(ngia_ctx *c, bool lists, int k, int alive) {
  ngia_spec *sp = c->spec;
  cudaStream_t st = c->stream;
  const int P = c->db.type ? 5 : 2;
  const int lw = (int)std::max<uint32_t>(1u, (1u << (c->prm.w * (P == 2 ? 2 : 5))) / 32u);
  const RepStore rs{c->db.words, sp->d.rs_off, nullptr, nullptr, nullptr, sp->d.lists, kSpecMax, lw, sp->d.first};
  if (lists) {
    if (P == 2)
      k_rep_lists<2><<<k, 256, 0, st>>>(rs, c->prm, sp->d.lists);
    else
      k_rep_lists<5><<<k, 256, 0, st>>>(rs, c->prm, sp->d.lists);
    CKP(cudaGetLastError());
  }
  const dim3 fgrid((alive + kSpecTile - 1) / kSpecTile, k);
  const size_t fsm = lists ? 4 * (size_t)lw : 0;
  if (P == 2)
    k_spec_filter<2><<<fgrid, 256, fsm, st>>>(c->db, sp->d, sp->rb, c->prm, lw);
  else
    k_spec_filter<5><<<fgrid, 256, fsm, st>>>(c->db, sp->d, sp->rb, c->prm, lw);
  CKP(cudaGetLastError());
  CKP(round_launch<true>(sp->plan, c->db, rs, c->prm, sp->rb, st));
  k_spec_assign<<<(alive + 255) / 256, 256, 0, st>>>(c->rb, sp->d, sp->rb);
  CKP(cudaGetLastError());
  return spec_pick(c);
}

int spec_read(ngia_ctx *c) {
  ngia_spec *sp = c->spec;
  CKP(cudaMemcpyAsync(sp->h_ctl, sp->d_ctl, kCtlBytes, cudaMemcpyDeviceToHost, c->stream));
  CKP(cudaStreamSynchronize(c->stream));
  const SpecCtl *ctl = reinterpret_cast<const SpecCtl *>(sp->h_ctl + kCtlWords * sizeof(uint32_t));
  *c->h_state = ctl->st;
  sp->stats[0] = ctl->stats[0];
  sp->stats[1] = ctl->stats[1];
  return check_device_error(c);
}

}  // namespace

// With at most kRefGridThreads sequences every thread of the reference's
// short-word kernel holds at most one job, so its early return only leaves
// the short job itself untested — the pairwise rule of the round kernels.
bool spec_exact(const ngia_ctx *c) {
  return !c->db.has_short || c->prm.precise || c->db.n <= kRefGridThreads;
}

int spec_prepare(ngia_ctx *c) {
  int rc = spec_alloc(c);
  if (rc) return rc;
  ngia_spec *sp = c->spec;
  CKP(cudaMemsetAsync(sp->rb.stats, 0, 2 * sizeof(unsigned long long), c->stream));
  sp->stats[0] = sp->stats[1] = 0;
  CKP(cudaMemsetAsync(sp->d_ctl, 0, kCtlBytes, c->stream));
  sp->big = false;
  sp->budget = kSpecBudget;
  if (const char *b = getenv("NGIA_SPEC_BUDGET")) sp->budget = std::max(1, std::min(kSpecBudget, atoi(b)));
  sp->max_alive = kSpecMaxAlive;
  if (const char *m = getenv("NGIA_SPEC_MAX_ALIVE")) sp->max_alive = std::max(2, atoi(m));
  return NGIA_OK;
}

int spec_bytes(int type, int64_t n, int nb, int num_sms, int64_t *bytes, int64_t *rows) {
  ngia_spec sp;
  const int rc = spec_layout(&sp, type, n, nb, num_sms);
  *bytes = (int64_t)sp.mem.bytes();
  *rows = 4 * sp.plan.scratch_words;
  return rc;
}

void spec_free(ngia_ctx *c) {
  ngia_spec *sp = c->spec;
  if (!sp) return;
  sp->mem.give();
  delete sp;
  c->spec = nullptr;
}

// Runs up to max_iters representatives (all, for max_iters <= 0): plain
// iterations while the unclustered set is above the round budget (or when the
// rounds would not be exact), speculative rounds after that.
int spec_step(ngia_ctx *c, int64_t max_iters) {
  ngia_spec *sp = c->spec;
  if (!sp) return fail(NGIA_E_STATE, "spec: driver not prepared");
  const int64_t it0 = c->h_state->iter;
  const int64_t limit = max_iters > 0 ? it0 + max_iters : LLONG_MAX;
  c->h_state->iter_limit = limit;
  CKP(cudaMemcpyAsync(&c->rb.st->iter_limit, &c->h_state->iter_limit, sizeof(int64_t), cudaMemcpyHostToDevice,
                      c->stream));
  const bool exact = spec_exact(c);
  const bool lists = !c->prm.precise;
  bool picked = false;  // a pick for the next round is in flight
  for (int64_t guard = 0; !c->h_state->done && c->h_state->iter < limit; guard++) {
    if (guard > 2 * (int64_t)c->db.n + 8)
      return fail(NGIA_E_STATE, "spec: more steps than sequences");
    if (!exact || sp->big) {
      // one-representative iterations in the captured loop: the rest of the
      // step when rounds would not be exact, else a few before the next look
      // at the unclustered set
      const int64_t room = limit - c->h_state->iter;
      const int64_t n_it = exact ? std::min<int64_t>(room, kSpecRecheck) : room;
      // captured on first use (databases that start below the threshold,
      // such as serving leftovers, never need it)
      int rc0 = ensure_graph(c);
      if (rc0) return rc0;
      c->h_state->iter_limit = c->h_state->iter + n_it;
      CKP(cudaMemcpyAsync(&c->rb.st->iter_limit, &c->h_state->iter_limit, sizeof(int64_t), cudaMemcpyHostToDevice,
                          c->stream));
      CKP(cudaGraphLaunch(c->graph_exec, c->stream));
      int rc = pull_state(c);
      if (rc) return rc;
      c->h_state->iter_limit = limit;  // the rounds' own limit again
      CKP(cudaMemcpyAsync(&c->rb.st->iter_limit, &c->h_state->iter_limit, sizeof(int64_t), cudaMemcpyHostToDevice,
                          c->stream));
      picked = false;
      if (exact) sp->big = false;  // look at the unclustered set again
      continue;
    }
    if (!picked) {
      int rc = spec_pick(c);
      if (!rc) rc = spec_read(c);
      if (rc) return rc;
      picked = true;
    }
    const SpecCtl *ctl = reinterpret_cast<const SpecCtl *>(sp->h_ctl + kCtlWords * sizeof(uint32_t));
    if (ctl->k == 0) {
      picked = false;
      if (ctl->alive == 0 || c->h_state->done) break;
      if (c->h_state->iter >= limit || c->h_state->err) break;
      sp->big = true;  // above the budget: plain iterations for a while
      continue;
    }
    int rc = spec_launch_round(c, lists, ctl->k, ctl->alive);
    if (rc) return rc;
    rc = spec_read(c);  // this round applied, the next one picked
    if (rc) return rc;
    const uint32_t *qc = ctl->prev;  // this round's queue counters
    for (int k = 0; k < kServeClasses; k++)
      if (qc[k] > sp->rb.cap) return fail(NGIA_E_LIMIT, "spec: a round queued more pairs than its budget");
    if (ctl->err) return fail(NGIA_E_DEVICE, "spec: inconsistent acceptance masks");
  }
  return NGIA_OK;
}

void spec_stats(const ngia_ctx *c, int64_t *pairs, int64_t *cells) {
  *pairs = c->spec ? (int64_t)c->spec->stats[0] : 0;
  *cells = c->spec ? (int64_t)c->spec->stats[1] : 0;
}

}  // namespace drv
}  // namespace ngia
