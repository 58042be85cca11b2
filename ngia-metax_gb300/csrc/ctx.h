// ctx.h — the library context behind the opaque ngia_ctx handle and the
// host-side launchers each kernel translation unit provides.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "../../include/ngia.h"
#include "common.cuh"

// Several device arrays in one allocation, each on a 256-byte boundary: a
// cudaMalloc and its cudaFree take 2 us of host time on GB300 where the driver
// has room in a chunk of its own, else 60 to 110, and a context has some 30
// arrays.  Opening, clustering and closing a database of 500 short records,
// ms: 1.82; in three allocations 1.65; with the rounds' queues sized by the
// database 1.52; without pinned memory 1.25.
// (No container that can throw: the arrays are added inside C entry points.
// Sizes saturate, so that a record count nobody can have makes the allocation
// fail instead of wrapping the sum to a small one.)
struct DevBlock {
  template <class T>
  void add(T **p, size_t count) {
    constexpr size_t most = (size_t)1 << 48;
    if (count == 0) count = 1;
    if (used < kItems) items[used] = {(void **)p, count > most / sizeof(T) ? most : (sizeof(T) * count + 255) & ~(size_t)255};
    used++;
  }
  size_t bytes() const {
    size_t total = 0;
    for (int i = 0; i < used && i < kItems; i++) total += items[i].bytes;
    return total;
  }
  cudaError_t take() {
    cudaError_t e = used <= kItems ? cudaMalloc(&base, bytes()) : cudaErrorInvalidValue;
    char *at = (char *)base;
    for (int i = 0; i < used && i < kItems; i++) {
      *items[i].p = e == cudaSuccess ? at : nullptr;
      at += items[i].bytes;
    }
    used = 0;
    if (e != cudaSuccess) cudaGetLastError();  // the caller reports it: not the next launch's
    return e;
  }
  void give() {
    cudaFree(base);
    base = nullptr;
  }
  struct Item {
    void **p;
    size_t bytes;
  };
  static constexpr int kItems = 24;
  Item items[kItems];
  int used = 0;
  void *base = nullptr;
};

struct ngia_spec;  // speculative-round driver state (spec.cu)
static_assert(ngia::kNumClasses == 7, "per-class initialisers of ngia_ctx");

struct ngia_ctx {
  int device = 0;
  int num_sms = 0;
  cudaStream_t stream = nullptr;
  ngia::DevDB db{};
  // device arrays of the database (mem_db) and of a run (mem_run)
  DevBlock mem_db, mem_run;
  uint32_t *d_words = nullptr;
  int64_t *d_off = nullptr;
  int32_t *d_len = nullptr, *d_net = nullptr;
  uint32_t *d_cnt = nullptr;
  uint32_t *d_codes = nullptr;  // protein residue-code streams (DevDB::codes)
  int64_t n_words = 0;
  int32_t longest = 0, shortest = 0;
  // capacity of the allocations (a context can be reloaded with any database
  // within it: serving slots)
  int64_t cap_n = 0, cap_words = 0;
  int32_t cap_nb = 0;
  int32_t *d_flags = nullptr;  // loader results: max blocks, short record, bad record, n - db.long_n
  int32_t *h_flags = nullptr;  // host mirror (behind h_state)
  // run buffers
  ngia::RunBufs rb{};
  // Host mirror.  Pinned for contexts that share the GPU with others (a copy
  // into it does not hold up the thread that drives them); pageable for a
  // context of its own, which waits for each copy anyway: allocating and
  // freeing a process's only pinned page takes 270 us on GB300, a copy into
  // pageable memory a few more than into pinned.
  ngia::RunState *h_state = nullptr;
  unsigned char *h_ctl = nullptr;  // kMirrorCtl bytes of it: the speculative driver's (behind h_flags)
  // pair scores: the calls' candidates and results, grown to the largest call
  DevBlock mem_score;
  int32_t score_cap = 0, *d_score_cands = nullptr, *d_score_out = nullptr;
  ngia::RunParams prm{};
  int mode = 0;
  bool begun = false;
  // launch shapes
  int grid_filter = 0;
  int grid_align[ngia::kNumClasses] = {0};
  int grid_wave[ngia::kNumClasses] = {0};  // CTAs of the group-per-pair kernels
  int warp_pairs = -1;  // a class with at most this many pairs runs a group per pair
  int warp_pairs_default = -1;  // the above as sized for this context's grids
  // settings that change speed only (set by ngia_autotune / ngia_set_tuning):
  // test order (0 auto, 1 short words first, 2 alignment first), lockstep
  // refill threshold, group-per-pair cut-off (-1: keep warp_pairs_default)
  int tuned_word_order = 0, tuned_refill = 32, tuned_warp_pairs = -1;
  // per length bucket (alignment class): group-per-pair cut-off (-1: the
  // context's) and CTA divisor; the composition filter's words per warp
  int cls_warp_pairs[ngia::kNumClasses] = {-1, -1, -1, -1, -1, -1, -1};
  int cls_grid_div[ngia::kNumClasses] = {1, 1, 1, 1, 1, 1, 1};
  int filter_tile = 8;
  int tune_gen = 0;             // bumped by every change of the settings above
  int graph_tune_gen = -1;      // tune_gen the captured graph was built with
  int graph_warp_pairs = -1;    // warp_pairs the captured graph was built with
  // graph form of the greedy loop
  cudaGraphExec_t graph_exec = nullptr;
  cudaGraph_t graph = nullptr;
  bool graph_ready = false;
  ngia::RunParams graph_prm{};
  cudaStream_t side[ngia::kNumClasses] = {nullptr};  // created with the first graph, as are join_ev
  cudaEvent_t fork_ev = nullptr, join_ev[ngia::kNumClasses] = {nullptr};
  // timing: whole steps, and (profiling, plain form) filter / align stages
  cudaEvent_t ev_step0 = nullptr, ev_step1 = nullptr, ev_p0 = nullptr, ev_p1 = nullptr, ev_p2 = nullptr;
  cudaEvent_t ev_cls[ngia::kNumClasses + 1] = {nullptr};
  bool profiling = false;
  bool batch_member = false;  // grids sized to the job; serial class launches
  double ms_filter = 0.0, ms_align = 0.0, ms_class[ngia::kNumClasses] = {0.0};
  float last_step_ms = 0.f;
  ngia_spec *spec = nullptr;  // NGIA_MODE_SPEC buffers, allocated on first use
};

constexpr size_t kMirrorCtl = 1024;

namespace ngia {
// api.cu: driver internals shared with batch.cu / serve.cu
namespace drv {
int open_ctx(const ngia_db_view *v, bool batch_member, ngia_ctx **out);
// A context with room for cap_n records, cap_words record words and records
// of up to cap_nb plane blocks, holding no database until reload_ctx.
int open_ctx_capacity(int type, int64_t cap_n, int64_t cap_words, int cap_nb, ngia_ctx **out);
// Its device bytes.
int ctx_bytes(int type, int64_t cap_n, int64_t cap_words, int cap_nb, int num_sms, int64_t *bytes);
// Loads a database within the capacity (stream-ordered copies on the
// context's stream; waits for that stream only).
int reload_ctx(ngia_ctx *c, const ngia_db_view *v);
// begin a run whose unclustered set is the given device bitmap (bit i =
// sequence i takes part), instead of every sequence.
int begin_subset(ngia_ctx *c, const ngia_params *p, int32_t mode, const uint32_t *d_alive);
// graph form of the greedy loop (captured once per parameter set)
int build_graph(ngia_ctx *c);
int ensure_graph(ngia_ctx *c);  // build_graph unless the captured one is current
void destroy_graph(ngia_ctx *c);
int pull_state(ngia_ctx *c);
int check_device_error(ngia_ctx *c);  // of the mirrored run state
int enqueue_iteration(ngia_ctx *c, bool graph, cudaGraphConditionalHandle cond);
void fill_stats(const ngia_ctx *c, ngia_stats *stats);
int validate_params(int type, const ngia_params *p);
int word_can_pay(int type, int shortest, const ngia::RunParams &prm);
// spec.cu: speculative rounds (NGIA_MODE_SPEC)
int spec_prepare(ngia_ctx *c);                 // buffers for the context's capacity; zeroed masks
int spec_step(ngia_ctx *c, int64_t max_iters);  // up to max_iters representatives (<= 0: all)
void spec_free(ngia_ctx *c);
// Device bytes of the driver of a context of this capacity, and those of its
// widest class's rows among them.
int spec_bytes(int type, int64_t n, int nb, int num_sms, int64_t *bytes, int64_t *rows);
bool spec_exact(const ngia_ctx *c);            // rounds reproduce the greedy loop exactly
void spec_stats(const ngia_ctx *c, int64_t *pairs, int64_t *cells);
}  // namespace drv
// loader.cu / filter.cu
cudaError_t launch_loader(ngia_ctx *c, int32_t *d_maxnb, int32_t *d_short, int32_t *d_bad, int32_t *d_end);
cudaError_t launch_init_run(ngia_ctx *c);
cudaError_t launch_prep(ngia_ctx *c, int score_rep);
cudaError_t launch_filter(ngia_ctx *c);
cudaError_t launch_next(ngia_ctx *c, unsigned long long cond_handle, int use_cond);
cudaError_t launch_subset_start(ngia_ctx *c, const uint32_t *d_alive);
cudaError_t launch_score_classify(ngia_ctx *c, int n);
// align.cu
cudaError_t launch_align(ngia_ctx *c, int cls, cudaStream_t s, int score_mode);
int align_occupancy(int type, int cls, int max_nb, bool wave);
int align_threads();
int wave_pairs_per_cta(int type, int cls);
bool wave_fits(int type, int max_nb);  // group-per-pair kernels hold records of this many blocks
cudaError_t align_configure(int type, int max_nb);
cudaError_t filter_configure();
// pool.cu: the pooled batch form (NGIA_MODE_POOL), one pool per record type
namespace pool {
struct Group;
int group_open(const std::vector<ngia_ctx *> &jobs, Group **out);  // jobs of one type
int group_fill(Group *g, cudaStream_t s);  // the jobs' current run buffers and parameters
int group_enqueue_round(Group *g, cudaStream_t s, cudaGraphConditionalHandle cond);
int group_size(const Group *g);
void group_close(Group *g);
}  // namespace pool
}  // namespace ngia
