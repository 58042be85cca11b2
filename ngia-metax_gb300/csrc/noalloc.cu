// noalloc.cu — banded-LCS scores of one representative against a batch of
// queries, for callers that cannot allocate device memory.
//
// Who needs this: host applications whose CUDA memory is owned by someone
// else — a framework or pool allocator that has reserved the device memory and
// hands out sub-buffers, or a latency-bound service loop that must not call
// cudaMalloc/cudaFree (they can synchronise the device and take milliseconds).
// Such a caller already holds its inputs and outputs in device memory; this
// entry point uses them as given and allocates nothing.
//
// Three forms:
//  * up to noalloc_groups pairs per SM, a group of threads per pair (wave.cuh:
//    rows in registers, match table and query codes in shared memory), 8 of
//    them for more than a few pairs;
//  * above that, representatives of up to 112 blocks: a thread per pair, the
//    band rows in a shared-memory ring, register tiles (tile.cuh);
//  * proteins whose match table does not fit shared memory: a thread per
//    pair with its working row (one 32-bit word per 32 representative
//    residues) in a fixed file-scope device array, g_noalloc_rows, of
//    kNoAllocWords words (4 MiB).
// GB300, whole calls: 4,096 DNA queries of 1,450 residues 747 -> 117 us, 1,000
// proteins of 380 residues 278 -> 43 us (against the third form for all).
//
// Every GPU that loads this library keeps that array until the process
// exits.  Its size caps the representative at 65,536 residues (2,048 words
// per thread row); the grid of the third form is sized so that every
// thread's row fits.
//
// Host code must not use the array's name as a device address: the first call
// on each device looks its address up with cudaGetSymbolAddress (with that
// device current) and caches it; make that first call before any stream
// capture.  The cached address belongs to the module loaded in the device's
// primary context: after a cudaDeviceReset it would be stale, so the entry
// point is not for use across a device reset.  Each call copies the
// representative's two header words to the host to size its grid, which
// waits for `stream` to reach that copy.  All calls share the array, so calls
// whose kernels overlap on the GPU (different streams, or concurrent host
// threads) race on it; serialise them.  Nothing in the array has to start at
// zero: each thread initialises its row for every pair it scores.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "../host/host_common.h"
#include "common.cuh"
#include "tile.cuh"
#include "wave.cuh"

namespace {

constexpr int kNoAllocWords = 1 << 20;  // 4 MiB of per-thread rows
constexpr int kThreads = 128;
static_assert(kThreads == ngia::kAlignThreads, "the ring and the groups of four warps");
// Pairs per SM up to which a group per pair is faster than a thread per pair,
// which takes a pair's latency whatever their number.  That latency grows
// faster with the representative than a group's share of an SM, where a step's
// fixed costs count (DNA of 4 to 46 blocks: 34 to 256 us for a thread, 41 to
// 224 for groups of 8 with 80 pairs per SM), so the line rises with its blocks.
// GB300, us for 8 threads per pair and for a thread, at the pairs per SM on
// both sides of the line:
//   DNA, 7 blocks        42, 42 (20)   42, 41 (26)
//       13               55, 61 (32)   65, 61 (40)
//       19               80, 88 (40)   93, 87 (50)
//       25               99, 117 (40)  116, 116 (56)
//       32               140, 153 (64) 167, 153 (72)
//       46               224, 256 (80) 256, 255 (90)
//      107               893, 1,070 (64) 1,084, 1,069 (80)
//   protein, 7 blocks    45, 48 (14)   49, 47 (26)   (seven operations per match
//       12               73, 77 (40)   83, 78 (50)    word of a thread instead of
//       19               133, 142 (72) 158, 142 (90)  three: later)
//       29               235, 262 (105)
constexpr int noalloc_groups(int P, int nb1) {
  return P == 2 ? std::min(std::min(12 + 2 * nb1, 26 + 5 * nb1 / 4), 80) : std::max(12, std::min(4 * nb1, 112));
}
constexpr size_t kNoAllocSmemMost = 226 * 1024;

__device__ __align__(256) uint32_t g_noalloc_rows[kNoAllocWords];

uint32_t *g_rows_addr[64] = {nullptr};  // per-device address of g_noalloc_rows
std::mutex g_rows_mu;

// Generic (any band width) banded bit-parallel LCS of the representative
// staged in shared memory against one query record, in the reference's
// (query block i, rep block j, residue k) loop order (func.cu:473-514); the
// 32 column carries of a block are packed into one word.  line[j * stride]
// is this thread's working row j.
template <int P>
__device__ int banded_lcs(const uint32_t *s_pl, int nb1, int net1, int L1, const uint32_t *q, int hw, float s,
                          uint32_t *line, int64_t stride) {
  const int L2 = (int)q[0], net2 = (int)q[1];
  const int nq = (net2 + 31) >> 5;
  const int B = ngia::band_blocks(L1, L2, s);
  const uint32_t *qpl = q + hw;
  const uint32_t vlast = (net1 & 31) ? ((1u << (net1 & 31)) - 1u) : 0xFFFFFFFFu;
  for (int j = 0; j < nb1; j++) line[j * stride] = 0xFFFFFFFFu;
  for (int i = 0; i < nq; i++) {
    const int cols = ((i + 1) * 32 > net2) ? (net2 & 31) : 32;
    uint32_t col[P];
#pragma unroll
    for (int p = 0; p < P; p++) col[p] = qpl[i * P + p];
    const int jstart = max(i - B, 0), jend = min(i + B, nb1 - 1);
    uint32_t cw = 0;
    for (int j = jstart; j <= jend; j++) {
      uint32_t R[P];
#pragma unroll
      for (int p = 0; p < P; p++) R[p] = s_pl[j * P + p];
      uint32_t row = line[j * stride], ncw = 0;
      for (int k = 0; k < cols; k++) {
        uint32_t x = row;
#pragma unroll
        for (int p = 0; p < P; p++) x &= ~(R[p] ^ (0u - ((col[p] >> k) & 1u)));
        const unsigned long long t = (unsigned long long)row + x + ((cw >> k) & 1u);
        ncw |= (uint32_t)(t >> 32) << k;
        row = (uint32_t)t | (row ^ x);
      }
      line[j * stride] = row;
      cw = ncw;
    }
  }
  int sum = 0;
  for (int j = 0; j < nb1; j++) sum += __popc(~line[j * stride] & (j == nb1 - 1 ? vlast : 0xFFFFFFFFu));
  return sum;
}

template <int P>
__global__ void __launch_bounds__(kThreads) k_noalloc_scores(const uint32_t *__restrict__ words, int64_t rep_off,
                                                             const int64_t *__restrict__ query_off, int n, float s,
                                                             int *__restrict__ scores, uint32_t *rows,
                                                             int64_t lanes, int cap_blocks) {
  extern __shared__ uint32_t s_pl[];
  constexpr int hw = P == 2 ? 6 : 30;
  const uint32_t *rep = words + rep_off;
  const int L1 = (int)rep[0], net1 = (int)rep[1];
  const int nb1 = (net1 + 31) / 32;
  if (nb1 > cap_blocks) return;  // the host checked this; never index past the rows
  for (int t = threadIdx.x; t < nb1 * P; t += blockDim.x) s_pl[t] = rep[hw + t];
  __syncthreads();
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t *line = rows + g;
  for (int64_t k = g; k < n; k += lanes) {
    const uint32_t *q = words + query_off[k];
    const uint32_t L2 = q[0], net2 = q[1];
    if (L2 > (uint32_t)ngia::kMaxLenDev || net2 > L2) {
      scores[k] = -1;  // not a makeDB record
      continue;
    }
    scores[k] = banded_lcs<P>(s_pl, nb1, net1, L1, q, hw, s, line, lanes);
  }
}

// Length and score of a query that needs no alignment: -1 for a record that
// makeDB cannot have written, 0 where the band or a sequence is empty.
// Returns true when there is an alignment to do.
__device__ __forceinline__ bool noalloc_pair(const uint32_t *q, int nb1, int L1, float s, int &net2, int &B, int *score) {
  const uint32_t L2 = q[0];
  net2 = (int)q[1];
  if (L2 > (uint32_t)ngia::kMaxLenDev || (uint32_t)net2 > L2) {
    *score = -1;
    return false;
  }
  B = ngia::band_blocks(L1, (int)L2, s);
  *score = 0;
  return B >= 0 && nb1 > 0 && net2 > 0;
}

// A group of 32 NW threads per pair.  Shared memory: match table | code rings.
// (Query indexes of this and the next two kernels are unsigned: the last stride
// goes past 2^31.  As 64-bit ones a call of 100 queries against 2,600 residues
// took 124 us instead of 117.)
template <int P, int NW, int WMAX>
__global__ void __launch_bounds__(kThreads) k_noalloc_wave(const uint32_t *__restrict__ words, int64_t rep_off,
                                                           const int64_t *__restrict__ query_off, int n, float s,
                                                           int *__restrict__ scores, int cap_blocks) {
  extern __shared__ __align__(16) uint32_t s_mem[];
  __shared__ uint32_t s_xch[4 * NW];
  constexpr int hw = P == 2 ? 6 : 30, kGroups = kThreads / 32 / NW;
  const uint32_t *rep = words + rep_off;
  const int L1 = (int)rep[0], net1 = (int)rep[1], nb1 = (net1 + 31) / 32;
  if (nb1 > cap_blocks) return;  // the host sized shared memory for this many
  const int group = (int)(threadIdx.x >> 5) / NW;
  const bool lead = threadIdx.x % (32 * NW) == 0;
  const uint32_t vlast = (net1 & 31) ? ((1u << (net1 & 31)) - 1u) : 0xFFFFFFFFu;
  uint32_t *ring = s_mem + ngia::wave_table_words(P, nb1) + group * ngia::kWaveRingWords;
  ngia::wave_table<P>(rep + hw, nb1, vlast, s_mem, threadIdx.x, kThreads);
  __syncthreads();
  unsigned long long cells = 0;
  for (uint32_t k = blockIdx.x * kGroups + group; k < (uint32_t)n; k += gridDim.x * kGroups) {
    const uint32_t *q = words + query_off[k];
    int net2 = 0, B = 0, score = 0;
    if (noalloc_pair(q, nb1, L1, s, net2, B, &score))
      score = ngia::wave_any<P, NW, WMAX>(s_mem, nb1, q + hw, (net2 + 31) / 32, net2, B, B, ngia::kNoCut, ring, s_xch,
                                          cells);
    if (lead) scores[k] = score;
  }
}

// Four pairs per warp (wave.cuh).  Shared memory: match table | code rings.
template <int P>
__global__ void __launch_bounds__(kThreads) k_noalloc_sub(const uint32_t *__restrict__ words, int64_t rep_off,
                                                          const int64_t *__restrict__ query_off, int n, float s,
                                                          int *__restrict__ scores, int cap_blocks) {
  extern __shared__ __align__(16) uint32_t s_mem[];
  constexpr int hw = P == 2 ? 6 : 30, kGroups = kThreads / ngia::kSubGroup;
  const uint32_t *rep = words + rep_off;
  const int L1 = (int)rep[0], net1 = (int)rep[1], nb1 = (net1 + 31) / 32;
  if (nb1 > cap_blocks) return;  // the host sized shared memory for this many
  const int group = threadIdx.x / ngia::kSubGroup;
  const uint32_t vlast = (net1 & 31) ? ((1u << (net1 & 31)) - 1u) : 0xFFFFFFFFu;
  uint32_t *ring = s_mem + ngia::wave_table_words(P, nb1) + group * ngia::kSubRingWords;
  ngia::wave_table<P>(rep + hw, nb1, vlast, s_mem, threadIdx.x, kThreads);
  __syncthreads();
  unsigned long long cells = 0;
  const int first = threadIdx.x / 32 * ngia::kSubs;  // the warp's first pair of the CTA's
  for (uint32_t k0 = blockIdx.x * kGroups + first; k0 < (uint32_t)n; k0 += gridDim.x * kGroups) {  // warp-uniform
    const uint32_t k = k0 + (uint32_t)(group - first);
    const uint32_t *q = words;
    int net2 = 0, B = 0, score = 0;
    bool run = false;
    if (k < (uint32_t)n) {
      q = words + query_off[k];
      run = noalloc_pair(q, nb1, L1, s, net2, B, &score);
    }
    const int got = ngia::sub_any<P>(s_mem, nb1, q + hw, run ? (net2 + 31) / 32 : 0, net2, B, B, ngia::kNoCut, ring, cells);
    if (run) score = got;
    if (k < (uint32_t)n && threadIdx.x % ngia::kSubGroup == 0) scores[k] = score;
  }
}

// A thread per pair, 32 neighbouring queries per warp.  Shared memory: rep
// planes | row ring | match table (the layout of the clustering kernel
// without its k-mer bitset).
template <int P, int RING>
__global__ void __launch_bounds__(kThreads, ngia::tiled_min_blocks(P))
    k_noalloc_tiled(const uint32_t *__restrict__ words, int64_t rep_off, const int64_t *__restrict__ query_off, int n,
                    float s, int *__restrict__ scores, int cap_blocks) {
  using Ring = typename ngia::RingOf<RING>::T;
  extern __shared__ __align__(16) uint32_t s_mem[];
  constexpr int hw = P == 2 ? 6 : 30;
  constexpr unsigned kAll = ngia::kFullMask;
  const uint32_t *rep = words + rep_off;
  const int L1 = (int)rep[0], net1 = (int)rep[1], nb1 = (net1 + 31) / 32;
  if (nb1 > cap_blocks) return;
  const uint32_t vlast = (net1 & 31) ? ((1u << (net1 & 31)) - 1u) : 0xFFFFFFFFu;
  const int planes = (cap_blocks * P + 3) & ~3;
  for (int t = threadIdx.x; t < nb1 * P; t += kThreads) s_mem[t] = rep[hw + t];
  __syncthreads();
  uint32_t *s_eq = s_mem + planes + RING * kThreads;
  if constexpr (P == 2) {
    ngia::build_eq(s_mem, nb1, s_eq);
    __syncthreads();
  }
  const uint32_t s_eq_s = ngia::smem_u32(s_eq);
  (void)s_eq_s;
  const uint32_t one_rt = 1u + (uint32_t)(nb1 < 0);
  const ngia::FmaK fk(one_rt);
  (void)fk;
  Ring ring;
  ring.base = s_mem + planes + threadIdx.x;
  const int lane = threadIdx.x & 31;
  for (uint32_t k0 = blockIdx.x * kThreads + threadIdx.x - lane; k0 < (uint32_t)n; k0 += gridDim.x * kThreads) {
    const uint32_t k = k0 + (uint32_t)lane;
    int net2 = 0, B = 0, score = 0, nq = 0, js = 0, je = -1, frozen = 0, zw = 0;
    const uint32_t *qpl = words;
    if (k < (uint32_t)n) {
      const uint32_t *q = words + query_off[k];
      if (noalloc_pair(q, nb1, L1, s, net2, B, &score)) {
        qpl = q + hw;
        nq = (net2 + 31) / 32;
        je = min(B, nb1 - 1);
        ring.reset();
        for (int j = 0; j <= je; j++) ring[j] = 0xFFFFFFFFu;
      }
    }
    for (int i = 0; __any_sync(kAll, i < nq); i++) {  // warp-uniform
      const bool busy = i < nq;
      const int rows = busy ? je - js + 1 : 0;
      const int slots = (int)__reduce_max_sync(kAll, (unsigned)rows);
      if (busy) {
        const int cols = min(32, net2 - 32 * i);
        uint32_t cur[P];
#pragma unroll
        for (int p = 0; p < P; p++) cur[p] = __ldg(qpl + i * P + p);
        zw = ngia::tile_block<P, P == 2>(ring, s_eq_s, s_mem, js, je, nb1, slots, cols, cur, fk);
        const bool last = i + 1 >= nq || ngia::band_advance(ring, i + 1, B, nb1, net1, vlast, net2 - 32 * (i + 1),
                                                            ngia::kNoCut, js, je, frozen, zw) != ngia::kBandGo;
        if (last) {
          score = frozen;
          for (int j = js; j <= je; j++) score += __popc(~ring[j] & (j == nb1 - 1 ? vlast : 0xFFFFFFFFu));
          nq = 0;
        }
      }
    }
    if (k < (uint32_t)n) scores[k] = score;
  }
}

using NoAllocFn = void (*)(const uint32_t *, int64_t, const int64_t *, int, float, int *, int);

// Raises a kernel's dynamic shared memory limit to `bytes` (never lowers it).
cudaError_t noalloc_configure(NoAllocFn fn, int slot, size_t bytes) {
  static std::mutex mu;
  static size_t have[64][16] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(mu);
  if (bytes <= have[dev][slot]) return cudaSuccess;
  e = cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) have[dev][slot] = bytes;
  return e;
}

// Address of g_noalloc_rows on the current device, looked up once per device.
int rows_address(uint32_t **out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return ngia::fail(NGIA_E_CUDA, "ngia_rep_scores_noalloc: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= 64) return ngia::fail(NGIA_E_LIMIT, "ngia_rep_scores_noalloc: device %d >= 64", dev);
  std::lock_guard<std::mutex> lock(g_rows_mu);
  if (!g_rows_addr[dev]) {
    void *p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_rows);
    if (e != cudaSuccess || !p)
      return ngia::fail(NGIA_E_CUDA, "ngia_rep_scores_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
    g_rows_addr[dev] = (uint32_t *)p;
  }
  *out = g_rows_addr[dev];
  return NGIA_OK;
}

}  // namespace

extern "C" int ngia_rep_scores_noalloc(const uint32_t *d_words, int64_t rep_off, const int64_t *d_query_off,
                                       int32_t n, int32_t type, float similarity, int32_t *d_scores,
                                       void *stream) {
  if (!d_words || (n > 0 && (!d_query_off || !d_scores)) || n < 0 || rep_off < 0)
    return ngia::fail(NGIA_E_ARG, "ngia_rep_scores_noalloc: bad argument");
  if (type != 0 && type != 1) return ngia::fail(NGIA_E_ARG, "ngia_rep_scores_noalloc: type %d not 0/1", type);
  if (!(similarity >= 0.1f && similarity <= 1.0f))
    return ngia::fail(NGIA_E_ARG, "ngia_rep_scores_noalloc: similarity outside [0.1, 1.0]");
  uint32_t *rows = nullptr;
  int rc = rows_address(&rows);
  if (rc) return rc;
  if (n == 0) return NGIA_OK;
  cudaStream_t st = (cudaStream_t)stream;
  uint32_t hdr[2] = {0, 0};  // representative raw and net length
  cudaError_t e = cudaMemcpyAsync(hdr, d_words + rep_off, sizeof(hdr), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return ngia::fail(NGIA_E_CUDA, "ngia_rep_scores_noalloc: %s", cudaGetErrorString(e));
  if (hdr[0] > (uint32_t)ngia::kMaxLenDev || hdr[1] > hdr[0])
    return ngia::fail(NGIA_E_LIMIT,
                      "ngia_rep_scores_noalloc: representative of %u residues (net %u); the fixed working "
                      "rows hold at most 65,536",
                      hdr[0], hdr[1]);
  const int nb1 = ((int)hdr[1] + 31) / 32;
  const int P = type == 0 ? 2 : 5;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const bool many = n > noalloc_groups(P, nb1) * std::max(sms, 1) && nb1 <= ngia::kWideWindow;
  const int form = nb1 <= 64 ? 0 : nb1 <= 128 ? 1 : 2;  // a warp, a CTA of one row word per thread, of up to 16
  NoAllocFn fn;
  size_t smem;
  int per;  // pairs per CTA
  const bool sub = !many && n > ngia::sub_from(P, nb1 > 64 ? 0 : 1, 56 * std::max(sms, 1)) && nb1 <= 16 * ngia::kSubGroup;
  if (many) {
    const int ring = nb1 <= ngia::kSmallWindow ? 64 : 128;
    fn = P == 2 ? (ring == 64 ? k_noalloc_tiled<2, 64> : k_noalloc_tiled<2, 128>)
                : (ring == 64 ? k_noalloc_tiled<5, 64> : k_noalloc_tiled<5, 128>);
    smem = 4 * (size_t)(((nb1 * P + 3) & ~3) + ring * kThreads + (P == 2 ? ngia::eq_words(nb1) : 0));
    per = kThreads;
  } else if (sub) {
    fn = P == 2 ? k_noalloc_sub<2> : k_noalloc_sub<5>;
    per = kThreads / ngia::kSubGroup;
    smem = 4 * ((size_t)ngia::wave_table_words(P, nb1) + (size_t)per * ngia::kSubRingWords);
  } else {
    fn = P == 2 ? (form == 0 ? k_noalloc_wave<2, 1, 2> : form == 1 ? k_noalloc_wave<2, 4, 1> : k_noalloc_wave<2, 4, 16>)
                : (form == 0 ? k_noalloc_wave<5, 1, 2> : form == 1 ? k_noalloc_wave<5, 4, 1> : k_noalloc_wave<5, 4, 16>);
    per = form == 0 ? kThreads / 32 : 1;
    smem = 4 * ((size_t)ngia::wave_table_words(P, nb1) + (size_t)per * ngia::kWaveRingWords);
  }
  if (smem <= kNoAllocSmemMost) {
    e = noalloc_configure(fn, (P == 2 ? 0 : 8) + (many ? 4 + (nb1 <= ngia::kSmallWindow ? 0 : 1) : sub ? 6 : form), smem);
    if (e != cudaSuccess) return ngia::fail(NGIA_E_CUDA, "ngia_rep_scores_noalloc: %s", cudaGetErrorString(e));
    const int grid = (int)std::min<int64_t>(std::max(sms, 1) * 8, ((int64_t)n + per - 1) / per);
    fn<<<grid, kThreads, smem, st>>>(d_words, rep_off, d_query_off, n, similarity, d_scores, nb1);
  } else {  // a protein's table of more than 1,700 blocks
    // Every thread owns one row of nb1 words; the grid is as large as the
    // array allows (at least 4 CTAs: 2,048-word rows x 512 threads).
    const int64_t max_lanes = kNoAllocWords / (nb1 > 0 ? nb1 : 1);
    int grid = (int)std::min<int64_t>((int64_t)std::max(sms, 1) * 4, max_lanes / kThreads);
    grid = (int)std::max<int64_t>(1, std::min<int64_t>(grid, ((int64_t)n + kThreads - 1) / kThreads));
    const int64_t lanes = (int64_t)grid * kThreads;
    const int cap_blocks = (int)(kNoAllocWords / lanes);
    k_noalloc_scores<5><<<grid, kThreads, sizeof(uint32_t) * (size_t)(nb1 * P), st>>>(
        d_words, rep_off, d_query_off, n, similarity, d_scores, rows, lanes, cap_blocks);
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return ngia::fail(NGIA_E_CUDA, "ngia_rep_scores_noalloc: %s", cudaGetErrorString(e));
  return NGIA_OK;
}
