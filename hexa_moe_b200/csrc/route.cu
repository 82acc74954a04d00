// Routing: segment the T*top_k routed rows into contiguous, padded per-expert segments.
//
// No host synchronisation, deterministic (equal to a stable sort by expert).  Every row goes to
//   pad_offsets[e] + (rows of e in earlier blocks) + (rows of e in earlier warps) + (rows of e earlier in the warp's chunk).
// Bound: latency (the ids of [131072, 2] are 1 MB).  By size:
//   up to kSmallRows rows, up to 256 experts   one launch: route_place with a single block of 32 warps
//   block count x experts up to kMaxTotals     two launches: route_count writes every block's histogram, then each block of
//                                              route_place adds up the histograms itself (a few 10 KB from L2, by all its
//                                              threads) instead of waiting for one block to scan them serially; the side
//                                              tables are shared out over the blocks
//   beyond that (the re-reading would cost more than a scan) three launches: route_hist, route_scan, route_scatter
// [131072, 2] ids, 64 experts: 10 + 34 + 11 us with the three launches, 3 + 9 us with two; [2048, 2], 8 experts:
// 7 + 5 + 9 us with three, 8 us with one.
// HBM traffic: ids are read twice (8 B per routed row; once by the single block), row_token and token_row written once.
#include <stdarg.h>
#include <stdlib.h>

#include "hexa_common.cuh"

namespace hexa {
namespace {

constexpr int kRowsPerWarp = 512;
constexpr int kMaxExperts = 4096;  // keeps both shared-memory tables under 48 KB

__device__ __forceinline__ int load_id(const int32_t* ids, int64_t f, int64_t T, int64_t stride_t, int64_t stride_k) {
  int64_t j = f / T;
  int64_t t = f - j * T;
  return ids[t * stride_t + j * stride_k];
}

__global__ void route_hist(const int32_t* ids, int64_t T, int64_t n_rows, int64_t stride_t,
                           int64_t stride_k, int E, int32_t* __restrict__ chunk_hist) {
  wait_for_previous();
  extern __shared__ int32_t sm[];
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int32_t* h = sm + warp * E;
  for (int e = lane; e < E; e += 32) h[e] = 0;
  __syncwarp();
  const int64_t chunk = (int64_t)blockIdx.x * warps + warp;
  const int64_t begin = chunk * kRowsPerWarp;
  if (begin < n_rows) {
    const int64_t end = min(begin + (int64_t)kRowsPerWarp, n_rows);
    for (int64_t f = begin + lane; f < end; f += 32) {
      int e = load_id(ids, f, T, stride_t, stride_k);
      if (e >= 0 && e < E) atomicAdd(&h[e], 1);
    }
    __syncwarp();
    for (int e = lane; e < E; e += 32) chunk_hist[chunk * E + e] = h[e];
  }
}

__global__ void __launch_bounds__(1024)
route_scan(int32_t* __restrict__ chunk_hist, int64_t n_chunks, int E, int align, int64_t row_capacity,
           int32_t* __restrict__ counts, int32_t* __restrict__ seg_offsets, int32_t* __restrict__ pad_offsets,
           int32_t* __restrict__ row_token, int32_t* __restrict__ tile_expert, int32_t* __restrict__ pair_off,
           int32_t* __restrict__ pair_block, int64_t pair_cap) {
  wait_for_previous();
  extern __shared__ int32_t sm[];
  int32_t* s_cnt = sm;          // [E]
  int32_t* s_pad = sm + E;      // [E + 1]
  // per-expert exclusive scan over chunks (thread per expert: coalesced across experts)
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int32_t run = 0;
    int64_t c = 0;
    for (; c + 4 <= n_chunks; c += 4) {
      int32_t v0 = chunk_hist[(c + 0) * E + e], v1 = chunk_hist[(c + 1) * E + e];
      int32_t v2 = chunk_hist[(c + 2) * E + e], v3 = chunk_hist[(c + 3) * E + e];
      chunk_hist[(c + 0) * E + e] = run; run += v0;
      chunk_hist[(c + 1) * E + e] = run; run += v1;
      chunk_hist[(c + 2) * E + e] = run; run += v2;
      chunk_hist[(c + 3) * E + e] = run; run += v3;
    }
    for (; c < n_chunks; ++c) {
      int32_t v = chunk_hist[c * E + e];
      chunk_hist[c * E + e] = run; run += v;
    }
    s_cnt[e] = run;
    counts[e] = run;
  }
  __syncthreads();
  // exclusive scans over experts (unpadded and padded) by warp 0, 32 experts per step
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int32_t carry_seg = 0, carry_pad = 0, carry_pair = 0;
    for (int base = 0; base < E; base += 32) {
      int e = base + lane;
      int32_t c = e < E ? s_cnt[e] : 0;
      int32_t p = (c + align - 1) / align * align;
      int32_t q = (p / kRowTile + 1) / 2;      // pair tiles: two 128-row blocks each, the last one may be half empty
      int32_t ic = c, ip = p, iq = q;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int32_t tc = __shfl_up_sync(0xffffffffu, ic, o), tp = __shfl_up_sync(0xffffffffu, ip, o);
        int32_t tq = __shfl_up_sync(0xffffffffu, iq, o);
        if (lane >= o) { ic += tc; ip += tp; iq += tq; }
      }
      if (e < E) {
        seg_offsets[e] = carry_seg + ic - c;
        int32_t po = carry_pad + ip - p;
        pad_offsets[e] = po;
        s_pad[e] = po;
        if (pair_block) pair_off[e] = carry_pair + iq - q;
      }
      carry_seg += __shfl_sync(0xffffffffu, ic, 31);
      carry_pad += __shfl_sync(0xffffffffu, ip, 31);
      carry_pair += __shfl_sync(0xffffffffu, iq, 31);
    }
    if (lane == 0) {
      seg_offsets[E] = carry_seg;
      pad_offsets[E] = carry_pad;
      s_pad[E] = carry_pad;
      if (pair_block) pair_off[E] = carry_pair;
    }
  }
  __syncthreads();
  // pair-tile list for CTA-pair GEMMs: entry = (first 128-row block) * 2 + (the next block belongs to the same expert)
  if (pair_block) {
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
      const int32_t b0 = s_pad[e] / kRowTile, nb = (s_pad[e + 1] - s_pad[e]) / kRowTile;
      int32_t o = pair_off[e];
      for (int32_t i = 0; i < nb; i += 2, ++o)
        if (o < pair_cap) pair_block[o] = (b0 + i) * 2 + (i + 1 < nb ? 1 : 0);
    }
    const int32_t total = pair_off[E];
    for (int64_t i = total + threadIdx.x; i < pair_cap; i += blockDim.x) pair_block[i] = -1;
  }
  // tile -> expert: binary search for the segment that holds the tile's first row
  const int64_t n_tiles = row_capacity / align;
  const int32_t n_pad = s_pad[E];
  for (int64_t i = threadIdx.x; i < n_tiles; i += blockDim.x) {
    int32_t row = (int32_t)(i * align);
    int32_t val = -1;
    if (row < n_pad) {
      int lo = 0, hi = E;  // largest e with s_pad[e] <= row (empty experts share an offset: take the last)
      while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (s_pad[mid] <= row) lo = mid; else hi = mid;
      }
      val = lo;
    }
    tile_expert[i] = val;
  }
  // pad slots of every segment
  for (int64_t i = threadIdx.x; i < (int64_t)E * align; i += blockDim.x) {
    int e = (int)(i / align), o = (int)(i % align);
    int32_t slot = s_pad[e] + s_cnt[e] + o;
    if (slot < s_pad[e + 1]) row_token[slot] = -1;
  }
}

__global__ void route_scatter(const int32_t* ids, int64_t T, int top_k, int64_t n_rows, int64_t stride_t,
                              int64_t stride_k, int E, const int32_t* chunk_base,
                              const int32_t* pad_offsets, int32_t* __restrict__ row_token,
                              int32_t* __restrict__ token_row) {
  wait_for_previous();
  extern __shared__ int32_t sm[];
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int32_t* cur = sm + warp * E;
  const int64_t chunk = (int64_t)blockIdx.x * warps + warp;
  const int64_t begin = chunk * kRowsPerWarp;
  if (begin >= n_rows) return;  // whole warp leaves together
  for (int e = lane; e < E; e += 32) cur[e] = pad_offsets[e] + chunk_base[chunk * E + e];
  __syncwarp();
  const int64_t end = min(begin + (int64_t)kRowsPerWarp, n_rows);
  for (int64_t f0 = begin; f0 < end; f0 += 32) {
    const int64_t f = f0 + lane;
    int e = -1;
    int64_t j = 0, t = 0;
    if (f < end) {
      j = f / T; t = f - j * T;
      e = ids[t * stride_t + j * stride_k];
      if (e < 0 || e >= E) e = -1;
    }
    const unsigned peers = __match_any_sync(0xffffffffu, e);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    int32_t pos = -1;
    if (e >= 0) pos = cur[e] + rank;
    __syncwarp();
    if (e >= 0 && rank == 0) cur[e] += __popc(peers);
    __syncwarp();
    if (f < end) {
      token_row[t * top_k + j] = pos;
      if (pos >= 0) row_token[pos] = (int32_t)t;
    }
  }
}

// ---- one or two launches ------------------------------------------------------------------------------------------------
// A block has 2048 rows when there are several: 16 warps of 128 rows, because a warp places its rows 32 at a time, one
// __match_any_sync after the other ([131072, 2] ids, 64 experts: 3.3 + 8.7 us; 8 warps of 256 rows 5.0 + 12.9).
constexpr int kIters = 4, kLoneIters = 8;          // 32-row groups of a warp
constexpr int kCountWarps = 16;
constexpr int kBlockRows = kCountWarps * 32 * kIters;
constexpr int64_t kSmallRows = 32 * 32 * kLoneIters;       // rows of the single block of 32 warps
constexpr int kSmallExperts = 256, kCountExperts = 512;    // (WARPS + 4) * E + 2 words of shared memory stay under 48 KB
constexpr int64_t kMaxTotals = 65536;

struct Ids {
  const int32_t* p;
  uint32_t T;
  int64_t stride_t, stride_k;
  int E;
  __device__ __forceinline__ int at(uint32_t f, uint32_t& t, uint32_t& j) const {
    j = f / T;
    t = f - j * T;
    const int e = p[(int64_t)t * stride_t + (int64_t)j * stride_k];
    return e >= 0 && e < E ? e : -1;
  }
};

__global__ void __launch_bounds__(kCountWarps * 32)
route_count(Ids ids, uint32_t n_rows, int32_t* __restrict__ totals) {
  wait_for_previous();
  extern __shared__ int32_t sm[];
  for (int e = threadIdx.x; e < ids.E; e += blockDim.x) sm[e] = 0;
  __syncthreads();
  int e[kIters];
  const uint32_t f0 = blockIdx.x * (uint32_t)kBlockRows + threadIdx.x;
#pragma unroll
  for (int i = 0; i < kIters; ++i) {
    const uint32_t f = f0 + (uint32_t)i * blockDim.x;
    uint32_t t, j;
    e[i] = f < n_rows ? ids.at(f, t, j) : -1;
  }
#pragma unroll
  for (int i = 0; i < kIters; ++i)
    if (e[i] >= 0) atomicAdd(&sm[e[i]], 1);
  __syncthreads();
  for (int x = threadIdx.x; x < ids.E; x += blockDim.x) totals[(int64_t)blockIdx.x * ids.E + x] = sm[x];
}

struct Tables {
  int32_t *counts, *seg_offsets, *pad_offsets, *row_token, *token_row, *tile_expert, *pair_block;
  int64_t row_capacity, pair_cap;
  int align;
};

// largest e < E with offs[e] <= x (empty experts share an offset: the last one owns it)
__device__ __forceinline__ int owner(const int32_t* offs, int E, int32_t x) {
  int lo = 0, hi = E;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (offs[mid] <= x) lo = mid; else hi = mid;
  }
  return lo;
}

// totals: one histogram per block, or null when this is the only block
template <int WARPS, int ITERS>
__global__ void __launch_bounds__(WARPS * 32)
route_place(Ids ids, int top_k, uint32_t n_rows, uint32_t rows_per_warp, const int32_t* totals, Tables out) {
  wait_for_previous();
  extern __shared__ int32_t sm[];
  const int E = ids.E;
  int32_t* hist = sm;                    // [WARPS][E]: counts, then the next free row of each expert for each warp
  int32_t* before = hist + WARPS * E;    // [E] rows of earlier blocks
  int32_t* total = before + E;           // [E]
  int32_t* pad = total + E;              // [E + 1]
  int32_t* pair = pad + E + 1;           // [E + 1]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t chunk = (blockIdx.x * (uint32_t)WARPS + (uint32_t)warp) * rows_per_warp;
  const uint32_t chunk_end = min(chunk + rows_per_warp, n_rows);
  int e[ITERS];
  uint32_t t[ITERS], slot[ITERS];      // slot = t * top_k + j
#pragma unroll
  for (int i = 0; i < ITERS; ++i) {
    const uint32_t f = chunk + (uint32_t)i * 32 + (uint32_t)lane;
    e[i] = -1;
    t[i] = slot[i] = 0;
    if (f < chunk_end) {
      uint32_t j;
      e[i] = ids.at(f, t[i], j);
      slot[i] = t[i] * (uint32_t)top_k + j;
    }
  }
  for (int x = threadIdx.x; x < (WARPS + 2) * E; x += WARPS * 32) sm[x] = 0;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ITERS; ++i)
    if (e[i] >= 0) atomicAdd(&hist[warp * E + e[i]], 1);
  if (totals) {      // integer sums: the order of the additions is immaterial
    const int slices = max(1, WARPS * 32 / E);
    for (int x = threadIdx.x; x < slices * E; x += WARPS * 32) {
      const int ex = x % E;
      int b_sum = 0, a_sum = 0;
#pragma unroll 8
      for (int b = x / E; b < (int)gridDim.x; b += slices) {
        const int v = totals[(int64_t)b * E + ex];
        a_sum += v;
        b_sum += b < (int)blockIdx.x ? v : 0;
      }
      atomicAdd(&total[ex], a_sum);
      atomicAdd(&before[ex], b_sum);
    }
  }
  __syncthreads();
  for (int x = threadIdx.x; x < E; x += WARPS * 32) {      // exclusive scan over the block's warps
    int run = before[x];
#pragma unroll 8
    for (int w = 0; w < WARPS; ++w) {
      const int v = hist[w * E + x];
      hist[w * E + x] = run;
      run += v;
    }
    if (!totals) total[x] = run;
  }
  __syncthreads();
  // exclusive scans over experts (unpadded, padded, pair tiles) by warp 0, 32 experts per step
  if (warp == 0) {
    int32_t carry_seg = 0, carry_pad = 0, carry_pair = 0;
    const bool writes = blockIdx.x == 0;
    for (int base = 0; base < E; base += 32) {
      const int x = base + lane;
      const int32_t c = x < E ? total[x] : 0;
      const int32_t p = (c + out.align - 1) / out.align * out.align;
      const int32_t q = (p / kRowTile + 1) / 2;      // two 128-row blocks each, the last one may be half empty
      int32_t ic = c, ip = p, iq = q;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int32_t tc = __shfl_up_sync(0xffffffffu, ic, o), tp = __shfl_up_sync(0xffffffffu, ip, o);
        const int32_t tq = __shfl_up_sync(0xffffffffu, iq, o);
        if (lane >= o) { ic += tc; ip += tp; iq += tq; }
      }
      if (x < E) {
        pad[x] = carry_pad + ip - p;
        pair[x] = carry_pair + iq - q;
        if (writes) {
          out.counts[x] = c;
          out.seg_offsets[x] = carry_seg + ic - c;
          out.pad_offsets[x] = carry_pad + ip - p;
        }
      }
      carry_seg += __shfl_sync(0xffffffffu, ic, 31);
      carry_pad += __shfl_sync(0xffffffffu, ip, 31);
      carry_pair += __shfl_sync(0xffffffffu, iq, 31);
    }
    if (lane == 0) {
      pad[E] = carry_pad;
      pair[E] = carry_pair;
      if (writes) { out.seg_offsets[E] = carry_seg; out.pad_offsets[E] = carry_pad; }
    }
  }
  __syncthreads();
  // this warp's rows, 32 at a time in order
  for (int x = lane; x < E; x += 32) hist[warp * E + x] += pad[x];
  __syncwarp();
  int32_t* cur = hist + warp * E;
#pragma unroll
  for (int i = 0; i < ITERS; ++i) {
    const uint32_t f = chunk + (uint32_t)i * 32;
    if (f >= chunk_end) break;      // uniform across the warp
    const unsigned peers = __match_any_sync(0xffffffffu, e[i]);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    int32_t pos = -1;
    if (e[i] >= 0) pos = cur[e[i]] + rank;
    __syncwarp();
    if (e[i] >= 0 && rank == 0) cur[e[i]] += __popc(peers);
    __syncwarp();
    if (f + (uint32_t)lane < chunk_end) {
      out.token_row[slot[i]] = pos;
      if (pos >= 0) out.row_token[pos] = (int32_t)t[i];
    }
  }
  // side tables, shared out over the grid
  const int64_t tid = (int64_t)blockIdx.x * (WARPS * 32) + threadIdx.x, threads = (int64_t)gridDim.x * (WARPS * 32);
  if (out.pair_block) {      // entry = (first 128-row block) * 2 + (the next block belongs to the same expert)
    for (int64_t i = tid; i < out.pair_cap; i += threads) {
      int32_t v = -1;
      if (i < pair[E]) {
        const int x = owner(pair, E, (int32_t)i);
        const int32_t o = ((int32_t)i - pair[x]) * 2, nb = (pad[x + 1] - pad[x]) / kRowTile;
        v = (pad[x] / kRowTile + o) * 2 + (o + 1 < nb ? 1 : 0);
      }
      out.pair_block[i] = v;
    }
  }
  for (int64_t i = tid; i < out.row_capacity / out.align; i += threads) {
    const int32_t row = (int32_t)(i * out.align);
    out.tile_expert[i] = row < pad[E] ? owner(pad, E, row) : -1;
  }
  const uint32_t align = (uint32_t)out.align, slots = (uint32_t)E * align;      // the host has checked that they fit in 31 bits
  for (uint32_t i = (uint32_t)tid; i < slots; i += (uint32_t)threads) {         // pad slots
    const uint32_t x = i / align, o = i - x * align;
    const int32_t row = pad[x] + total[x] + (int32_t)o;
    if (row < pad[x + 1]) out.row_token[row] = -1;
  }
}

// One expert id per token from the reference's lists: entry i of tok_ids is a token id + 1 (0: pad) and belongs to expert
// exp_ids[i / chunk].  Slot 0 is the pads' and is not part of the result; a negative entry counts from the end, as an index
// does, and an entry outside [-(num_toks + 1), num_toks] is an error: it writes nothing and leaves a code in the status word.
template <typename I>
__global__ void __launch_bounds__(256)
ids_from_lists_kernel(const I* tok_ids, const int32_t* exp_ids, int64_t n, int chunk, int64_t num_toks,
                      int32_t* __restrict__ ids, int32_t* status) {
  wait_for_previous();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int64_t slot = (int64_t)tok_ids[i];
  if (slot > num_toks || slot < -(num_toks + 1)) {
    report_status(status, kStatusBadToken);
    return;
  }
  if (slot < 0) slot += num_toks + 1;
  if (slot > 0) ids[slot - 1] = exp_ids[i / chunk];
}

// 1, 2 or 3 launches, see the head of this file
int route_plan(int64_t n_rows, int E) {
  if (n_rows <= kSmallRows && E <= kSmallExperts) return 1;
  if (n_rows > 0 && E <= kCountExperts && ceil_div(n_rows, kBlockRows) * E <= kMaxTotals) return 2;
  return 3;
}

}  // namespace

// ---- error plumbing shared by every translation unit ------------------------------------------
static thread_local char g_err[512] = "no error";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

// Status words are per device, not per host thread: the kernels of one training step are launched from the
// Python thread (forward) and from the autograd engine's thread (backward), and both must report to the same word.
struct StatusSlot {
  int32_t* word;        // where kernels store their code (device-accessible)
  int host_readable;    // the word lives in pinned host memory: entry points can look at it before they launch
};
static StatusSlot g_status[64];
static uint64_t g_wait_limit_ns = 2000000000ull;
constexpr int kDebugBits = 4 | 8;
static int g_tc_debug = -1;

static int current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  return dev;
}
int32_t* status_word() {
  const int dev = current_device();
  return dev < 0 ? nullptr : __atomic_load_n(&g_status[dev].word, __ATOMIC_ACQUIRE);
}
int status_pending() {
  const int dev = current_device();
  if (dev < 0) return 0;
  int32_t* w = __atomic_load_n(&g_status[dev].word, __ATOMIC_ACQUIRE);
  if (!w || !g_status[dev].host_readable) return 0;
  return (int)*reinterpret_cast<volatile int32_t*>(w);
}
uint64_t wait_limit_ns() { return g_wait_limit_ns; }
int tc_debug_flags() {
  if (g_tc_debug < 0) {
    const char* s = getenv("HEXA_TC_DEBUG");
    g_tc_debug = s ? atoi(s) & kDebugBits : 0;
  }
  return g_tc_debug;
}

static uint64_t g_launches = 0;
void count_launch() { __atomic_fetch_add(&g_launches, 1, __ATOMIC_RELAXED); }

static int g_sm_limit = 0;
int sm_limit() { return g_sm_limit; }

int sm_count() {
  static int cached[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

}  // namespace hexa

using namespace hexa;

extern "C" int hexa_version(void) { return 100; }
extern "C" uint64_t hexa_launch_count(void) { return __atomic_load_n(&hexa::g_launches, __ATOMIC_RELAXED); }
extern "C" int hexa_set_sm_limit(int n) {
  hexa::g_sm_limit = n > 0 ? n : 0;
  return HEXA_OK;
}
extern "C" const char* hexa_last_error_string(void) { return hexa::g_err; }
extern "C" int hexa_set_status_word(int32_t* status) {
  const int dev = hexa::current_device();
  HEXA_REQUIRE(dev >= 0, "hexa_set_status_word: no current CUDA device (or ordinal >= 64)");
  int host = 0;
  if (status) {
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, status) == cudaSuccess) host = at.type == cudaMemoryTypeHost;
    else (void)cudaGetLastError();
  }
  hexa::g_status[dev].host_readable = host;
  __atomic_store_n(&hexa::g_status[dev].word, status, __ATOMIC_RELEASE);
  return HEXA_OK;
}
extern "C" int hexa_pending_device_status(void) { return hexa::status_pending(); }
extern "C" int hexa_set_wait_limit_ns(uint64_t ns) {
  HEXA_REQUIRE(ns >= 1000, "hexa_set_wait_limit_ns: the limit must be at least 1000 ns");
  hexa::g_wait_limit_ns = ns;
  return HEXA_OK;
}
extern "C" int hexa_set_tc_debug(int flags) {
  HEXA_REQUIRE((flags & ~hexa::kDebugBits) == 0, "hexa_set_tc_debug: flags must be a combination of bits 2 and 3");
  hexa::g_tc_debug = flags;
  return HEXA_OK;
}

extern "C" int64_t hexa_route_row_capacity(int64_t T, int top_k, int E, int align) {
  if (T < 0 || top_k <= 0 || E <= 0 || align <= 0) return -1;
  int64_t cap = T * top_k + (int64_t)E * (align - 1);
  return ceil_div(cap, align) * align;
}

extern "C" size_t hexa_route_workspace_bytes(int64_t T, int top_k, int E) {
  if (T < 0 || top_k <= 0 || E <= 0) return 0;
  int64_t chunks = ceil_div(T * top_k, kRowsPerWarp);
  if (chunks < 1) chunks = 1;
  return ((size_t)chunks * (size_t)E + (size_t)E + 1) * sizeof(int32_t);   // per-chunk histograms + pair-tile offsets
}

extern "C" int64_t hexa_route_pair_capacity(int64_t T, int top_k, int E) {
  const int64_t cap = hexa_route_row_capacity(T, top_k, E, kRowTile);
  if (cap < 0) return -1;
  return cap / (2 * kRowTile) + E + 1;   // every expert may end on a half-filled pair; one terminator
}

extern "C" int hexa_route(const int32_t* ids, int64_t T, int top_k, int64_t stride_t, int64_t stride_k, int E,
                          int align, int32_t* counts, int32_t* seg_offsets, int32_t* pad_offsets,
                          int32_t* row_token, int32_t* token_row, int32_t* tile_expert, int32_t* pair_block,
                          void* workspace, size_t workspace_bytes, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  HEXA_REQUIRE(T >= 0 && top_k > 0 && E > 0 && E <= kMaxExperts && align > 0, "hexa_route: bad sizes T=%lld k=%d E=%d align=%d",
               (long long)T, top_k, E, align);
  HEXA_REQUIRE(T * top_k + (int64_t)E * align < (int64_t)INT32_MAX, "hexa_route: too many rows for int32 indices");
  HEXA_REQUIRE(counts && seg_offsets && pad_offsets && row_token && token_row && tile_expert && workspace,
               "hexa_route: null output or workspace pointer");
  HEXA_REQUIRE(T == 0 || ids, "hexa_route: null ids");
  const size_t need = hexa_route_workspace_bytes(T, top_k, E);
  if (workspace_bytes < need) {
    set_error("hexa_route: workspace %zu bytes < required %zu", workspace_bytes, need);
    return HEXA_ERR_WORKSPACE;
  }
  HEXA_REQUIRE(pair_block == nullptr || align == kRowTile, "hexa_route: the pair-tile list needs align = %d", kRowTile);
  const int64_t n_rows = T * top_k;
  const int64_t row_cap = hexa_route_row_capacity(T, top_k, E, align);
  const int64_t pair_cap = pair_block ? hexa_route_pair_capacity(T, top_k, E) : 0;
  const int plan = route_plan(n_rows, E);
  if (plan <= 2) {
    const Ids in{ids, (uint32_t)(T > 0 ? T : 1), stride_t, stride_k, E};
    const Tables out{counts, seg_offsets, pad_offsets, row_token, token_row, tile_expert, pair_block, row_cap, pair_cap, align};
    if (plan == 1) {
      const uint32_t rows_per_warp = (uint32_t)ceil_div(ceil_div(n_rows, 32), 32) * 32;
      after_previous(route_place<32, kLoneIters>, 1, 1024, (36 * (size_t)E + 2) * sizeof(int32_t), stream)(in, top_k, (uint32_t)n_rows, rows_per_warp, nullptr, out);
    } else {
      const unsigned blocks = (unsigned)ceil_div(n_rows, kBlockRows);
      int32_t* totals = (int32_t*)workspace;      // blocks * E words, fewer than the chunk histograms of the third plan
      after_previous(route_count, blocks, kCountWarps * 32, (size_t)E * sizeof(int32_t), stream)(in, (uint32_t)n_rows, totals);
      HEXA_LAUNCH_CHECK("route_count");
      after_previous(route_place<kCountWarps, kIters>, blocks, kCountWarps * 32, ((kCountWarps + 4) * (size_t)E + 2) * sizeof(int32_t), stream)(
          in, top_k, (uint32_t)n_rows, 32 * kIters, totals, out);
    }
    HEXA_LAUNCH_CHECK("route_place");
    return HEXA_OK;
  }
  const int64_t n_chunks = ceil_div(n_rows, kRowsPerWarp);
  int32_t* chunk_hist = (int32_t*)workspace;
  int warps = (int)(48 * 1024 / (4 * (int64_t)E));
  warps = warps < 1 ? 1 : (warps > 8 ? 8 : warps);
  const size_t smem = (size_t)warps * E * sizeof(int32_t);
  if (n_chunks > 0) {
    after_previous(route_hist, (unsigned)ceil_div(n_chunks, warps), warps * 32, smem, stream)(ids, T, n_rows, stride_t, stride_k, E,
                                                                                chunk_hist);
    HEXA_LAUNCH_CHECK("route_hist");
  }
  int32_t* pair_off = chunk_hist + (size_t)(n_chunks > 0 ? n_chunks : 1) * E;
  after_previous(route_scan, 1, 1024, (2 * (size_t)E + 1) * sizeof(int32_t), stream)(
      chunk_hist, n_chunks, E, align, row_cap, counts, seg_offsets, pad_offsets, row_token, tile_expert, pair_off, pair_block,
      pair_cap);
  HEXA_LAUNCH_CHECK("route_scan");
  if (n_chunks > 0) {
    after_previous(route_scatter, (unsigned)ceil_div(n_chunks, warps), warps * 32, smem, stream)(
        ids, T, top_k, n_rows, stride_t, stride_k, E, chunk_hist, pad_offsets, row_token, token_row);
    HEXA_LAUNCH_CHECK("route_scatter");
  }
  return HEXA_OK;
}

extern "C" int hexa_route_launches(int64_t T, int top_k, int E) {
  return T < 0 || top_k <= 0 || E <= 0 ? 0 : route_plan(T * top_k, E);
}

namespace {
template <typename I>
int ids_from_lists(const I* tok_ids, const int32_t* exp_ids, int64_t n, int chunk, int64_t num_toks, int32_t* ids, cudaStream_t stream) {
  HEXA_REQUIRE(n >= 0 && chunk > 0 && num_toks >= 0 && ceil_div(n, 256) < INT32_MAX, "hexa_ids_from_lists: bad sizes");
  HEXA_REQUIRE((num_toks == 0 || ids) && (n == 0 || (tok_ids && exp_ids)), "hexa_ids_from_lists: null pointer");
  if (num_toks > 0) HEXA_CUDA(cudaMemsetAsync(ids, 0xFF, (size_t)num_toks * sizeof(int32_t), stream));      // -1: token in no segment
  if (n == 0) return HEXA_OK;
  after_previous(ids_from_lists_kernel<I>, (unsigned)ceil_div(n, 256), 256, 0, stream)(tok_ids, exp_ids, n, chunk, num_toks, ids, status_word());
  HEXA_LAUNCH_CHECK("ids_from_lists_kernel");
  return HEXA_OK;
}
}  // namespace

extern "C" int hexa_ids_from_lists(const int32_t* tok_ids, const int32_t* exp_ids, int64_t n, int chunk, int64_t num_toks, int32_t* ids,
                                   void* stream_) {
  return ids_from_lists(tok_ids, exp_ids, n, chunk, num_toks, ids, (cudaStream_t)stream_);
}
extern "C" int hexa_ids_from_lists_i64(const int64_t* tok_ids, const int32_t* exp_ids, int64_t n, int chunk, int64_t num_toks,
                                       int32_t* ids, void* stream_) {
  return ids_from_lists(reinterpret_cast<const long long*>(tok_ids), exp_ids, n, chunk, num_toks, ids, (cudaStream_t)stream_);
}
