// ESMM and ESTMM on fp32 data with the tensor cores (sm_100a), at no less precision than a chain of fp32 FMAs.
//
// Every operand value is written as hi + mid + lo, three bf16 terms that carry all 24 bits of an fp32 value, in three planes
// (split_planes_kernel).  A product then needs the six largest of the nine term products (the other three are below 2^-24
// of it).  What the tensor core lacks is not operand bits but rounding: its accumulator truncates, a bias of half an ulp per
// instruction, so it is never given a long sum.  Per 64-deep k-block the six products of both operands' planes are
// accumulated in TMEM, smallest first, and the epilogue warps add every k-block's result to fp32 registers with ordinary
// rounded additions.  Relative error (2-norm, against 64 bits) of a 256 x 256 result of normal data, FMA chain / this:
//   k = 96: 1.8e-7 / 0.8e-7    128: 2.0e-7 / 0.8e-7    512: 4.1e-7 / 1.0e-7    2048: 8.1e-7 / 1.3e-7    8192: 1.6e-6 / 2.2e-7
// (positive data, the worst for truncation: 1.4 / 0.8, 1.7 / 0.9, 3.5 / 1.0, 7.0 / 1.2, 14 / 2.0 e-7; with 128-deep blocks the bias
// doubles and reaches the FMA chain's error at k = 128, over the whole k it exceeds it).
// Not every operand has such planes.  A value that is not finite, or that a bf16 cannot hold, has none; one below 2^-109 has a
// third term under bf16's smallest step, 2^-133 (operands of 2^-116: 2.2e-6 where the FMA chain has 2.9e-7, of 2^-124: 5.6e-4);
// products that leave fp32's range come out of six terms of either sign as NaN where a chain gives infinity; and when every
// product lies near the lower end (2^-64 x 2^-64) the chain is closer.  So the split takes the largest magnitude of either
// operand and looks for values without planes, an idle warp of the GEMM makes one verdict of it (planes_hold), and the
// CUDA-core kernel, launched behind, redoes the whole operator where the verdict says so (else it returns at once).
//
// Bound: the tensor pipe, six MMAs where bf16 data needs one.  A CTA pair computes a 256 x 256 tile (each CTA its own 128
// rows of A and half of B, as the 16-bit kernel does); a stage is one k-block of both operands' three planes, 96 KB per
// CTA, two stages: 24 MMAs of 128 cycles each cover a stage's load.  Warp 0 loads, one thread of warp 1 of the leader issues,
// 16 epilogue warps keep the tile's sums in registers (64 per thread), drain one of two TMEM accumulators per k-block and
// store through 64B-swizzled staging tiles.  The activation and its derivative are a pass over the result
// (epilogue_rows_kernel): in the epilogue they would hold up the next tile's k-blocks.
// fp32 layer of 8192 tokens, d=512, hidden 2048, 8 experts, top-2 (a launch, CUDA cores / this): fc1 + GELU 811 / 259 us,
// fc2 790 / 224, GELU' 848 / 312, weight gradient 822 / 235.
#include "gemm_launch.h"
#include "hexa_common.cuh"
#include "tc_ptx.cuh"

namespace hexa {
namespace {

constexpr int BLOCK_M = 128, BLOCK_N = 256, BLOCK_K = 64, UMMA_K = 16;
constexpr int kPlanes = 3;
constexpr int kEpiWarps = 16, kParts = 4, kPartCols = BLOCK_N / kParts, kSlab = 16;
constexpr int kThreads = 32 * (2 + kEpiWarps);
constexpr uint32_t kOperandBytes = kPlanes * 128 * BLOCK_K * 2;      // 128 rows (A) or columns (half of B) of one k-block: 48 KB
constexpr uint32_t kStageBytes = 2 * kOperandBytes;
constexpr int kStages = 2;
constexpr uint32_t kStageTile = 128 * 64;                            // 128 rows x 16 fp32 columns
constexpr uint32_t kTmemCols = 2 * BLOCK_N;
constexpr size_t kSmemBytes = 1024 + (size_t)kStages * kStageBytes + kParts * kStageTile + 256;
static_assert(kSmemBytes <= 232448, "more shared memory than one CTA can have (227 KB)");

enum Mode { NK = 0, KN = 1, TN = 2 };      // ESMM with b [n][k] / b [k][n], ESTMM

struct Params {
  const int32_t *tile_expert, *pad_offsets, *row_token, *pair_block;
  int64_t max_pairs;
  const float* bias;
  int64_t ldbias;
  int64_t n, k, m;
  int E;
  uint32_t nt, per_expert, total_tiles;
  const uint32_t* maxima;   // [2][n_maxima] per block of the split: largest magnitude of a, of b (bits; kNoPlanes: a value without planes)
  int n_maxima;
  int terms;                // the most products one result can have
  int32_t* redo;            // the verdict, for the kernel behind this one
  int debug;      // test aid (hexa_set_tc_debug): bit 2 = the producer neither loads nor arrives, every wait runs into its limit
  int32_t* status;
  uint64_t wait_limit_ns;
  bool next_may_start;                  // no SM limit is set, see wait_for_previous
};

struct Tile {
  int e, row0, col0, m0, num_kb;
  bool valid;      // this CTA has rows to store
};

constexpr uint32_t kNoPlanes = 0xffffffffu;

// May the products be made from planes?  amax, bmax: bits of the operands' largest magnitudes.
__device__ __forceinline__ bool planes_hold(uint32_t amax, uint32_t bmax, int terms) {
  if (amax == kNoPlanes || bmax == kNoPlanes) return false;
  if (amax == 0 || bmax == 0) return true;      // all zero
  const int ea = (int)(amax >> 23) - 126, eb = (int)(bmax >> 23) - 126;      // |a| < 2^ea, |b| < 2^eb
  const int log_terms = 32 - __clz(terms);                                   // terms < 2^log_terms
  return ea + eb + log_terms <= 127      // no partial sum reaches 2^128
         && ea + eb >= -100;             // the largest products carry all their terms
}

template <int MODE>
__device__ __forceinline__ bool get_tile(const Params& p, uint32_t t, int rank, Tile& tile) {
  if (MODE == TN) {
    if (t >= p.total_tiles) return false;
    const uint32_t e = t / p.per_expert, rem = t - e * p.per_expert, mrow = rem / p.nt;
    tile.e = (int)e;
    tile.m0 = ((int)mrow * 2 + rank) * BLOCK_M;
    tile.col0 = (int)(rem - mrow * p.nt) * BLOCK_N;
    tile.row0 = p.pad_offsets[e];
    tile.num_kb = (p.pad_offsets[e + 1] - tile.row0) / BLOCK_K;
    tile.valid = tile.m0 < p.m;
    return true;
  }
  const uint32_t row_tile = t / p.nt;
  if (row_tile >= (uint32_t)p.max_pairs) return false;
  const int pb = p.pair_block[row_tile];
  if (pb < 0) return false;
  tile.e = p.tile_expert[pb >> 1];
  tile.valid = rank == 0 || (pb & 1);
  tile.row0 = ((pb >> 1) + rank) * BLOCK_M;
  tile.col0 = (int)(t - row_tile * p.nt) * BLOCK_N;
  tile.m0 = 0;
  tile.num_kb = (int)((p.k + BLOCK_K - 1) / BLOCK_K);
  return tile.e >= 0;
}

template <int MODE>
__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ CUtensorMap tmC, const Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* store_bufs = smem + (size_t)kStages * kStageBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(store_bufs + kParts * kStageTile);
  uint64_t* full = bars;                       // [kStages] producers -> MMA          (used in the leader CTA)
  uint64_t* empty = bars + kStages;            // [kStages] MMA -> producer           (one per CTA, multicast commit)
  uint64_t* acc_full = bars + 2 * kStages;     // [2] MMA -> epilogue, one k-block's sums  (one per CTA, multicast commit)
  uint64_t* acc_empty = acc_full + 2;          // [2] epilogues -> MMA                (used in the leader CTA)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();     // 0 = leader of the pair
  const uint32_t tile_first = blockIdx.x >> 1, tile_step = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], kEpiWarps * 2); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  wait_for_previous(p.next_may_start);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (every CTA)
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      Tile tile;
      const uint32_t lead_full0 = map_to_cta(&full[0], 0);
      for (uint32_t t = tile_first; ok && get_tile<MODE>(p, t, rank, tile); t += tile_step) {
        const int bcol = tile.col0 + rank * 128;
        for (int kb = 0; kb < tile.num_kb; ++kb) {
          if (!(ok = mbar_wait_fast(&empty[stage], phase ^ 1, abort_flag, p.status, 1, p.wait_limit_ns))) break;
          uint8_t* sA = smem + (size_t)stage * kStageBytes;
          uint8_t* sB = sA + kOperandBytes;
          const uint32_t lead_full = lead_full0 + 8u * (uint32_t)stage;
          if (p.debug & 4) {
            if (++stage == kStages) { stage = 0; phase ^= 1; }
            continue;
          }
          if (rank == 0) mbar_expect_tx(&full[stage], 2 * kStageBytes);      // both CTAs' bytes
          if (MODE == TN) {      // 64 columns of all three planes per load
            const int r = tile.row0 + kb * BLOCK_K;
#pragma unroll
            for (int c = 0; c < 2; ++c) tma_load_3d_pair(sA + c * (kOperandBytes / 2), &tmA, lead_full, tile.m0 + c * 64, r, 0);
#pragma unroll
            for (int c = 0; c < 2; ++c) tma_load_3d_pair(sB + c * (kOperandBytes / 2), &tmB, lead_full, bcol + c * 64, r, 0);
          } else {
            tma_load_3d_pair(sA, &tmA, lead_full, kb * BLOCK_K, tile.row0, 0);
            if (MODE == NK) {
              tma_load_4d_pair(sB, &tmB, lead_full, kb * BLOCK_K, bcol, tile.e, 0);
            } else {
#pragma unroll
              for (int c = 0; c < 2; ++c)
                tma_load_4d_pair(sB + c * (kOperandBytes / 2), &tmB, lead_full, bcol + c * 64, kb * BLOCK_K, tile.e, 0);
            }
          }
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only)
    if (lane == 0 && rank == 0) {
      constexpr bool kAMn = MODE == TN, kBMn = MODE != NK;
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((kAMn ? 1u : 0u) << 15) | ((kBMn ? 1u : 0u) << 16) |
                             ((uint32_t)(BLOCK_N >> 3) << 17) | ((uint32_t)((BLOCK_M * 2) >> 4) << 24);
      // K-major: planes 16 KB apart, 8-row groups 1 KB apart, 32 bytes per K = 16.  MN-major: 64-column chunks (three planes
      // of 8 KB each) 24 KB apart, 8-k groups 1 KB apart, 2 KB per K = 16.
      constexpr uint32_t a_plane = (kAMn ? 8192u : 16384u) >> 4, b_plane = (kBMn ? 8192u : 16384u) >> 4;
      constexpr uint32_t a_step = (kAMn ? 2048u : 32u) >> 4, b_step = (kBMn ? 2048u : 32u) >> 4;
      const uint32_t s0 = smem_u32(smem);
      const uint64_t adesc0 = make_smem_desc(s0, kAMn ? kOperandBytes / 2 : 16, 1024);
      const uint64_t bdesc0 = make_smem_desc(s0 + kOperandBytes, kBMn ? kOperandBytes / 2 : 16, 1024);
      constexpr uint64_t kStageDesc = kStageBytes >> 4;
      int stage = 0;
      uint32_t phase = 0, chunk = 0;
      bool ok = true;
      Tile tile;
      for (uint32_t t = tile_first; ok && get_tile<MODE>(p, t, rank, tile); t += tile_step) {
        for (int kb = 0; kb < tile.num_kb; ++kb, ++chunk) {
          const uint32_t acc = chunk & 1;
          if (!(ok = mbar_wait_fast(&acc_empty[acc], ((chunk >> 1) & 1u) ^ 1, abort_flag, p.status, 2, p.wait_limit_ns))) break;
          if (!(ok = mbar_wait_fast(&full[stage], phase, abort_flag, p.status, 3, p.wait_limit_ns))) break;
          tc_fence_after();
          const uint64_t adesc = adesc0 + (uint64_t)stage * kStageDesc, bdesc = bdesc0 + (uint64_t)stage * kStageDesc;
          const uint32_t d_tmem = tmem_base + acc * BLOCK_N;
          // planes (a, b) of the six products, smallest first: lo hi, hi lo, mid mid, mid hi, hi mid, hi hi
          constexpr int pa[6] = {2, 0, 1, 1, 0, 0}, pb[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
          for (int q = 0; q < 6; ++q)
#pragma unroll
            for (int j = 0; j < BLOCK_K / UMMA_K; ++j)
              umma_f16_pair(d_tmem, adesc + (uint64_t)(pa[q] * a_plane + j * a_step), bdesc + (uint64_t)(pb[q] * b_plane + j * b_step),
                            idesc, q + j == 0 ? 0u : 1u);
          umma_commit_pair(&empty[stage]);
          umma_commit_pair(&acc_full[acc]);
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
    if (blockIdx.x == 1) {      // the second CTA of the first pair issues nothing
      uint32_t amax = 0, bmax = 0;
      for (int i = lane; i < p.n_maxima; i += 32) {
        amax = max(amax, p.maxima[i]);
        bmax = max(bmax, p.maxima[p.n_maxima + i]);
      }
      amax = __reduce_max_sync(0xffffffffu, amax);
      bmax = __reduce_max_sync(0xffffffffu, bmax);
      if (lane == 0) *p.redo = planes_hold(amax, bmax, p.terms) ? 0 : 1;
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue (every CTA, its own 128 rows)
    const int q = warp & 3, part = (warp - 2) >> 2;
    const bool leader = (q == 2) && lane == 0;
    uint8_t* buf = store_bufs + part * kStageTile;
    const int rloc = q * 32 + lane;
    uint32_t chunk = 0;
    Tile tile;
    for (uint32_t t = tile_first; get_tile<MODE>(p, t, rank, tile); t += tile_step) {
      float sum[kPartCols];
#pragma unroll
      for (int i = 0; i < kPartCols; ++i) sum[i] = 0.f;
      bool good = true;
      for (int kb = 0; kb < tile.num_kb; ++kb, ++chunk) {
        const uint32_t acc = chunk & 1;
        // one verdict per warp: what follows is for all 32 lanes or none
        good = __all_sync(0xffffffffu, mbar_wait(&acc_full[acc], (chunk >> 1) & 1u, abort_flag, p.status, 4, p.wait_limit_ns));
        if (!good) break;
        tc_fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + acc * BLOCK_N + (uint32_t)(part * kPartCols);
#pragma unroll
        for (int s = 0; s < kPartCols / kSlab; ++s) {
          uint32_t v[16];
          tmem_ld16(taddr + s * kSlab, v);
#pragma unroll
          for (int i = 0; i < 16; ++i) sum[s * kSlab + i] += __uint_as_float(v[i]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (rank != 0) mbar_arrive_cluster(map_to_cta(&acc_empty[acc], 0));
          else mbar_arrive(&acc_empty[acc]);
        }
      }
      // the four warps of a group leave together
      if (!group_all(1 + part, good)) break;
      if (!tile.valid) continue;      // uniform across the CTA
      const int64_t row = (int64_t)(MODE == TN ? tile.m0 : tile.row0) + rloc;
      const bool live = MODE != TN && p.bias != nullptr && (p.row_token == nullptr || p.row_token[row] >= 0);
#pragma unroll
      for (int s = 0; s < kPartCols / kSlab; ++s) {
        const int64_t col = (int64_t)tile.col0 + part * kPartCols + s * kSlab;
        if (col < p.n) {      // uniform across the group
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float v = sum[s * kSlab + i];
            if (live && col + i < p.n) v += p.bias[(int64_t)tile.e * p.ldbias + col + i];
            w[i] = __float_as_uint(v);
          }
          if (leader) bulk_wait_read<0>();   // the previous store has finished reading the buffer
          group_sync(1 + part);
          stage_row(buf, rloc, w);
          fence_async_smem();
          group_sync(1 + part);
          if (leader) {
            if (MODE == TN) tma_store_3d(&tmC, buf, (int)col, tile.m0, tile.e);
            else tma_store_2d(&tmC, buf, (int)col, tile.row0);
            bulk_commit();
          }
        }
      }
    }
    if (leader) bulk_wait_all();
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // no CTA leaves while its peer may still signal its barriers or read its shared memory
  if (warp == 1) {
    if (*abort_flag) {  // error path: give copies / MMAs in flight a bounded moment to land
      for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

// ---- operands as planes ---------------------------------------------------------------------------------------------------
struct Side {
  const float* src;
  int64_t ld, estride, rows, cols;      // per matrix; `E` of them
  int64_t E;
  const int32_t* limit;                 // device-side row count (rows beyond it hold nothing), or null
  __nv_bfloat16* dst;                   // [kPlanes][E][rows][pitch]
  int64_t pitch, plane;
  int vec;                              // rows are whole 16-byte groups
};

// Magnitude of a value as ordered bits, kNoPlanes where three bf16 terms cannot hold it: not finite, rounded to infinity by
// the first term, or so small that the third falls below bf16's smallest step.
__device__ __forceinline__ uint32_t magnitude(float x) {
  const uint32_t m = __float_as_uint(x) & 0x7fffffffu;
  constexpr uint32_t least = (uint32_t)(127 - 109) << 23, most = 0x7f7f7fffu;      // the largest value that rounds to a finite bf16
  return m - least <= most - least || m == 0 ? m : kNoPlanes;
}

// A warp per row, both operands in one launch; maxima[block], maxima[blocks + block] = the largest magnitude of this block's
// rows of a and of b.
__global__ void __launch_bounds__(256)
split_planes_kernel(const Side a, const Side b, uint32_t* __restrict__ maxima) {
  wait_for_previous();
  __shared__ uint32_t seen[2][8];
  const int lane = threadIdx.x & 31;
  const int64_t rows_a = a.limit ? min((int64_t)*a.limit, a.rows) : a.rows * a.E;
  const int64_t rows_b = b.limit ? min((int64_t)*b.limit, b.rows) : b.rows * b.E;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  uint32_t most[2] = {0, 0};
  for (int64_t w = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < rows_a + rows_b; w += warps) {
    const bool first = w < rows_a;
    const Side& s = first ? a : b;
    const int64_t flat = first ? w : w - rows_a, e = flat / s.rows, r = flat - e * s.rows;
    const float* src = s.src + e * s.estride + r * s.ld;
    __nv_bfloat16* dst = s.dst + flat * s.pitch;
    const int64_t plane = s.plane;
    uint32_t m = 0;
    if (s.vec) {
      for (int64_t c0 = lane * 4; c0 < s.cols; c0 += 4 * 128) {
        float4 v[4];      // requested before the first store, which ordinary loads would stay behind
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (c0 + u * 128 < s.cols) v[u] = *reinterpret_cast<const float4*>(src + c0 + u * 128);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int64_t c = c0 + u * 128;
          if (c >= s.cols) break;
          float x[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
          for (int i = 0; i < 4; ++i) m = max(m, magnitude(x[i]));
#pragma unroll
          for (int q = 0; q < kPlanes; ++q) {
            __nv_bfloat162 h[2] = {__floats2bfloat162_rn(x[0], x[1]), __floats2bfloat162_rn(x[2], x[3])};
            *reinterpret_cast<uint2*>(dst + q * plane + c) = *reinterpret_cast<const uint2*>(h);
            x[0] -= __low2float(h[0]); x[1] -= __high2float(h[0]);
            x[2] -= __low2float(h[1]); x[3] -= __high2float(h[1]);
          }
        }
      }
    } else {
      for (int64_t c = lane; c < s.cols; c += 32) {
        float x = src[c];
        m = max(m, magnitude(x));
#pragma unroll
        for (int q = 0; q < kPlanes; ++q) {
          const __nv_bfloat16 h = __float2bfloat16_rn(x);
          dst[q * plane + c] = h;
          x -= __bfloat162float(h);
        }
      }
    }
    if (first) most[0] = max(most[0], m);
    else most[1] = max(most[1], m);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint32_t m = __reduce_max_sync(0xffffffffu, most[i]);
    if (lane == 0) seen[i][threadIdx.x >> 5] = m;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    uint32_t m = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) m = max(m, seen[threadIdx.x][i]);
    maxima[(int64_t)threadIdx.x * gridDim.x + blockIdx.x] = m;
  }
}

// c = act(x) (x may be c itself) or c = c * act'(x), x [rows, cols], over the rows in use
template <int V>
__global__ void __launch_bounds__(256)
epilogue_rows_kernel(const float* x, int64_t ldx, float* c, int64_t ldc, const int32_t* row_token,
                     const int32_t* pad_offsets, int E, int64_t cols, int epilogue, int act) {
  wait_for_previous();
  const int64_t rows = pad_offsets[E], per_row = cols / V;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < rows * per_row; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / per_row, col = (i - r * per_row) * V;
    const bool live = row_token == nullptr || row_token[r] >= 0;
    float xv[V], cv[V];
    if (V == 4) {
      *reinterpret_cast<float4*>(xv) = *reinterpret_cast<const float4*>(x + r * ldx + col);
      if (epilogue == HEXA_EPI_DACT) *reinterpret_cast<float4*>(cv) = *reinterpret_cast<const float4*>(c + r * ldc + col);
    } else {
      xv[0] = x[r * ldx + col];
      if (epilogue == HEXA_EPI_DACT) cv[0] = c[r * ldc + col];
    }
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const float v = epilogue == HEXA_EPI_DACT ? cv[j] * act_grad(act, xv[j]) : act_apply(act, xv[j]);
      cv[j] = live ? v : 0.f;
    }
    if (V == 4) *reinterpret_cast<float4*>(c + r * ldc + col) = *reinterpret_cast<const float4*>(cv);
    else c[r * ldc + col] = cv[0];
  }
}

// ---- host side --------------------------------------------------------------------------------------------------------------
constexpr int kMaxSplitBlocks = 2048;
constexpr size_t kFlagBytes = (2 * kMaxSplitBlocks + 64) * sizeof(int32_t);      // the blocks' maxima, the verdict
constexpr size_t kMaxWorkspace = (size_t)2 << 30;      // scratch a call may take; beyond it the CUDA cores do the work

int64_t pitch_of(int64_t cols) { return (cols + 7) / 8 * 8; }
size_t plane_bytes(int64_t rows, int64_t cols) { return (size_t)((rows * pitch_of(cols) * 2 * kPlanes + 255) / 256 * 256); }

// Where the tensor cores win, by a model of both sides in us.  Here: full waves of 256 x 256 tiles at 1.9 us per k-block and
// 5 us to fill, drain and store, the planes (10 bytes per value) and the epilogue pass at 6 TB/s, 12 us for three more
// launches; it comes within 10 % of [16384, 3072 x 768] top-2 (919 us, CUDA cores 3333), [8192, 2048 x 512] top-2 (274 / 811)
// and 5000 rows over 32 experts (212 / 393).  CUDA cores: whole tiles at the 44 TFLOP/s of the 128-tile kernel or the 30 of
// the 64-tile one.  Between the two the line lies around 2-3 GFLOP; 15 % is kept as margin.
bool pays(int64_t tiles, int64_t kb, double split_values, double pass_values, int64_t simt_m, int64_t simt_n, double simt_depth) {
  const double waves = (double)ceil_div(tiles, sm_count() / 2);
  const double tc = waves * ((double)kb * 1.9 + 5.0) + 10.0 * (split_values + pass_values) / 6e6 + 12.0;
  const bool large = ceil_div(simt_m, 128) * ceil_div(simt_n, 128) >= 2 * (int64_t)sm_count();
  const int64_t tile = large ? 128 : 64;
  const double flops = 2.0 * (double)(ceil_div(simt_m, tile) * ceil_div(simt_n, tile) * tile * tile) * simt_depth;
  return tc * 1.15 < flops / (large ? 44e6 : 30e6);
}

// Writes both operands' planes and tells `p` where their maxima are and the verdict goes.
int split_launch(const Side& a, const Side& b, uint8_t* ws, int64_t terms, Params& p, cudaStream_t stream) {
  const int64_t want = ceil_div(a.rows * a.E + b.rows * b.E, 8);
  int64_t blocks = (int64_t)sm_count() * 8;
  if (blocks > kMaxSplitBlocks) blocks = kMaxSplitBlocks;
  if (want < blocks) blocks = want > 0 ? want : 1;
  uint32_t* maxima = reinterpret_cast<uint32_t*>(ws);
  after_previous(split_planes_kernel, (unsigned)blocks, 256, 0, stream)(a, b, maxima);
  HEXA_LAUNCH_CHECK("split_planes_kernel");
  p.maxima = maxima;
  p.n_maxima = (int)blocks;
  p.terms = (int)(terms < INT32_MAX ? terms : INT32_MAX);
  p.redo = reinterpret_cast<int32_t*>(ws) + 2 * kMaxSplitBlocks;
  return HEXA_OK;
}

Side make_side(const void* src, int64_t ld, int64_t estride, int64_t E, int64_t rows, int64_t cols, const int32_t* limit, void* dst) {
  Side s{static_cast<const float*>(src), ld, estride, rows, cols, E, limit, static_cast<__nv_bfloat16*>(dst), pitch_of(cols), 0, 0};
  s.plane = E * rows * s.pitch;
  s.vec = aligned16(src) && ld % 4 == 0 && (E == 1 || estride % 4 == 0) && cols % 4 == 0;
  return s;
}

int plane_map(CUtensorMap* tm, const Side& s, bool with_expert, uint32_t box0, uint32_t box1) {
  const uint64_t row = (uint64_t)s.pitch * 2;
  if (with_expert) {
    const uint64_t dims[4] = {(uint64_t)s.cols, (uint64_t)s.rows, (uint64_t)s.E, kPlanes};
    const uint64_t str[3] = {row, row * (uint64_t)s.rows, (uint64_t)s.plane * 2};
    const uint32_t box[4] = {box0, box1, 1, kPlanes};
    return encode_tensor_map(tm, s.dst, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
  }
  const uint64_t dims[3] = {(uint64_t)s.cols, (uint64_t)s.rows, kPlanes};
  const uint64_t str[2] = {row, (uint64_t)s.plane * 2};
  const uint32_t box[3] = {box0, box1, kPlanes};
  return encode_tensor_map(tm, s.dst, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

template <int MODE>
int launch(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC, const Params& p, int64_t max_tiles, cudaStream_t stream) {
  static bool attr_set[64] = {false};
  static int max_clusters[64] = {0};
  auto kernel = gemm_f32_kernel<MODE>;
  int dev = 0;
  HEXA_CUDA(cudaGetDevice(&dev));
  HEXA_REQUIRE(dev >= 0 && dev < 64, "device ordinal %d out of range", dev);
  if (!attr_set[dev]) {
    HEXA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
    attr_set[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // see after_previous
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  if (max_clusters[dev] == 0) {
    cfg.gridDim = dim3(2 * (unsigned)(sm_count() / 2));
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) { (void)cudaGetLastError(); n = sm_count() / 2; }
    max_clusters[dev] = n;
  }
  int64_t pairs = max_tiles < max_clusters[dev] ? max_tiles : max_clusters[dev];
  if (sm_limit() > 0 && pairs > sm_limit() / 2) pairs = sm_limit() / 2;
  cfg.gridDim = dim3((unsigned)(2 * (pairs > 0 ? pairs : 1)));
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, tmA, tmB, tmC, p);
  if (e != cudaSuccess) {
    set_error("launch of gemm_f32_kernel<%d> failed: %s", MODE, cudaGetErrorString(e));
    return HEXA_ERR_CUDA;
  }
  count_launch();
  return HEXA_OK;
}

}  // namespace

size_t esmm_f32_workspace_bytes(int E, int64_t row_cap, int64_t n_out, int64_t k) {
  if (E <= 0 || row_cap <= 0 || n_out <= 0 || k <= 0) return 0;
  const int64_t pairs = row_cap / (2 * kRowTile) + E / 2;
  const double rows = (double)row_cap, n = (double)n_out, kk = (double)k;
  if (!pays(pairs * ceil_div(n_out, BLOCK_N), ceil_div(k, BLOCK_K), rows * kk + (double)E * n * kk, rows * n, row_cap, n_out, kk)) return 0;
  // either layout of b: the wider pitch of the two
  const size_t b = plane_bytes((int64_t)E * n_out, k), bt = plane_bytes((int64_t)E * k, n_out);
  const size_t total = kFlagBytes + plane_bytes(row_cap, k) + (b > bt ? b : bt);
  return total <= kMaxWorkspace ? total : 0;
}

size_t estmm_f32_workspace_bytes(int E, int64_t row_cap, int64_t m, int64_t n) {
  if (E <= 0 || row_cap <= 0 || m <= 0 || n <= 0) return 0;
  // A chain of few FMAs is as exact as its last rounding, planes are not: relative error of an expert's gradient from 1 row
  // 2.5e-8 as a chain, 4.5e-8 from planes, from 8 rows 5.4 / 4.7 (positive data 4.7 / 4.8), from 16 rows 7.4 / 4.8 (6.3 / 4.9).
  // Of the capacity up to 127 rows per expert are padding, the rest is the real rows.
  if (row_cap - 127 * (int64_t)E < 16 * (int64_t)E) return 0;
  const int64_t tiles = (int64_t)E * ceil_div(m, 2 * BLOCK_M) * ceil_div(n, BLOCK_N);
  const double rows = (double)row_cap;
  if (!pays(tiles, ceil_div(row_cap / BLOCK_K, E), rows * (double)(m + n), 0.0, m * E, n, rows / E)) return 0;
  const size_t total = kFlagBytes + plane_bytes(row_cap, m) + plane_bytes(row_cap, n);
  return total <= kMaxWorkspace ? total : 0;
}

int esmm_f32_launch(const void* a, int64_t lda, const void* b, int b_layout, int64_t ldb, int64_t b_estride, const float* bias,
                    int64_t ldbias, void* aux, int64_t ldaux, void* c, int64_t ldc, const int32_t* tile_expert,
                    const int32_t* pad_offsets, const int32_t* row_token, const int32_t* pair_block, int E, int64_t row_cap,
                    int64_t n_out, int64_t k, int epilogue, int act, cudaStream_t stream, void* workspace) {
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  const bool nk = b_layout == HEXA_B_NK;
  const Side sa = make_side(a, lda, 0, 1, row_cap, k, pad_offsets + E, ws + kFlagBytes);
  const Side sb = make_side(b, ldb, b_estride, E, nk ? n_out : k, nk ? k : n_out, nullptr, ws + kFlagBytes + plane_bytes(row_cap, k));
  Params p{};
  int rc = split_launch(sa, sb, ws, k, p, stream);
  if (rc) return rc;
  CUtensorMap tmA, tmB, tmC;
  if ((rc = plane_map(&tmA, sa, false, BLOCK_K, BLOCK_M))) return rc;
  if ((rc = nk ? plane_map(&tmB, sb, true, BLOCK_K, 128) : plane_map(&tmB, sb, true, 64, BLOCK_K))) return rc;
  // the linear result: where the saved pre-activation belongs, else in c
  const bool pre = epilogue == HEXA_EPI_ACT && aux != nullptr;
  {
    const uint64_t dims[2] = {(uint64_t)n_out, (uint64_t)row_cap};
    const uint64_t str[1] = {(uint64_t)(pre ? ldaux : ldc) * 4};
    const uint32_t box[2] = {kSlab, BLOCK_M};
    if ((rc = encode_tensor_map(&tmC, pre ? aux : c, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_64B))) return rc;
  }
  p.tile_expert = tile_expert; p.pad_offsets = pad_offsets; p.row_token = row_token; p.pair_block = pair_block;
  p.max_pairs = row_cap / (2 * BLOCK_M) + E;
  p.bias = bias; p.ldbias = ldbias; p.n = n_out; p.k = k; p.E = E;
  p.nt = (uint32_t)ceil_div(n_out, BLOCK_N);
  p.status = status_word(); p.debug = tc_debug_flags(); p.wait_limit_ns = wait_limit_ns(); p.next_may_start = sm_limit() == 0;
  HEXA_REQUIRE((row_cap / BLOCK_M + E + 1) * (int64_t)p.nt < (int64_t)0x7fffffff, "hexa_esmm: too many output tiles for a 32-bit tile index");
  const int64_t max_tiles = p.max_pairs * (int64_t)p.nt;
  rc = nk ? launch<NK>(tmA, tmB, tmC, p, max_tiles, stream) : launch<KN>(tmA, tmB, tmC, p, max_tiles, stream);
  if (rc) return rc;
  if (epilogue != HEXA_EPI_LINEAR) {
    const float* x = static_cast<const float*>(epilogue == HEXA_EPI_DACT || pre ? aux : c);
    const int64_t ldx = epilogue == HEXA_EPI_DACT || pre ? ldaux : ldc;
    const bool v4 = n_out % 4 == 0 && ldx % 4 == 0 && ldc % 4 == 0 && aligned16(x) && aligned16(c);
    const unsigned grid = (unsigned)sm_count() * 8;
    if (v4) after_previous(epilogue_rows_kernel<4>, grid, 256, 0, stream)(x, ldx, static_cast<float*>(c), ldc, row_token, pad_offsets, E, n_out, epilogue, act);
    else after_previous(epilogue_rows_kernel<1>, grid, 256, 0, stream)(x, ldx, static_cast<float*>(c), ldc, row_token, pad_offsets, E, n_out, epilogue, act);
    HEXA_LAUNCH_CHECK("epilogue_rows_kernel");
  }
  return esmm_simt_launch(a, lda, b, b_layout, ldb, b_estride, bias, ldbias, aux, ldaux, c, ldc, tile_expert, pad_offsets, row_token, E,
                          row_cap, n_out, k, HEXA_F32, epilogue, act, stream, 0, E, 0, p.redo);
}

int estmm_f32_launch(const void* pp, int64_t ldp, const void* q, int64_t ldq, const int32_t* pad_offsets, int E, int64_t row_cap,
                     int64_t m, int64_t n, void* out, int64_t ldo, int64_t o_estride, cudaStream_t stream, void* workspace) {
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  const Side sp = make_side(pp, ldp, 0, 1, row_cap, m, pad_offsets + E, ws + kFlagBytes);
  const Side sq = make_side(q, ldq, 0, 1, row_cap, n, pad_offsets + E, ws + kFlagBytes + plane_bytes(row_cap, m));
  Params p{};
  int rc = split_launch(sp, sq, ws, row_cap, p, stream);
  if (rc) return rc;
  CUtensorMap tmA, tmB, tmC;
  if ((rc = plane_map(&tmA, sp, false, 64, BLOCK_K))) return rc;
  if ((rc = plane_map(&tmB, sq, false, 64, BLOCK_K))) return rc;
  {
    const uint64_t dims[3] = {(uint64_t)n, (uint64_t)m, (uint64_t)E};
    const uint64_t str[2] = {(uint64_t)ldo * 4, (uint64_t)o_estride * 4};
    const uint32_t box[3] = {kSlab, BLOCK_M, 1};
    if ((rc = encode_tensor_map(&tmC, out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_64B))) return rc;
  }
  p.pad_offsets = pad_offsets; p.n = n; p.m = m; p.E = E;
  p.nt = (uint32_t)ceil_div(n, BLOCK_N);
  const int64_t per_expert = ceil_div(m, 2 * BLOCK_M) * (int64_t)p.nt;
  HEXA_REQUIRE(per_expert * E < (int64_t)0x7fffffff, "hexa_estmm: too many output tiles for a 32-bit tile index");
  p.per_expert = (uint32_t)per_expert;
  p.total_tiles = (uint32_t)(per_expert * E);
  p.status = status_word(); p.debug = tc_debug_flags(); p.wait_limit_ns = wait_limit_ns(); p.next_may_start = sm_limit() == 0;
  rc = launch<TN>(tmA, tmB, tmC, p, per_expert * E, stream);
  if (rc) return rc;
  return estmm_simt_launch(pp, ldp, q, ldq, pad_offsets, E, m, n, out, ldo, o_estride, m, 0, HEXA_F32, HEXA_F32, 0, stream, p.redo);
}

}  // namespace hexa
