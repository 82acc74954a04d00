// tcgen05 / TMEM / TMA grouped GEMMs on the sorted-row layout (sm_100a only):
//   ESMM   c[r,:]  = a[r,:] x b[expert(r)]   (b K-major "NK" or N-major "KN"), fused bias / activation /
//                    activation-derivative epilogue, pad rows written as zeros
//   ESTMM  out[e]  = p_e^T x q_e             (contraction over the expert's ragged row segment; both
//                    operands are MN-major in shared memory, no transposed copy is ever made)
//
// Persistent kernel, static tile list.  Two flavours of the same code (template parameter CTAS):
//   CTAS = 1  one CTA per SM computes a 128 x BN tile (tcgen05 cta_group::1)
//   CTAS = 2  a cluster of two CTAs on neighbouring SMs computes a 256 x 256 tile (cta_group::2): each CTA
//             loads its own 128 rows of A and only HALF of the B tile, the pair's MMA reads both halves, and
//             each CTA keeps its 128 x 256 accumulator in its own TMEM.  Shared-memory fill traffic per MMA
//             drops from 48 KB to 32 KB per SM per 64-deep k-block, which is what bounds the 1-CTA kernel.
//             No TMA multicast is used.
// Warp roles in every CTA:
//   warp 0      TMA producer: 128B-swizzled k-blocks of A and B into a ring of shared-memory stages
//   warp 1      MMA issuer (only in the pair's leader CTA when CTAS = 2): one thread issues tcgen05.mma
//               (K = 16 per instruction) into one of two TMEM accumulators; tcgen05.commit frees ring slots
//               and publishes finished accumulators (multicast to both CTAs of a pair)
//   warps 2..17 epilogue: tcgen05.ld of the accumulator (lane quadrant = warp % 4, each group of four warps owns a column
//               range), fused epilogue math; results go through 64B-swizzled staging tiles and one TMA store per 128x32
//               block (an unsplit ESTMM with fp32, accumulating or scattered output stores from registers).  A kernel per
//               epilogue (Out below), because they want different things of shared memory:
//                 LINEAR, ACT  every warp stages and stores its own 32 rows (ACT: pre-activation and output side by side, two
//                         staging tiles per group), so that no warp waits for the group between the tile's first barrier
//                         and the next tile: fc1 + GELU of [18432, 2048 x 512] 77 -> 69 us, 32 experts x 144 rows x
//                         [4096 x 1024] 93 -> 87 us, long k-loops within 2 % (ESTMM's stores measured 10 % slower this way)
//                 DACT    two staging tiles per group that first receive the saved pre-activation by TMA, a block ahead,
//                         and are overwritten in place by the result.  Reading it with per-thread loads (32 rows x 16 B
//                         per instruction, each behind the previous block's math) cost 214 us where this costs 171
//                         ([32768 rows, 3072 x 768], bf16, GELU'; 1336 where 1240 at [131072, 4096 x 1024] skewed)
//                 STAGED  ESTMM's 16-bit [E, m, n] outputs: 145 us with register stores (a row per lane, half-used
//                         sectors), 75 through the staging tile (32 experts x 4096 x 1024 from 144 rows each; long
//                         segments measure the same either way)
//                 PARTIAL a split ESTMM's fp32 partial results: the accumulator is drained every few k-blocks into fp32
//                         registers, which bounds its truncating chains whatever the length of a chunk, and the sums
//                         leave through the staging tile (see estmm_tc_plan)
//               The tile's bias is put into shared memory by the group a tile ahead (fc1 + GELU of [32768 rows, 3072 x 768]:
//               209 -> 196 us, the 16 per-thread global loads of a block sat in front of the math; 171-177 with the stores per
//               warp).  Loading all 32
//               columns of a block from TMEM at once instead of 16 + 16 spilled and was 20 % slower.
// so the epilogue of tile i overlaps the MMAs of tile i+1.  Every mbarrier wait is bounded: after ~2 s a CTA
// raises an abort flag, records a code in the status word and drains; both CTAs of a pair always reach the
// closing cluster barrier.
//
// Segments are aligned to 128 rows, so an ESMM row block never straddles two experts and an ESTMM k-block
// (64 rows) never reads another expert's rows; pad rows hold zeros and add nothing.  A pair tile takes two
// consecutive row blocks of the same expert (list built by the routing step); an expert with an odd number of
// blocks leaves the second CTA of its last pair without rows to store.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <stdlib.h>

#include "gemm_launch.h"
#include "hexa_common.cuh"
#include "tc_ptx.cuh"

namespace hexa {
namespace {

constexpr int BLOCK_M = 128;
constexpr int BLOCK_K = 64;   // one 128-byte swizzle span of 16-bit elements
constexpr int UMMA_K = 16;
constexpr uint32_t kABytes = BLOCK_M * BLOCK_K * 2;  // 16 KB

enum Mode { ESMM_NK = 0, ESMM_KN = 1, ESTMM = 2 };

struct Params {
  const int32_t* tile_expert;
  const int32_t* pad_offsets;
  const int32_t* row_token;
  const int32_t* pair_block;   // CTAS = 2, ESMM: per pair tile (first 128-row block) * 2 + (second block belongs to the same expert), -1 ends the list
  int64_t max_pairs;
  const void* bias;
  int64_t ldbias;
  int bias16;       // the bias is of the data's type instead of fp32
  void* aux;
  int64_t ldaux;
  void* c;          // ESMM: c ; ESTMM: out
  int64_t ldc;
  int64_t c_estride;  // ESTMM only
  int64_t m_split, split_stride;  // ESTMM: output row m lives at (m / m_split) * split_stride + (m % m_split) * ldc
  void* c_split[16];  // ESTMM, n_split > 0: slice m / m_split of the output goes to this base instead (it may be
  int n_split;        // another GPU's memory: the reduce-scatter layout written straight into the owners' buffers)
  int64_t n;        // output columns
  int64_t k;        // ESMM: contraction length ; ESTMM: unused
  int64_t m;        // ESTMM: output rows per expert
  int E;
  uint32_t nt;          // tile columns of the output: ceil(n / BN)
  uint32_t per_expert;  // ESTMM: tiles per expert = tile rows x tile columns x splits
  uint32_t total_tiles; // ESTMM: E x per_expert ; ESMM single-CTA: unused (the row count is device-side)
  int e_begin, e_end;   // ESMM: only tiles of experts in [e_begin, e_end) are computed by this launch
  int epilogue, act;
  int is_bf16;      // 16-bit flavour of the inputs (and of 16-bit outputs)
  int out_f32;      // ESTMM: fp32 output
  int beta;         // ESTMM: accumulate into out
  int splits;       // ESTMM: > 1 = every expert's row segment is cut into this many chunks, each its own tile, whose fp32
                    //        partial results [splits, E, m, n] are added in chunk order by estmm_reduce_kernel
  int chains;       // ESTMM with splits > 1: a chunk's k-blocks are accumulated in this many chains
  float* colsum;    // ESMM, optional: fp32 [row_capacity / 128, n]; row b receives the column sums of the 128 output rows
                    // of block b, taken from the values as they are stored (after rounding to the 16-bit type)
  int debug;        // test aid (hexa_set_tc_debug): bit 2 = the producer neither loads nor arrives, bit 3 = the derivative's saved
                    // pre-activation is not requested, so that the waits behind them run into their limit
  int32_t* status;
  uint64_t wait_limit_ns;   // limit of every mbarrier wait (hexa_set_wait_limit_ns; default 2 s)
  bool next_may_start;      // no SM limit is set, see wait_for_previous
};

// What the epilogue does with an accumulator.  ESMM: HEXA_EPI_LINEAR / HEXA_EPI_ACT / HEXA_EPI_DACT; ESTMM: stores from
// registers (any output form) or through staging tiles (16-bit [E, m, n] outputs; fp32 partial results of a split).
enum Out { OUT_LINEAR = HEXA_EPI_LINEAR, OUT_ACT = HEXA_EPI_ACT, OUT_DACT = HEXA_EPI_DACT, OUT_REGISTERS = 3, OUT_STAGED = 4, OUT_PARTIAL = 5 };

template <int BN, int CTAS, int MODE, int OUT> struct Cfg {
  static constexpr int kEpiWarps = 16;
  static constexpr int kThreads = 32 * (2 + kEpiWarps);
  static constexpr int kParts = kEpiWarps / 4;          // groups of four warps; each owns BN / kParts columns of every tile
  static constexpr int kBlocks = BN / kParts / 32;      // as this many 128 x 32 blocks
#ifndef HEXA_TC_SMEM_SLACK      // bytes kept for aligning the dynamic shared memory base to 1 KB by hand
#define HEXA_TC_SMEM_SLACK 1024
#endif
  // 128 x 32 staging tiles per group: one where the epilogue has nothing to wait for but its own stores; two where it
  // writes two outputs (ACT) or reads the saved pre-activation through the same tile (DACT); none for register stores.
  // The ring has the rest of the shared memory (32 KB per slot; 48 KB for single-CTA 256-column tiles).
  static constexpr int kBufs = OUT == OUT_REGISTERS ? 0 : (OUT == OUT_ACT || OUT == OUT_DACT) ? 2 : 1;
  static constexpr uint32_t kBBytes = (BN / CTAS) * BLOCK_K * 2;   // this CTA's share of the B tile
  static constexpr uint32_t kStageBytes = kABytes + kBBytes;
  static constexpr uint32_t kTmemCols = 2 * BN;  // two accumulators; 256 or 512, a power of two
  static constexpr uint32_t kStoreBufBytes = 128 * 64;   // [128 rows x 32 16-bit columns]
  static constexpr uint32_t kStoreBytes = kBufs * kParts * kStoreBufBytes;
  static constexpr uint32_t kBiasBytes = MODE == ESTMM ? 0 : BN * 4;      // the tile's bias, a part per group
  static constexpr int kStages = (232448 - HEXA_TC_SMEM_SLACK - 512 - kBiasBytes - kStoreBytes) / kStageBytes;
  static constexpr size_t kSmemBytes = HEXA_TC_SMEM_SLACK + (size_t)kStages * kStageBytes + kStoreBytes + kBiasBytes + 512 /*barriers*/;
  static_assert(kSmemBytes <= 232448, "more shared memory than one CTA can have (227 KB)");
};

struct Tile {
  int e;          // expert
  int row0;       // ESMM: first sorted row of this CTA's block ; ESTMM: first row of the expert's segment
  int col0;       // first output column of the tile
  int m0;         // ESTMM: first output row of this CTA's block
  int num_kb;     // k-blocks to accumulate
  int valid;      // this CTA has rows to store (the second CTA of a pair may not)
  int skip;       // ESMM: the tile's expert is outside the launch's expert range (every role skips it alike)
  int split;      // ESTMM with splits > 1: which chunk of the segment this tile covers
  int chain;      // ... and how many k-blocks one accumulation takes
};

// Tile t of the static list, as seen by CTA `rank` of its pair (rank = 0 when CTAS = 1).  Returns false past the end.
// The tile index and every quantity it is divided by are 32-bit (the host checks the tile count): the lookup runs once
// per tile in each of the three roles, two of which are single threads that the tensor pipe waits for, and a 64-bit
// division is a ~100-instruction sequence.
template <int BN, int MODE, int CTAS>
__device__ __forceinline__ bool get_tile(const Params& p, uint32_t t, int rank, Tile& tile) {
  if (MODE == ESTMM) {
    if (t >= p.total_tiles) return false;
    const uint32_t S = (uint32_t)p.splits;
    const uint32_t e = t / p.per_expert;
    const uint32_t in_e = t - e * p.per_expert;
    const uint32_t rem = in_e / S;
    const uint32_t c = in_e - rem * S;
    const uint32_t mrow = rem / p.nt;
    tile.e = (int)e;
    tile.m0 = ((int)mrow * CTAS + rank) * BLOCK_M;
    tile.col0 = (int)(rem - mrow * p.nt) * BN;
    const int seg0 = p.pad_offsets[e];
    const int kb_all = (p.pad_offsets[e + 1] - seg0) / BLOCK_K;
    const int kb_per = (kb_all + (int)S - 1) / (int)S;       // chunks of equal length, the last ones may be short or empty
    const int kb0 = (int)c * kb_per;
    tile.row0 = seg0 + kb0 * BLOCK_K;
    tile.num_kb = max(0, min(kb_per, kb_all - kb0));
    tile.split = (int)c;
    tile.chain = max(1, (kb_per + p.chains - 1) / p.chains);
    tile.skip = 0;
    tile.valid = tile.m0 < p.m;
    return true;
  } else {
    const uint32_t row_tile = t / p.nt;          // pair index (CTAS = 2) or 128-row block
    uint32_t mb;
    if (CTAS == 2) {
      if (row_tile >= (uint32_t)p.max_pairs) return false;
      const int pb = p.pair_block[row_tile];
      if (pb < 0) return false;
      mb = (uint32_t)(pb >> 1);
      tile.e = p.tile_expert[mb];
      tile.valid = rank == 0 || (pb & 1);
      mb += (uint32_t)rank;
    } else {
      const uint32_t mblocks = (uint32_t)(p.pad_offsets[p.E] / BLOCK_M);
      if (row_tile >= mblocks) return false;
      mb = row_tile;
      tile.e = p.tile_expert[mb];
      tile.valid = 1;
    }
    tile.row0 = (int)(mb * BLOCK_M);
    tile.col0 = (int)(t - row_tile * p.nt) * BN;
    tile.m0 = 0;
    tile.num_kb = (int)((p.k + BLOCK_K - 1) / BLOCK_K);
    tile.skip = tile.e < p.e_begin || tile.e >= p.e_end;
    return tile.e >= 0;
  }
}

// Half of that row: 16 columns = chunks 2 hf and 2 hf + 1.
__device__ __forceinline__ void stage_half(uint8_t* buf, int r, int hf, const uint32_t (&w)[8]) {
  uint8_t* row = buf + r * 64;
  const int x = (r >> 1) & 3;
#pragma unroll
  for (int c = 0; c < 2; ++c)
    *reinterpret_cast<uint4*>(row + (((2 * hf + c) ^ x) << 4)) = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
}
__device__ __forceinline__ void load_half(const uint8_t* buf, int r, int hf, uint32_t (&w)[8]) {
  const uint8_t* row = buf + r * 64;
  const int x = (r >> 1) & 3;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const uint4 a = *reinterpret_cast<const uint4*>(row + (((2 * hf + c) ^ x) << 4));
    w[4 * c] = a.x; w[4 * c + 1] = a.y; w[4 * c + 2] = a.z; w[4 * c + 3] = a.w;
  }
}

// Values of 16 columns of one row for the two possible outputs of the ESMM epilogue: y = acc + bias packed as it
// is (the saved pre-activation), o = the layer output of this GEMM.  Rows that are padding come out as zeros without a
// select per element: their accumulator is exactly zero (the A operand's pad rows are zeros), the caller has masked
// their bias, and every activation here maps 0 to 0 (the derivative epilogue multiplies the zero accumulator).  Working
// on 16 columns at a time keeps few enough values live for the compiler to interleave the independent activations.
template <int OUT, int ACT, int is_bf16>
__device__ __forceinline__ void epi_values16(const float (&f)[16], const uint32_t (&x)[8], uint32_t* y, uint32_t* o) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (OUT == OUT_DACT) {
      o[i] = pack2(f[2 * i] * act_grad_fast<ACT>(unpack_lo(x[i], is_bf16)),
                   f[2 * i + 1] * act_grad_fast<ACT>(unpack_hi(x[i], is_bf16)), is_bf16);
    } else if (OUT == OUT_ACT) {
      y[i] = pack2(f[2 * i], f[2 * i + 1], is_bf16);
      o[i] = pack2(act_fast<ACT>(f[2 * i]), act_fast<ACT>(f[2 * i + 1]), is_bf16);
    } else {
      o[i] = pack2(f[2 * i], f[2 * i + 1], is_bf16);
    }
  }
}
template <int OUT>
__device__ __forceinline__ void epi_dispatch16(int act, int is_bf16, const float (&f)[16], const uint32_t (&x)[8], uint32_t* y, uint32_t* o) {
  // one specialisation per (activation, 16-bit flavour): no per-element branches
#define HEXA_EPI_CASE(A_)                                                  \
  case A_:                                                                 \
    if (is_bf16) epi_values16<OUT, A_, 1>(f, x, y, o);                     \
    else epi_values16<OUT, A_, 0>(f, x, y, o);                             \
    break;
  if (OUT == OUT_LINEAR) act = HEXA_ACT_NONE;
  switch (act) {
    HEXA_EPI_CASE(HEXA_ACT_RELU)
    HEXA_EPI_CASE(HEXA_ACT_GELU)
    HEXA_EPI_CASE(HEXA_ACT_GELU_TANH)
    HEXA_EPI_CASE(HEXA_ACT_SILU)
    default:
      if (is_bf16) epi_values16<OUT, HEXA_ACT_NONE, 1>(f, x, y, o);
      else epi_values16<OUT, HEXA_ACT_NONE, 0>(f, x, y, o);
  }
#undef HEXA_EPI_CASE
}

// The tile list as the epilogue walks it (ESMM): the entry of the next tile is requested while this one is worked on.
// entry = (first 128-row block of the tile) * 2 + (the second block is this expert's as well), -1 past the end.
template <int CTAS>
__device__ __forceinline__ int tile_entry(const Params& p, uint32_t t, uint32_t row_tiles) {
  const uint32_t row_tile = t / p.nt;
  if (row_tile >= row_tiles) return -1;
  return CTAS == 2 ? p.pair_block[row_tile] : (int)(row_tile * 2);
}

template <int BN, int MODE, int CTAS, int OUT>
__global__ void __launch_bounds__(Cfg<BN, CTAS, MODE, OUT>::kThreads, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmX, const Params p) {
  using C = Cfg<BN, CTAS, MODE, OUT>;
  constexpr int kEpiWarps = C::kEpiWarps;
  constexpr int kStages = C::kStages;
  constexpr int BNH = BN / CTAS;          // B columns this CTA loads
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  if (HEXA_TC_SMEM_SLACK < 1024 && smem != smem_raw) {      // without slack the base itself must be 1 KB aligned
    if (threadIdx.x == 0) report_status(p.status, 9);
    return;                                                  // uniform: every thread of every CTA sees the same base offset
  }
  uint8_t* store_bufs = smem + (size_t)kStages * C::kStageBytes;
  float* bias_s = reinterpret_cast<float*>(store_bufs + C::kStoreBytes);      // [BN] ESMM
  uint64_t* bars = reinterpret_cast<uint64_t*>(store_bufs + C::kStoreBytes + C::kBiasBytes);
  uint64_t* full = bars;                  // [kStages]  producers -> MMA     (used in the leader CTA)
  uint64_t* empty = bars + kStages;       // [kStages]  MMA -> producer      (one per CTA, multicast commit)
  uint64_t* acc_full = bars + 2 * kStages;        // [2] MMA -> epilogue     (one per CTA, multicast commit)
  uint64_t* acc_empty = bars + 2 * kStages + 2;   // [2] epilogues -> MMA    (used in the leader CTA)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint64_t* aux_full = bars + 2 * kStages + 8;   // [kParts][2] DACT: the saved pre-activation is in the group's staging tile

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = CTAS == 2 ? (int)cluster_ctarank() : 0;    // 0 = leader of the pair
  const uint32_t tile_first = CTAS == 2 ? (blockIdx.x >> 1) : blockIdx.x;
  const uint32_t tile_step = CTAS == 2 ? (gridDim.x >> 1) : gridDim.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], kEpiWarps * CTAS); }
    *abort_flag = 0;
    if (OUT == OUT_DACT)
      for (int g = 0; g < 2 * C::kParts; ++g) mbar_init(&aux_full[g], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // the allocating warp also frees; with CTAS = 2 the same warp of both CTAs takes part
    if (CTAS == 2) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(C::kTmemCols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(C::kTmemCols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (CTAS == 2) cluster_sync_all();   // the peer's barriers exist before anything is sent to them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  wait_for_previous(p.next_may_start);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (every CTA)
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      Tile tile;
      const uint32_t lead_full0 = CTAS == 2 ? map_to_cta(&full[0], 0) : 0u;   // the leader CTA's first full barrier
      for (uint32_t t = tile_first; ok && get_tile<BN, MODE, CTAS>(p, t, rank, tile); t += tile_step) {
        if (MODE != ESTMM && tile.skip) continue;
        for (int kb = 0; kb < tile.num_kb; ++kb) {
          if (!(ok = mbar_wait_fast(&empty[stage], phase ^ 1, abort_flag, p.status, 1, p.wait_limit_ns))) break;
          uint8_t* sA = smem + (size_t)stage * C::kStageBytes;
          uint8_t* sB = sA + kABytes;
          const int bcol = tile.col0 + rank * BNH;     // this CTA's share of the B columns
          if (p.debug & 4) {
            // nothing is loaded and nobody arrives: the consumers' waits run into their limit (error-path test)
          } else if (CTAS == 2) {
            // bytes of both CTAs are credited to the leader's barrier; only the leader arms it
            const uint32_t lead_full = lead_full0 + 8u * (uint32_t)stage;
            if (rank == 0) mbar_expect_tx(&full[stage], 2 * C::kStageBytes);
            if (MODE == ESTMM) {
              const int r = tile.row0 + kb * BLOCK_K;
#pragma unroll
              for (int c = 0; c < BLOCK_M / 64; ++c) tma_load_2d_pair(sA + c * 8192, &tmA, lead_full, tile.m0 + c * 64, r);
#pragma unroll
              for (int c = 0; c < BNH / 64; ++c) tma_load_2d_pair(sB + c * 8192, &tmB, lead_full, bcol + c * 64, r);
            } else {
              tma_load_2d_pair(sA, &tmA, lead_full, kb * BLOCK_K, tile.row0);
              if (MODE == ESMM_NK) {
                tma_load_3d_pair(sB, &tmB, lead_full, kb * BLOCK_K, bcol, tile.e);
              } else {
#pragma unroll
                for (int c = 0; c < BNH / 64; ++c) tma_load_3d_pair(sB + c * 8192, &tmB, lead_full, bcol + c * 64, kb * BLOCK_K, tile.e);
              }
            }
          } else {
            mbar_expect_tx(&full[stage], C::kStageBytes);
            if (MODE == ESTMM) {
              const int r = tile.row0 + kb * BLOCK_K;
#pragma unroll
              for (int c = 0; c < BLOCK_M / 64; ++c) tma_load_2d(sA + c * 8192, &tmA, &full[stage], tile.m0 + c * 64, r);
#pragma unroll
              for (int c = 0; c < BNH / 64; ++c) tma_load_2d(sB + c * 8192, &tmB, &full[stage], bcol + c * 64, r);
            } else {
              tma_load_2d(sA, &tmA, &full[stage], kb * BLOCK_K, tile.row0);
              if (MODE == ESMM_NK) {
                tma_load_3d(sB, &tmB, &full[stage], kb * BLOCK_K, bcol, tile.e);
              } else {
#pragma unroll
                for (int c = 0; c < BNH / 64; ++c) tma_load_3d(sB + c * 8192, &tmB, &full[stage], bcol + c * 64, kb * BLOCK_K, tile.e);
              }
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
      constexpr bool kAMn = (MODE == ESTMM), kBMn = (MODE != ESMM_NK);
      // instruction descriptor: fp32 accumulate, A/B format (0 = f16, 1 = bf16), majors, N>>3, M>>4
      // (M is 256 for a CTA pair: 128 rows from each CTA's shared memory into each CTA's TMEM)
      const uint32_t fmt = p.is_bf16 ? 1u : 0u;
      const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((kAMn ? 1u : 0u) << 15) | ((kBMn ? 1u : 0u) << 16) |
                             ((uint32_t)(BN >> 3) << 17) | ((uint32_t)((BLOCK_M * CTAS) >> 4) << 24);
      // K-major: 8-row groups 1024 B apart (SBO), LBO unused (1).  MN-major: 64-element column chunks
      // BLOCK_K*128 B apart (LBO), 8-k groups 1024 B apart (SBO).
      const uint32_t a_lbo = kAMn ? BLOCK_K * 128 : 16, b_lbo = kBMn ? BLOCK_K * 128 : 16;
      // start-address advance per K=16 step, in 16-byte units: 32 B inside the swizzle row (K-major)
      // or two 8-k groups = 2048 B (MN-major)
      const uint32_t a_step = kAMn ? (2048u >> 4) : (32u >> 4);
      const uint32_t b_step = kBMn ? (2048u >> 4) : (32u >> 4);
      // The issuing thread is the pacemaker of the whole kernel: everything loop-invariant is hoisted so that a
      // k-block costs one try_wait, two 64-bit adds, four MMAs and one commit.
      const uint32_t s0 = smem_u32(smem);
      const uint64_t adesc0 = make_smem_desc(s0, a_lbo, 1024);
      const uint64_t bdesc0 = make_smem_desc(s0 + kABytes, b_lbo, 1024);
      constexpr uint64_t kStageDesc = C::kStageBytes >> 4;    // descriptor start-address units per ring slot
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      Tile tile;
      int it = -1;
      for (uint32_t t = tile_first; ok && get_tile<BN, MODE, CTAS>(p, t, rank, tile); t += tile_step) {
        if (MODE != ESTMM && tile.skip) continue;
        int kb = 0;
        do {      // one accumulation: the whole tile, or (PARTIAL) the next chain of its k-blocks
          ++it;
          const int acc = it & 1;
          const uint32_t acc_phase = (uint32_t)(it >> 1) & 1u;
          if (!(ok = mbar_wait_fast(&acc_empty[acc], acc_phase ^ 1, abort_flag, p.status, 2, p.wait_limit_ns))) break;
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + (uint32_t)(acc * BN);
          uint32_t accumulate = 0;
          const int kb_end = OUT == OUT_PARTIAL ? min(kb + tile.chain, tile.num_kb) : tile.num_kb;
          for (; kb < kb_end; ++kb) {
            if (!(ok = mbar_wait_fast(&full[stage], phase, abort_flag, p.status, 3, p.wait_limit_ns))) break;
            const uint64_t adesc = adesc0 + (uint64_t)stage * kStageDesc;
            const uint64_t bdesc = bdesc0 + (uint64_t)stage * kStageDesc;
#pragma unroll
            for (int j = 0; j < BLOCK_K / UMMA_K; ++j) {
              if (CTAS == 2) umma_f16_pair(d_tmem, adesc + (uint64_t)(j * a_step), bdesc + (uint64_t)(j * b_step), idesc, j == 0 ? accumulate : 1u);
              else umma_f16(d_tmem, adesc + (uint64_t)(j * a_step), bdesc + (uint64_t)(j * b_step), idesc, j == 0 ? accumulate : 1u);
            }
            accumulate = 1;
            // slot reusable (in both CTAs) once these MMAs have read it
            if (CTAS == 2) umma_commit_pair(&empty[stage]); else umma_commit(&empty[stage]);
            if (++stage == kStages) { stage = 0; phase ^= 1; }
          }
          if (!ok) break;
          if (tile.num_kb > 0) {
            if (CTAS == 2) umma_commit_pair(&acc_full[acc]); else umma_commit(&acc_full[acc]);
          } else {  // empty segment: nothing to wait for, the epilogues write zeros
            mbar_arrive(&acc_full[acc]);
            if (CTAS == 2) mbar_arrive_cluster(map_to_cta(&acc_full[acc], 1));
          }
        } while (OUT == OUT_PARTIAL && kb < tile.num_kb);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue (every CTA, its own 128 rows)
    const int q = warp & 3;                 // TMEM lane quadrant this warp may read
    const int part = (warp - 2) >> 2;
    const int is_bf16 = p.is_bf16;
    const bool leader = (q == 2) && lane == 0;   // the first warp of every group of four issues the group's TMA copies
    uint8_t* bufs = store_bufs + (size_t)part * C::kBufs * C::kStoreBufBytes;
    const int rloc = q * 32 + lane;
    const int part_col = part * (BN / C::kParts);
    bool ok = true;
    int it = -1;
    // The four warps of a group meet at named barriers inside the tile, so they must leave together: after a wait that may
    // fail they meet at a barrier that gives all four the same verdict.
    auto accumulator_ready = [&](int acc, uint32_t acc_phase) {
      return group_all(1 + part, mbar_wait(&acc_full[acc], acc_phase, abort_flag, p.status, 4, p.wait_limit_ns));
    };
    auto accumulator_drained = [&](int acc) {      // hand it back to the (leader's) MMA warp
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CTAS == 2 && rank != 0) mbar_arrive_cluster(map_to_cta(&acc_empty[acc], 0));
        else mbar_arrive(&acc_empty[acc]);
      }
    };
    if constexpr (OUT == OUT_PARTIAL) {
      constexpr int kCols = C::kBlocks * 32;
      Tile tile;
      for (uint32_t t = tile_first; ok && get_tile<BN, MODE, CTAS>(p, t, rank, tile); t += tile_step) {
        float sum[kCols];
#pragma unroll
        for (int i = 0; i < kCols; ++i) sum[i] = 0.f;
        int kb = 0;
        do {
          ++it;
          const int acc = it & 1;
          if (!(ok = accumulator_ready(acc, (uint32_t)(it >> 1) & 1u))) break;
          tc_fence_after();
          const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * BN + part_col);
          if (tile.num_kb > 0) {
#pragma unroll
            for (int s = 0; s < kCols / 16; ++s) {
              uint32_t v[16];
              tmem_ld16(taddr + s * 16, v);
#pragma unroll
              for (int i = 0; i < 16; ++i) sum[s * 16 + i] += __uint_as_float(v[i]);
            }
          }
          accumulator_drained(acc);
          kb += tile.chain;
        } while (kb < tile.num_kb);
        if (!ok) break;
#pragma unroll
        for (int s = 0; s < kCols / 16; ++s) {
          const int64_t gcol = (int64_t)tile.col0 + part_col + s * 16;
          if (gcol < p.n && tile.valid) {      // uniform across the four warps of a group
            uint32_t w[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) w[i] = __float_as_uint(sum[s * 16 + i]);
            if (leader) bulk_wait_read<0>();   // the previous store has finished reading the buffer
            group_sync(1 + part);
            stage_row(bufs, rloc, w);
            fence_async_smem();
            group_sync(1 + part);
            if (leader) {      // rows and columns beyond the result are clipped
              tma_store_3d(&tmC, bufs, (int)gcol, tile.m0, tile.split * p.E + tile.e);
              bulk_commit();
            }
          }
        }
      }
    } else if constexpr (MODE == ESTMM) {
      Tile tile;
      for (uint32_t t = tile_first; get_tile<BN, MODE, CTAS>(p, t, rank, tile); t += tile_step) {
        ++it;
        const int acc = it & 1;
        if (!accumulator_ready(acc, (uint32_t)(it >> 1) & 1u)) break;
        tc_fence_after();
        const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * BN);
#pragma unroll 1
        for (int cc = 0; cc < C::kBlocks; ++cc) {
          const int cloc = part_col + cc * 32;
          const int64_t gcol = (int64_t)tile.col0 + cloc;
          if (gcol >= p.n || !tile.valid) break;  // uniform across the four warps of a group
          uint32_t v[32];
          if (tile.num_kb > 0) {
            tmem_ld32(t_row + (uint32_t)cloc, v);
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0u;
          }
          if constexpr (OUT == OUT_STAGED) {      // rows and columns beyond the output are clipped by the store
            uint32_t w[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) w[i] = pack2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]), is_bf16);
            if (leader) bulk_wait_read<0>();   // the previous store has finished reading the buffer
            group_sync(1 + part);
            stage_row(bufs, rloc, w);
            fence_async_smem();
            group_sync(1 + part);
            if (leader) {
              tma_store_3d(&tmC, bufs, (int)gcol, tile.m0, tile.e);
              bulk_commit();
            }
            continue;
          }
          const int64_t mrow = (int64_t)tile.m0 + rloc;
          if (mrow < p.m) {
            if (p.out_f32) {
              float* o = (p.n_split ? reinterpret_cast<float*>(p.c_split[mrow / p.m_split])
                                    : reinterpret_cast<float*>(p.c) + (mrow / p.m_split) * p.split_stride) +
                         (int64_t)tile.e * p.c_estride + (mrow % p.m_split) * p.ldc + gcol;
#pragma unroll
              for (int g = 0; g < 8; ++g) {
                if (gcol + g * 4 < p.n) {
                  float4 w = make_float4(__uint_as_float(v[4 * g]), __uint_as_float(v[4 * g + 1]),
                                         __uint_as_float(v[4 * g + 2]), __uint_as_float(v[4 * g + 3]));
                  if (p.beta) {
                    float4 old = *reinterpret_cast<float4*>(o + g * 4);
                    w.x += old.x; w.y += old.y; w.z += old.z; w.w += old.w;
                  }
                  *reinterpret_cast<float4*>(o + g * 4) = w;
                }
              }
            } else {
              uint16_t* o = (p.n_split ? reinterpret_cast<uint16_t*>(p.c_split[mrow / p.m_split])
                                       : reinterpret_cast<uint16_t*>(p.c) + (mrow / p.m_split) * p.split_stride) +
                            (int64_t)tile.e * p.c_estride + (mrow % p.m_split) * p.ldc + gcol;
#pragma unroll
              for (int g = 0; g < 4; ++g) {
                if (gcol + g * 8 < p.n) {
                  uint4 w;
                  uint32_t* wp = reinterpret_cast<uint32_t*>(&w);
                  if (p.beta) {
                    uint4 old = *reinterpret_cast<uint4*>(o + g * 8);
                    const uint32_t* op = reinterpret_cast<const uint32_t*>(&old);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                      wp[i] = pack2(__uint_as_float(v[8 * g + 2 * i]) + unpack_lo(op[i], is_bf16),
                                    __uint_as_float(v[8 * g + 2 * i + 1]) + unpack_hi(op[i], is_bf16), is_bf16);
                  } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                      wp[i] = pack2(__uint_as_float(v[8 * g + 2 * i]), __uint_as_float(v[8 * g + 2 * i + 1]), is_bf16);
                  }
                  *reinterpret_cast<uint4*>(o + g * 8) = w;
                }
              }
            }
          }
        }
        accumulator_drained(acc);
      }
    } else {
      const uint32_t row_tiles = CTAS == 2 ? (uint32_t)p.max_pairs : (uint32_t)(p.pad_offsets[p.E] / BLOCK_M);
      uint32_t t = tile_first;
      int entry = tile_entry<CTAS>(p, t, row_tiles);
      int e = entry >= 0 ? p.tile_expert[entry >> 1] : -1;
      uint32_t seq = 0;             // DACT: blocks done so far; block i uses staging tile i & 1
      bool requested = false;       // DACT, leader: the block about to start has its aux load under way
      auto request_aux = [&](uint32_t block, int64_t col, int row0) {
        if (p.debug & 8) return;
        uint64_t* bar = &aux_full[part * 2 + (block & 1)];
        mbar_expect_tx(bar, C::kStoreBufBytes);
        tma_load_2d(bufs + (block & 1) * C::kStoreBufBytes, &tmX, bar, (int)col, row0);
      };
      // Thread i of a group holds the bias of the group's i-th column of the tile ahead; it goes to shared memory between a
      // barrier that every warp reaches after its last read of the tile before (DACT: the last block's) and the tile's first.
      constexpr int kPartCols = BN / C::kParts;
      const int gi = q * 32 + lane;
      auto bias_of = [&](int expert, uint32_t tile_index) {
        const int64_t col = (int64_t)(tile_index % p.nt) * BN + part_col + gi;
        if (p.bias == nullptr || gi >= kPartCols || col >= p.n) return 0.f;
        const int64_t at = (int64_t)expert * p.ldbias + col;
        if (!p.bias16) return static_cast<const float*>(p.bias)[at];
        return unpack_lo(static_cast<const uint16_t*>(p.bias)[at], is_bf16);
      };
      float bias_next = entry >= 0 && e >= 0 ? bias_of(e, t) : 0.f;
      while (ok && entry >= 0 && e >= 0) {
        const uint32_t t_next = t + tile_step;
        if (OUT != OUT_DACT && p.bias != nullptr) group_sync(1 + part);
        if (gi < kPartCols) bias_s[part_col + gi] = bias_next;
        const int next = tile_entry<CTAS>(p, t_next, row_tiles);
        const int e_next = next >= 0 ? p.tile_expert[next >> 1] : -1;
        if (e >= p.e_begin && e < p.e_end) {
          ++it;
          const int acc = it & 1;
          const bool valid = rank == 0 || (entry & 1);
          const int row0 = ((entry >> 1) + rank) * BLOCK_M;
          const int64_t col0 = (int64_t)(t % p.nt) * BN;
          const int64_t r = (int64_t)row0 + rloc;
          // a pad row skips the bias, which is the only thing that could make it non-zero
          const bool live = p.bias != nullptr && valid && (p.row_token == nullptr || p.row_token[r] >= 0);
          if (!accumulator_ready(acc, (uint32_t)(it >> 1) & 1u)) break;
          tc_fence_after();
          const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * BN);
#pragma unroll 1
          for (int cc = 0; cc < C::kBlocks; ++cc) {
            const int cloc = part_col + cc * 32;
            const int64_t gcol = col0 + cloc;
            if (gcol >= p.n || !valid) break;  // uniform across the four warps of a group
            uint8_t* buf = bufs + (OUT == OUT_DACT ? (seq & 1) * C::kStoreBufBytes : 0);
            if (OUT == OUT_DACT) {
              // The other staging tile is free once its store has read it and the whole group is past its column sums
              // (the barrier): the next block's saved pre-activation is requested now and lands during this one.
              if (cc > 0) group_sync(1 + part);      // the first block's barrier was accumulator_ready's
              if (leader) {
                bulk_wait_read<0>();
                if (!requested) request_aux(seq, gcol, row0);
                requested = false;
                if (cc + 1 < C::kBlocks && gcol + 32 < p.n) {
                  request_aux(seq + 1, gcol + 32, row0);
                  requested = true;
                } else if (next >= 0 && (rank == 0 || (next & 1)) && e_next >= p.e_begin && e_next < p.e_end) {
                  const int64_t col_next = (int64_t)(t_next % p.nt) * BN + part_col;
                  if (col_next < p.n) {
                    request_aux(seq + 1, col_next, ((next >> 1) + rank) * BLOCK_M);
                    requested = true;
                  }
                }
              }
              __syncwarp();
              ok = mbar_wait_fast(&aux_full[part * 2 + (seq & 1)], (seq >> 1) & 1u, abort_flag, p.status, 5, p.wait_limit_ns);
            }
            const bool two = OUT == OUT_ACT && p.aux != nullptr;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
              uint32_t v[16];
              tmem_ld16(t_row + (uint32_t)(cloc + hf * 16), v);      // ESMM tiles always have k-blocks
              float f[16];
#pragma unroll
              for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(v[i]);
              if (live) {
                const float4* bp = reinterpret_cast<const float4*>(bias_s + cloc + hf * 16);
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                  const float4 bv = bp[g];
                  f[4 * g] += bv.x; f[4 * g + 1] += bv.y; f[4 * g + 2] += bv.z; f[4 * g + 3] += bv.w;
                }
              }
              uint32_t x[8], y[8], o[8];
              if (OUT == OUT_DACT) load_half(buf, rloc, hf, x);      // columns past the end came in as zeros
              epi_dispatch16<OUT>(p.act, is_bf16, f, x, y, o);
              // registers -> swizzled staging tile(s) -> one TMA store per 128x32 block (full 128-byte lines to L2)
              if (OUT != OUT_DACT && hf == 0) {      // (DACT writes over its own row of the saved pre-activation)
                if (lane == 0) bulk_wait_read<0>();  // this warp's previous stores have finished reading its rows of the buffers
                __syncwarp();
              }
              stage_half(buf, rloc, hf, o);
              if (two) stage_half(buf + C::kStoreBufBytes, rloc, hf, y);
            }
            fence_async_smem();
            if (OUT == OUT_DACT) {
              if (!(ok = group_all(1 + part, ok))) break;
              if (leader) {
                tma_store_2d(&tmC, buf, (int)gcol, row0);
                bulk_commit();
              }
            } else {      // every warp stores its own 32 rows: no warp waits for another
              __syncwarp();
              if (lane == 0) {
                uint8_t* mine = buf + q * 2048;
                if (two) tma_store_2d(&tmX, mine + C::kStoreBufBytes, (int)gcol, row0 + q * 32);
                tma_store_2d(&tmC, mine, (int)gcol, row0 + q * 32);
                bulk_commit();
              }
              if (p.colsum != nullptr) group_sync(1 + part);      // the other warps' rows are staged
            }
            ++seq;
            if (p.colsum != nullptr) {
              // Column sums of the block that now sits in the staging tile (the output as stored).  The warp whose TMEM
              // quadrant is q takes the 16-byte chunk q of every row: lane = (row mod 8) * 4 + 32-bit word within the
              // chunk (two columns), 16 rows per lane, then the eight row classes meet through three shuffles.  The eight
              // rows of one load fall into eight different groups of four banks (rows r, r+1 differ by 64 bytes, rows
              // r, r+2 by the swizzle): one conflict-free 128-byte wavefront per load.  Nothing else is synchronised:
              // every thread has finished reading before it arrives at the barrier that precedes the next write of the buffer.
              const int w4 = lane & 3, ro = lane >> 2;
              const uint8_t* src = buf + ro * 64 + ((q ^ ((ro >> 1) & 3)) << 4) + w4 * 4;   // (r >> 1) & 3 == (ro >> 1) & 3 for r = 8 i + ro
              float s0 = 0.f, s1 = 0.f;
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                const uint32_t v = *reinterpret_cast<const uint32_t*>(src + i * 512);
                s0 += unpack_lo(v, is_bf16);
                s1 += unpack_hi(v, is_bf16);
              }
#pragma unroll
              for (int d = 4; d < 32; d <<= 1) {
                s0 += __shfl_xor_sync(0xffffffffu, s0, d);
                s1 += __shfl_xor_sync(0xffffffffu, s1, d);
              }
              const int64_t col = gcol + q * 8 + w4 * 2;
              if (ro == 0 && col < p.n) {
                float* dst = p.colsum + (int64_t)(row0 / BLOCK_M) * p.n + col;
                dst[0] = s0;
                if (col + 1 < p.n) dst[1] = s1;
              }
              if (OUT != OUT_DACT) group_sync(1 + part);      // nobody overwrites rows that are still being added
            }
          }
          if (!ok) break;
          accumulator_drained(acc);
        }
        bias_next = next >= 0 && e_next >= 0 ? bias_of(e_next, t_next) : 0.f;
        t = t_next;
        entry = next;
        e = e_next;
      }
    }
    if (lane == 0) bulk_wait_all();   // staging buffers must outlive the stores that read them
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (CTAS == 2) cluster_sync_all();   // no CTA leaves while its peer may still signal its barriers or read its shared memory
  if (warp == 1) {
    if (*abort_flag) {  // error path: give copies / MMAs in flight a bounded moment to land
      for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    tc_fence_after();
    if (CTAS == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(C::kTmemCols) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(C::kTmemCols) : "memory");
  }
}

// Second pass of a split ESTMM: out = beta * out + sum over chunks (in chunk order) of the fp32 partial results, stored
// in the output's own type and layout.  One thread per four adjacent columns.
__global__ void __launch_bounds__(256)
estmm_reduce_kernel(const float* partial, int splits, int E, int64_t m, int64_t n, void* __restrict__ out, int64_t ldc,
                    int64_t c_estride, int64_t m_split, int64_t split_stride, int out_f32, int is_bf16, int beta) {
  wait_for_previous();
  const int64_t n4 = n / 4;
  const int64_t total = (int64_t)E * m * n4;
  const int64_t plane = (int64_t)E * m * n;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c4 = i % n4, row = i / n4;          // row = e * m + mrow
    const int64_t e = row / m, mrow = row - e * m;
    const float* src = partial + row * n + c4 * 4;
    float4 acc = *reinterpret_cast<const float4*>(src);
#pragma unroll 4
    for (int s = 1; s < splits; ++s) {
      const float4 v = *reinterpret_cast<const float4*>(src + (int64_t)s * plane);
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    const int64_t off = (mrow / m_split) * split_stride + e * c_estride + (mrow % m_split) * ldc + c4 * 4;
    if (out_f32) {
      float* o = reinterpret_cast<float*>(out) + off;
      if (beta) { const float4 old = *reinterpret_cast<float4*>(o); acc.x += old.x; acc.y += old.y; acc.z += old.z; acc.w += old.w; }
      *reinterpret_cast<float4*>(o) = acc;
    } else {
      uint16_t* o = reinterpret_cast<uint16_t*>(out) + off;
      if (beta) {
        const uint2 old = *reinterpret_cast<uint2*>(o);
        acc.x += unpack_lo(old.x, is_bf16); acc.y += unpack_hi(old.x, is_bf16);
        acc.z += unpack_lo(old.y, is_bf16); acc.w += unpack_hi(old.y, is_bf16);
      }
      *reinterpret_cast<uint2*>(o) = make_uint2(pack2(acc.x, acc.y, is_bf16), pack2(acc.z, acc.w, is_bf16));
    }
  }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
// rank-2 or rank-3 map over 16-bit elements, 128-byte swizzle unless told otherwise, zero fill out of bounds
int make_map(CUtensorMap* tm, const void* base, int is_bf16, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
             const uint32_t* box, CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
  return encode_tensor_map(tm, base, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, rank, dims,
                           strides_bytes, box, swizzle);
}

template <int BN, int MODE, int CTAS, int OUT>
int launch(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC, const CUtensorMap& tmX, const Params& p,
              int64_t max_tiles, cudaStream_t stream) {
  using C = Cfg<BN, CTAS, MODE, OUT>;
  static bool attr_set[64] = {false};
  static int max_clusters[64] = {0};
  auto kernel = gemm_tc_kernel<BN, MODE, CTAS, OUT>;
  int dev = 0;
  HEXA_CUDA(cudaGetDevice(&dev));
  HEXA_REQUIRE(dev >= 0 && dev < 64, "device ordinal %d out of range", dev);
  if (!attr_set[dev]) {
    HEXA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::kSmemBytes));
    attr_set[dev] = true;
  }
  if (max_tiles <= 0) return HEXA_OK;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(C::kThreads);
  cfg.dynamicSmemBytes = C::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // see after_previous
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  if (CTAS == 2) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
    if (max_clusters[dev] == 0) {   // how many CTA pairs the device can hold at once (one CTA per SM)
      cfg.gridDim = dim3(2 * (unsigned)(sm_count() / 2));
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) { (void)cudaGetLastError(); n = sm_count() / 2; }
      max_clusters[dev] = n;
    }
    int64_t pairs = max_tiles < max_clusters[dev] ? max_tiles : max_clusters[dev];
    if (sm_limit() > 0 && pairs > sm_limit() / 2) pairs = sm_limit() / 2;
    cfg.gridDim = dim3((unsigned)(2 * (pairs > 0 ? pairs : 1)));
  } else {
    int64_t ctas = max_tiles < sm_count() ? max_tiles : sm_count();
    if (sm_limit() > 0 && ctas > sm_limit()) ctas = sm_limit();
    cfg.gridDim = dim3((unsigned)ctas);
  }
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, tmA, tmB, tmC, tmX, p);
  if (e != cudaSuccess) {
    set_error("launch of gemm_tc_kernel<%d,%d,%d,%d> failed: %s", BN, MODE, CTAS, OUT, cudaGetErrorString(e));
    return HEXA_ERR_CUDA;
  }
  count_launch();
  return HEXA_OK;
}

int env_int(const char* name, int dflt) {
  const char* s = getenv(name);
  return s ? atoi(s) : dflt;
}

template <int BN, int MODE, int CTAS>
int launch_esmm(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC, const CUtensorMap& tmX, const Params& p,
                int64_t max_tiles, cudaStream_t stream) {
  if (p.epilogue == HEXA_EPI_ACT) return launch<BN, MODE, CTAS, OUT_ACT>(tmA, tmB, tmC, tmX, p, max_tiles, stream);
  if (p.epilogue == HEXA_EPI_DACT) return launch<BN, MODE, CTAS, OUT_DACT>(tmA, tmB, tmC, tmX, p, max_tiles, stream);
  return launch<BN, MODE, CTAS, OUT_LINEAR>(tmA, tmB, tmC, tmX, p, max_tiles, stream);
}
// HEXA_TC_CTAS=1 keeps every GEMM on single-CTA tiles (for A/B measurements); default: CTA pairs where they apply.
bool pairs_enabled() { static int v = -1; if (v < 0) v = env_int("HEXA_TC_CTAS", 2) == 1 ? 0 : 1; return v == 1; }

}  // namespace

namespace {
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &ptr, 12000, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
  }
  return fn;
}
}  // namespace

int encode_tensor_map(CUtensorMap* tm, const void* base, CUtensorMapDataType type, int rank, const uint64_t* dims,
                      const uint64_t* strides_bytes, const uint32_t* box, CUtensorMapSwizzle swizzle) {
  auto fn = encode_fn();
  if (!fn) { set_error("cuTensorMapEncodeTiled is not available from the driver"); return HEXA_ERR_CUDA; }
  cuuint64_t d[4]; cuuint64_t s[3]; cuuint32_t b[4]; cuuint32_t es[4] = {1, 1, 1, 1};
  for (int i = 0; i < rank; ++i) { d[i] = dims[i]; b[i] = box[i]; }
  for (int i = 0; i + 1 < rank; ++i) s[i] = strides_bytes[i];
  CUresult r = fn(tm, type, (cuuint32_t)rank, const_cast<void*>(base), d, s, b, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed with CUresult %d (rank %d dims %llu,%llu box %u,%u)", (int)r, rank,
              (unsigned long long)dims[0], (unsigned long long)dims[1], box[0], box[1]);
    return HEXA_ERR_CUDA;
  }
  return HEXA_OK;
}

bool esmm_tc_supported(const void* a, int64_t lda, const void* b, int64_t ldb, int64_t b_estride, const void* aux,
                       int64_t ldaux, const void* c, int64_t ldc, const float* bias, int64_t ldbias, int64_t n_out,
                       int dtype) {
  if (dtype != HEXA_F16 && dtype != HEXA_BF16) return false;
  if (!aligned16(a) || !aligned16(b) || !aligned16(c) || (aux && !aligned16(aux)) || (bias && !aligned16(bias))) return false;
  if (lda % 8 || ldb % 8 || b_estride % 8 || ldc % 8 || (aux && ldaux % 8) || (bias && ldbias % 4)) return false;
  // n_out itself may be any size (a rank's slice of an unevenly split hidden dimension): TMA stores clip at n_out and TMA
  // loads of the saved pre-activation fill with zeros.  Rows of aux and of an fp32 bias are asked for in whole 16-byte
  // chunks all the same: callers allocate them so (sorted_buffer, _f32), and what they get does not hang on the reads of
  // one version of the epilogue (its bias reads are scalar now, and a 16-bit bias needs no padding).
  const int64_t n8 = (n_out + 7) / 8 * 8, n4 = (n_out + 3) / 4 * 4;
  if ((aux && ldaux < n8) || (bias && ldbias < n4)) return false;
  return true;
}

// Whether an ESMM wider than 128 columns runs on single-CTA 128 x 128 tiles instead of CTA pairs' 256 x 256.  A pair tile takes
// two 128-row blocks of one expert: where experts have one block, or where there are fewer pair tiles than pairs, half of the SMs'
// work is for nothing, while the small tiles load an operand value twice as often.  Waves of either are estimated from static sizes
// (experts of up to 96 rows on average have one block, larger ones half a block or pair more than the rows fill), a wave of small
// tiles at 0.8 of a wave of pairs (measured 0.7 - 0.9; 0.6 with long rows of tiles, some of which
// one factor for all leaves with pairs although small tiles would be a little faster).  A launch of some experts has their share of the rows, and a cap on the SMs makes its
// waves.  Pairs / small tiles, us (fc1 + GELU, fc2):
//   300 rows x 1 [4096x1024] 15 24 / 11 23   16 x 32 [4096x1024] 34 29 / 31 26     700 x 7 [800x200] 14 13 / 9 9
//   1024 x 8 [3072x768] 21 20 / 17 19        2048 x 32 [4096x1024] 69 59 / 65 53   4096 x 64 [1024x256] 37 14 / 21 11
// and where the rule stays with pairs: 4608 x 32 [4096x1024] 79 65 / 103 86        4096 x 8 [3072x768] 34 22 / 39 34
//   18432 x 1 [2048x512] 58 32 / 69 46       4000 x 32 [4096x1024] 75 63 / 81 69   500 x 4 [4096x1024] (fc1) 20 / 19
// (128 x 256 tiles of one CTA were between the two at nearly all of these).
bool small_tiles(int E, int e_begin, int e_end, int64_t row_cap, int64_t n_out) {
  const int experts = (e_end < E ? e_end : E) - (e_begin > 0 ? e_begin : 0);
  if (experts <= 0) return false;
  const double all = (double)(row_cap > 127 * (int64_t)E ? row_cap - 127 * (int64_t)E : 1), rows = all * experts / E;
  const double met = rows < experts ? rows : experts, avg = all / E;
  const double blocks = met * (avg <= 96 ? 1.0 : avg / 128 + 0.5), pairs = met * (avg <= 128 ? 1.0 : avg / 256 + 0.5);
  const int sms = sm_limit() > 1 && sm_limit() < sm_count() ? sm_limit() : sm_count();
  const int64_t small_waves = ceil_div((int64_t)blocks * ceil_div(n_out, 128), sms);
  const int64_t pair_waves = ceil_div((int64_t)pairs * ceil_div(n_out, 256), sms / 2);
  return 0.8 * (double)small_waves < (double)pair_waves;
}

int esmm_tc_launch(const void* a, int64_t lda, const void* b, int b_layout, int64_t ldb, int64_t b_estride,
                   const void* bias, int64_t ldbias, void* aux, int64_t ldaux, void* c, int64_t ldc,
                   const int32_t* tile_expert, const int32_t* pad_offsets, const int32_t* row_token,
                   const int32_t* pair_block, int E, int64_t row_cap, int64_t n_out, int64_t k, int dtype, int epilogue,
                   int act, cudaStream_t stream, int e_begin, int e_end, int bias16, float* colsum) {
  if (row_cap == 0 || e_begin >= e_end) return HEXA_OK;
  const int is_bf16 = dtype == HEXA_BF16;
  const bool pairs = n_out > 128 && pair_block != nullptr && pairs_enabled() && !small_tiles(E, e_begin, e_end, row_cap, n_out);
  const int BN = pairs || (n_out > 128 && (pair_block == nullptr || !pairs_enabled())) ? 256 : 128;
  const int ctas = pairs ? 2 : 1;
  CUtensorMap tmA, tmB;
  {
    uint64_t dims[2] = {(uint64_t)k, (uint64_t)row_cap};
    uint64_t str[1] = {(uint64_t)lda * 2};
    uint32_t box[2] = {BLOCK_K, BLOCK_M};
    int rc = make_map(&tmA, a, is_bf16, 2, dims, str, box);
    if (rc) return rc;
  }
  if (b_layout == HEXA_B_NK) {
    uint64_t dims[3] = {(uint64_t)k, (uint64_t)n_out, (uint64_t)E};
    uint64_t str[2] = {(uint64_t)ldb * 2, (uint64_t)b_estride * 2};
    uint32_t box[3] = {BLOCK_K, (uint32_t)(BN / ctas), 1};   // each CTA of a pair loads half of the B rows
    int rc = make_map(&tmB, b, is_bf16, 3, dims, str, box);
    if (rc) return rc;
  } else {
    uint64_t dims[3] = {(uint64_t)n_out, (uint64_t)k, (uint64_t)E};
    uint64_t str[2] = {(uint64_t)ldb * 2, (uint64_t)b_estride * 2};
    uint32_t box[3] = {64, BLOCK_K, 1};
    int rc = make_map(&tmB, b, is_bf16, 3, dims, str, box);
    if (rc) return rc;
  }
  // output maps for the epilogue's TMA stores: [128 rows x 32 columns] boxes, 64-byte swizzle
  CUtensorMap tmC, tmX;
  {
    uint64_t dims[2] = {(uint64_t)n_out, (uint64_t)row_cap};
    uint32_t box[2] = {32, epilogue == HEXA_EPI_DACT ? (uint32_t)BLOCK_M : 32u};      // a group's rows, or a warp's
    uint64_t str[1] = {(uint64_t)ldc * 2};
    int rc = make_map(&tmC, c, is_bf16, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc) return rc;
    tmX = tmC;
    if (aux && epilogue != HEXA_EPI_LINEAR) {
      uint64_t strx[1] = {(uint64_t)ldaux * 2};
      rc = make_map(&tmX, aux, is_bf16, 2, dims, strx, box, CU_TENSOR_MAP_SWIZZLE_64B);
      if (rc) return rc;
    }
  }
  Params p{};
  p.tile_expert = tile_expert; p.pad_offsets = pad_offsets; p.row_token = row_token;
  p.pair_block = pair_block; p.max_pairs = row_cap / (2 * BLOCK_M) + E;
  p.bias = bias; p.ldbias = ldbias; p.bias16 = bias16; p.aux = aux; p.ldaux = ldaux; p.c = c; p.ldc = ldc;
  p.n = n_out; p.k = k; p.m = 0; p.E = E; p.e_begin = e_begin; p.e_end = e_end;
  p.epilogue = epilogue; p.act = act; p.is_bf16 = is_bf16; p.colsum = colsum;
  p.status = status_word(); p.debug = tc_debug_flags(); p.wait_limit_ns = wait_limit_ns(); p.next_may_start = sm_limit() == 0;
  const int64_t NT = ceil_div(n_out, BN);
  HEXA_REQUIRE((row_cap / BLOCK_M + E + 1) * NT < (int64_t)0x7fffffff, "hexa_esmm: too many output tiles for a 32-bit tile index");
  p.nt = (uint32_t)NT;
  if (ctas == 2) {
    const int64_t max_tiles = p.max_pairs * NT;
    return b_layout == HEXA_B_NK ? launch_esmm<256, ESMM_NK, 2>(tmA, tmB, tmC, tmX, p, max_tiles, stream)
                                 : launch_esmm<256, ESMM_KN, 2>(tmA, tmB, tmC, tmX, p, max_tiles, stream);
  }
  const int64_t max_tiles = (row_cap / BLOCK_M) * NT;
  if (b_layout == HEXA_B_NK)
    return BN == 256 ? launch_esmm<256, ESMM_NK, 1>(tmA, tmB, tmC, tmX, p, max_tiles, stream)
                     : launch_esmm<128, ESMM_NK, 1>(tmA, tmB, tmC, tmX, p, max_tiles, stream);
  return BN == 256 ? launch_esmm<256, ESMM_KN, 1>(tmA, tmB, tmC, tmX, p, max_tiles, stream)
                   : launch_esmm<128, ESMM_KN, 1>(tmA, tmB, tmC, tmX, p, max_tiles, stream);
}

bool estmm_tc_supported(const void* p, int64_t ldp, const void* q, int64_t ldq, const void* out, int64_t ldo,
                        int64_t o_estride, int64_t split_stride, int64_t n, int dtype, int out_dtype) {
  if (dtype != HEXA_F16 && dtype != HEXA_BF16) return false;
  if (out_dtype != HEXA_F32 && out_dtype != dtype) return false;
  if (!aligned16(p) || !aligned16(q) || !aligned16(out)) return false;
  const int ov = out_dtype == HEXA_F32 ? 4 : 8;
  if (ldp % 8 || ldq % 8 || ldo % ov || o_estride % ov || split_stride % ov || n % 8) return false;
  return true;
}

// How a split ESTMM is cut (chunks = 1: no split).  Only static sizes enter.  Few, long segments - the dense FFN's weight
// gradient (one "expert" owning every row), or a handful of experts with a small d x H - would leave most SMs idle behind a
// few serial k-loops, so where the output has fewer tiles than two per CTA pair (or CTA) every segment is cut into chunks, each a tile of its
// own.  Two things are chosen apart:
//   the length of a chain in the accumulator, which truncates: as many chains as make two tiles per CTA pair, of 8 k-blocks or more
//     of an average segment; chunks and chains are then both rounded up, so that a chain is never longer than that but may be
//     shorter ([5120 rows, 2048 x 512]: 4 chunks of 20 k-blocks, chains of 7; an expert far below the average: 1).  Relative error
//     of the fp32 result of [18432 rows, 2048 x 512] in 10 chains 1.9e-6, in 4 5.0e-6, in one 21e-6 (positive data 4.7 / 17 /
//     94e-6).  Between chains the sums are kept in fp32 registers;
//   the number of chunks, by time: full waves of a chunk's k-blocks at 0.29 us, 2 us to fill, drain and store a tile, and the
//     partial results, written and read once, at 5 TB/s (a drain between chains overlaps the next chain's MMAs and is not
//     counted).  At most as many as chains: the query asks for scratch of a chunk for each, and any that holds the chunks will do.
// One chunk per chain, partial results stored from registers / this, us: [18432 rows, 2048 x 512] 64 / 43, [65000, 256 x 1024]
// 61 / 45, [16384, 1024 x 256] x 8 35 / 24, [2000, 768 x 3072] 39 / 25; error of the first 1.9e-6 / 1.6e-6.
struct EstmmPlan { int chunks, chains, scratch; };      // chains per chunk, chunks the query asks scratch for
EstmmPlan estmm_tc_plan(int E, int64_t row_cap, int64_t m, int64_t n) {
  static int forced = -2;
  if (forced == -2) forced = env_int("HEXA_ESTMM_SPLITS", -1);       // A/B switch: 1 = never split
  if (n % 4) return {1, 1, 1};
  const int BN = n > 128 ? 256 : 128;
  const int ctas = (BN == 256 && m > BLOCK_M && pairs_enabled()) ? 2 : 1;
  const int64_t tiles = (int64_t)E * ceil_div(m, BLOCK_M * ctas) * ceil_div(n, BN);
  const int64_t slots = ctas == 2 ? sm_count() / 2 : sm_count();
  const int64_t avg_kb = row_cap / BLOCK_K / E;
  int64_t s = 1;
  if (tiles < 2 * slots) s = ceil_div(2 * slots, tiles);
  if (s > avg_kb / 8) s = avg_kb / 8;
  if (forced > 0) s = forced;
  if (s > 32) s = 32;
  if (s <= 1 || forced > 0) return {s < 1 ? 1 : (int)s, 1, s < 1 ? 1 : (int)s};
  const double plane_us = (double)E * (double)m * (double)n * 8.0 / 5e6;
  int best = 2;
  double best_us = 0.0;
  for (int c = 2; c <= s; ++c) {
    const double us = (double)ceil_div(tiles * c, slots) * ((double)ceil_div(avg_kb, c) * 0.29 + 2.0) + c * plane_us;
    if (c == 2 || us < best_us) { best = c; best_us = us; }
  }
  return {best, (int)ceil_div(s, best), (int)s};
}

size_t estmm_tc_workspace_bytes(int E, int64_t row_cap, int64_t m, int64_t n) {
  const int s = estmm_tc_plan(E, row_cap, m, n).scratch;
  return s > 1 ? (size_t)s * (size_t)E * (size_t)m * (size_t)n * sizeof(float) : 0;
}

int estmm_tc_launch(const void* pp, int64_t ldp, const void* q, int64_t ldq, const int32_t* pad_offsets, int E,
                    int64_t row_cap, int64_t m, int64_t n, void* out, int64_t ldo, int64_t o_estride, int64_t m_split,
                    int64_t split_stride, int dtype, int out_dtype, int beta, cudaStream_t stream, void* const* split_out,
                    int n_split, void* workspace, size_t workspace_bytes) {
  const int is_bf16 = dtype == HEXA_BF16;
  const int BN = n > 128 ? 256 : 128;
  const int ctas = (BN == 256 && m > BLOCK_M && pairs_enabled()) ? 2 : 1;
  const EstmmPlan plan = estmm_tc_plan(E, row_cap, m, n);
  int splits = n_split > 0 ? 1 : plan.chunks;
  if (splits > 1 && (!workspace || workspace_bytes < (size_t)splits * E * m * n * sizeof(float) || !aligned16(workspace)))
    splits = 1;      // without scratch the operator still runs, one tile per expert's whole segment
  CUtensorMap tmA, tmB;
  // the maps need at least one row even when no token was routed
  const uint64_t rows = row_cap > 0 ? (uint64_t)row_cap : 1;
  {
    uint64_t dims[2] = {(uint64_t)m, rows};
    uint64_t str[1] = {(uint64_t)ldp * 2};
    uint32_t box[2] = {64, BLOCK_K};
    int rc = make_map(&tmA, pp, is_bf16, 2, dims, str, box);
    if (rc) return rc;
  }
  {
    uint64_t dims[2] = {(uint64_t)n, rows};
    uint64_t str[1] = {(uint64_t)ldq * 2};
    uint32_t box[2] = {64, BLOCK_K};
    int rc = make_map(&tmB, q, is_bf16, 2, dims, str, box);
    if (rc) return rc;
  }
  Params p{};
  p.pad_offsets = pad_offsets; p.c = out; p.ldc = ldo; p.c_estride = o_estride; p.n = n; p.m = m; p.E = E;
  p.m_split = m_split; p.split_stride = split_stride;
  p.n_split = n_split;
  for (int i = 0; i < n_split && i < 16; ++i) p.c_split[i] = split_out[i];
  p.is_bf16 = is_bf16; p.out_f32 = out_dtype == HEXA_F32; p.beta = beta;
  p.splits = splits; p.chains = splits > 1 ? plan.chains : 1;
  p.status = status_word(); p.debug = tc_debug_flags(); p.wait_limit_ns = wait_limit_ns(); p.next_may_start = sm_limit() == 0;
  const int64_t max_tiles = (int64_t)E * ceil_div(m, BLOCK_M * ctas) * ceil_div(n, BN) * splits;
  HEXA_REQUIRE(max_tiles < (int64_t)0x7fffffff, "hexa_estmm: too many output tiles for a 32-bit tile index");
  p.nt = (uint32_t)ceil_div(n, BN);
  p.per_expert = (uint32_t)(ceil_div(m, BLOCK_M * ctas) * ceil_div(n, BN) * splits);
  p.total_tiles = (uint32_t)max_tiles;
  int rc;
  CUtensorMap tmC = tmA;      // a placeholder for register stores
  if (splits > 1) {
    const uint64_t dims[3] = {(uint64_t)n, (uint64_t)m, (uint64_t)splits * (uint64_t)E};
    const uint64_t str[2] = {(uint64_t)n * 4, (uint64_t)m * (uint64_t)n * 4};
    const uint32_t box[3] = {16, BLOCK_M, 1};
    rc = encode_tensor_map(&tmC, workspace, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc) return rc;
    if (ctas == 2) rc = launch<256, ESTMM, 2, OUT_PARTIAL>(tmA, tmB, tmC, tmA, p, max_tiles, stream);
    else rc = BN == 256 ? launch<256, ESTMM, 1, OUT_PARTIAL>(tmA, tmB, tmC, tmA, p, max_tiles, stream)
                        : launch<128, ESTMM, 1, OUT_PARTIAL>(tmA, tmB, tmC, tmA, p, max_tiles, stream);
    if (rc) return rc;
    const int64_t total = (int64_t)E * m * (n / 4);
    int64_t blocks = ceil_div(total, 256);
    if (blocks > (int64_t)sm_count() * 8) blocks = (int64_t)sm_count() * 8;
    after_previous(estmm_reduce_kernel, (unsigned)blocks, 256, 0, stream)(static_cast<const float*>(workspace), splits, E, m, n, out, ldo, o_estride,
                                                            p.m_split, p.split_stride, p.out_f32, is_bf16, beta);
    HEXA_LAUNCH_CHECK("estmm_reduce_kernel");
    return HEXA_OK;
  }
  if (n_split == 0 && m_split >= m && !beta && !p.out_f32) {
    uint64_t dims[3] = {(uint64_t)n, (uint64_t)m, (uint64_t)E};
    uint64_t str[2] = {(uint64_t)ldo * 2, (uint64_t)o_estride * 2};
    uint32_t box[3] = {32, BLOCK_M, 1};
    rc = make_map(&tmC, out, is_bf16, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc) return rc;
    if (ctas == 2) return launch<256, ESTMM, 2, OUT_STAGED>(tmA, tmB, tmC, tmA, p, max_tiles, stream);
    return BN == 256 ? launch<256, ESTMM, 1, OUT_STAGED>(tmA, tmB, tmC, tmA, p, max_tiles, stream)
                     : launch<128, ESTMM, 1, OUT_STAGED>(tmA, tmB, tmC, tmA, p, max_tiles, stream);
  }
  if (ctas == 2) return launch<256, ESTMM, 2, OUT_REGISTERS>(tmA, tmB, tmC, tmA, p, max_tiles, stream);
  return BN == 256 ? launch<256, ESTMM, 1, OUT_REGISTERS>(tmA, tmB, tmC, tmA, p, max_tiles, stream)
                   : launch<128, ESTMM, 1, OUT_REGISTERS>(tmA, tmB, tmC, tmA, p, max_tiles, stream);
}

}  // namespace hexa
