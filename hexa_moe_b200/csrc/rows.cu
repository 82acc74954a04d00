// HBM-bound row kernels on the sorted-row layout: gather, combine, pad-row masking and ESS.
//
// Bytes per unit (what the roofline of these kernels is computed from):
//   gather   reads cols*size per real row, writes cols*size per padded row, 4 B of row_token per row
//   combine  reads top_k*cols*size and writes cols*size per token, 4*top_k B of token_row
//   ESS      reads cols*size per padded row once; partials add 4*cols B per 128 rows (write + read).  The gather that
//            makes the rows can sum them on the way (hexa_gather_rows_ess): then only the partials are read.  [262144, 2048]
//            bf16 by token: gather 320 + both passes 168 us apart, 342 us together.
#include "hexa_common.cuh"

namespace hexa {
namespace {

// ---- gather: warp per sorted row, 16-byte vectors ---------------------------------------------
// Here and below, what a thread reads in several steps it requests before its first store: the loads are ordinary ones (see
// wait_for_previous), which the compiler leaves behind a store.
template <int VEC_BYTES>
__global__ void gather_rows_kernel(const uint8_t* src, int64_t src_ld_bytes,
                                   const int32_t* row_token, const int32_t* pad_offsets,
                                   int E, int64_t row_bytes, uint8_t* __restrict__ dst, int64_t dst_ld_bytes) {
  wait_for_previous();
  const int64_t n_pad = pad_offsets[E];
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n_pad) return;
  const int32_t tok = row_token[row];
  uint8_t* d = dst + row * dst_ld_bytes;
  if (VEC_BYTES == 16) {
    const int64_t n = row_bytes >> 4;
    if (tok >= 0) {
      const uint4* s = reinterpret_cast<const uint4*>(src + (int64_t)tok * src_ld_bytes);
      for (int64_t i = lane; i < n; i += 128) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (i + 32 * u < n) v[u] = s[i + 32 * u];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (i + 32 * u < n) reinterpret_cast<uint4*>(d)[i + 32 * u] = v[u];
      }
    } else {
      for (int64_t i = lane; i < n; i += 32) reinterpret_cast<uint4*>(d)[i] = make_uint4(0, 0, 0, 0);
    }
  } else {  // 2-byte granularity
    const int64_t n = row_bytes >> 1;
    const uint16_t* s = reinterpret_cast<const uint16_t*>(src + (int64_t)(tok >= 0 ? tok : 0) * src_ld_bytes);
    for (int64_t i = lane; i < n; i += 32) reinterpret_cast<uint16_t*>(d)[i] = tok >= 0 ? s[i] : (uint16_t)0;
  }
}

// ---- combine: warp per token, fp32 accumulation over the k routes in fixed order --------------
// K > 0: top_k known at compile time - the token's K row indices are read once, and the K row loads of a column
// chunk are issued together before anything is added (the adds keep the order j = 0..K-1, so the result does not
// depend on K being a template parameter).  K = 0: any top_k.
template <typename T, int K>
__global__ void combine_rows_kernel(const T* src, int64_t src_ld, const int32_t* token_row,
                                    int64_t num_tokens, int top_k, int64_t cols, T* __restrict__ dst, int64_t dst_ld) {
  wait_for_previous();
  constexpr int V = 16 / sizeof(T);
  const int lane = threadIdx.x & 31;
  const int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= num_tokens) return;
  const bool vec_ok = (cols % V == 0) && (src_ld % V == 0) && (dst_ld % V == 0);
  if (K > 0 && vec_ok) {
    const T* rows[K > 0 ? K : 1];
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const int32_t r = token_row[t * K + j];
      rows[j] = r >= 0 ? src + (int64_t)r * src_ld : nullptr;
    }
    using Raw = uint4[K > 0 ? K : 1];
    auto load = [&](int64_t c, Raw& raw) {
#pragma unroll
      for (int j = 0; j < K; ++j)
        raw[j] = rows[j] ? *reinterpret_cast<const uint4*>(rows[j] + c) : make_uint4(0, 0, 0, 0);
    };
    auto add = [&](int64_t c, const Raw& raw) {
      float acc[V];
#pragma unroll
      for (int i = 0; i < V; ++i) acc[i] = 0.f;
#pragma unroll
      for (int j = 0; j < K; ++j) {
        if (rows[j]) {      // an unrouted choice adds nothing (not even -0 + 0)
          const T* v = reinterpret_cast<const T*>(&raw[j]);
#pragma unroll
          for (int i = 0; i < V; ++i) acc[i] += to_f32<T>(v[i]);
        }
      }
      uint4 outv;
      T* o = reinterpret_cast<T*>(&outv);
#pragma unroll
      for (int i = 0; i < V; ++i) o[i] = from_f32<T>(acc[i]);
      *reinterpret_cast<uint4*>(dst + t * dst_ld + c) = outv;
    };
    int64_t c = (int64_t)lane * V;
    if (K <= 2) {      // two column chunks at a time; four rows of one are as many loads
      for (; c + 32 * V < cols; c += 64 * V) {
        Raw a, b;
        load(c, a);
        load(c + 32 * V, b);
        add(c, a);
        add(c + 32 * V, b);
      }
    }
    for (; c < cols; c += 32 * V) {
      Raw a;
      load(c, a);
      add(c, a);
    }
  } else if (vec_ok) {
    for (int64_t c = (int64_t)lane * V; c < cols; c += 32 * V) {
      float acc[V];
#pragma unroll
      for (int i = 0; i < V; ++i) acc[i] = 0.f;
      for (int j = 0; j < top_k; ++j) {
        const int32_t r = token_row[t * top_k + j];
        if (r < 0) continue;
        uint4 raw = *reinterpret_cast<const uint4*>(src + (int64_t)r * src_ld + c);
        const T* v = reinterpret_cast<const T*>(&raw);
#pragma unroll
        for (int i = 0; i < V; ++i) acc[i] += to_f32<T>(v[i]);
      }
      uint4 outv;
      T* o = reinterpret_cast<T*>(&outv);
#pragma unroll
      for (int i = 0; i < V; ++i) o[i] = from_f32<T>(acc[i]);
      *reinterpret_cast<uint4*>(dst + t * dst_ld + c) = outv;
    }
  } else {
    for (int64_t c = lane; c < cols; c += 32) {
      float acc = 0.f;
      for (int j = 0; j < top_k; ++j) {
        const int32_t r = token_row[t * top_k + j];
        if (r >= 0) acc += to_f32<T>(src[(int64_t)r * src_ld + c]);
      }
      dst[t * dst_ld + c] = from_f32<T>(acc);
    }
  }
}

template <typename T>
void combine_launch(const void* src, int64_t src_ld, const int32_t* token_row, int64_t T_, int top_k, int64_t cols, void* dst,
                    int64_t dst_ld, cudaStream_t stream) {
  const int warps = 8;
  const unsigned grid = (unsigned)ceil_div(T_, warps);
#define HEXA_COMBINE(K_)                                                                                              \
  after_previous(combine_rows_kernel<T, K_>, grid, warps * 32, 0, stream)((const T*)src, src_ld, token_row, T_, top_k, cols, (T*)dst, dst_ld)
  switch (top_k) {
    case 1: HEXA_COMBINE(1); break;
    case 2: HEXA_COMBINE(2); break;
    case 4: HEXA_COMBINE(4); break;
    default: HEXA_COMBINE(0); break;
  }
#undef HEXA_COMBINE
}

// ---- mask: zero the pad rows of a sorted buffer -------------------------------------------------
__global__ void mask_pad_rows_kernel(uint8_t* __restrict__ buf, int64_t ld_bytes, const int32_t* row_token,
                                     const int32_t* pad_offsets, int E, int64_t row_bytes) {
  wait_for_previous();
  const int64_t n_pad = pad_offsets[E];
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n_pad || row_token[row] >= 0) return;
  uint16_t* d = reinterpret_cast<uint16_t*>(buf + row * ld_bytes);
  for (int64_t i = lane; i < (row_bytes >> 1); i += 32) d[i] = 0;
}

// ---- ESS pass 1: column sums of one 128-row tile (one expert) ------------------------------------
// block = 32 column groups x 4 row groups; a thread sums 32 rows (r mod 4) of V adjacent columns, eight loads ahead of its stores, and
// the four sums are added in order.  The order is part of the result: a bias gradient is rounded to 16 bits from it.  Eight
// row groups of 16 rows, eight loads in flight, took 400 us with the gather at [262144, 2048] where this takes 342, and 110
// us where this takes 89 at [131072, 1024]; below a few thousand rows they were 1-4 us faster (a longer chain per thread).
// GATHER: the rows come from src[row_token[row]] (zeros for pad rows) and are written to dst as well.
constexpr int kEssCx = 32, kEssRy = 4;
template <typename T, bool GATHER>
__global__ void __launch_bounds__(kEssCx * kEssRy)
ess_partial_kernel(const T* src, int64_t src_ld, const int32_t* row_token,
                   const int32_t* pad_offsets, int E, int64_t cols, T* __restrict__ dst, int64_t dst_ld,
                   float* __restrict__ partial) {
  wait_for_previous();
  constexpr int V = 16 / sizeof(T);
  __shared__ float red[kEssRy][kEssCx * V];
  __shared__ int32_t tok_s[kRowTile];
  const int64_t n_pad = pad_offsets[E];
  const int64_t row0 = (int64_t)blockIdx.y * kRowTile;
  if (row0 >= n_pad) return;
  if (GATHER) {
    for (int i = threadIdx.x; i < kRowTile; i += kEssCx * kEssRy) tok_s[i] = row_token[row0 + i];
    __syncthreads();
  }
  const int cx = threadIdx.x & (kEssCx - 1), ry = threadIdx.x / kEssCx;
  const int64_t col = ((int64_t)blockIdx.x * kEssCx + cx) * V;
  float acc[V];
#pragma unroll
  for (int i = 0; i < V; ++i) acc[i] = 0.f;
  if (col < cols) {
    const bool vec_ok = GATHER || ((col + V <= cols) && (src_ld % V == 0));      // GATHER: checked by the host
    if (vec_ok) {
      constexpr int kRows = 8;      // at a time
#pragma unroll(GATHER ? 1 : kRowTile / (kRows * kEssRy))
      for (int r0 = ry; r0 < kRowTile; r0 += kRows * kEssRy) {
        uint4 raw[kRows];
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
          const int r = r0 + u * kEssRy;
          raw[u] = make_uint4(0, 0, 0, 0);
          if (GATHER) {
            const int32_t tok = tok_s[r];
            if (tok >= 0) raw[u] = *reinterpret_cast<const uint4*>(src + (int64_t)tok * src_ld + col);
          } else {
            raw[u] = *reinterpret_cast<const uint4*>(src + (row0 + r) * src_ld + col);
          }
        }
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
          if (GATHER) *reinterpret_cast<uint4*>(dst + (row0 + r0 + u * kEssRy) * dst_ld + col) = raw[u];
          const T* v = reinterpret_cast<const T*>(&raw[u]);
#pragma unroll
          for (int i = 0; i < V; ++i) acc[i] += to_f32<T>(v[i]);
        }
      }
    } else {
      for (int r = ry; r < kRowTile; r += kEssRy) {
        const T* p = src + (row0 + r) * src_ld + col;
#pragma unroll
        for (int i = 0; i < V; ++i)
          if (col + i < cols) acc[i] += to_f32<T>(p[i]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < V; ++i) red[ry][cx * V + i] = acc[i];
  __syncthreads();
  for (int c = threadIdx.x; c < kEssCx * V; c += kEssCx * kEssRy) {
    const int64_t gc = (int64_t)blockIdx.x * kEssCx * V + c;
    if (gc >= cols) continue;
    float s = red[0][c];
#pragma unroll
    for (int y = 1; y < kEssRy; ++y) s += red[y][c];
    partial[(int64_t)blockIdx.y * cols + gc] = s;
  }
}

// ---- ESS pass 2: per expert, add its tiles' partial rows in ascending order -----------------------
// 32 columns per block.  The additions of a column are one chain, whose order the results keep, so what is shared out is the
// reading: eight warps fetch 64 tiles' rows at a time into shared memory, the next 64 already under way while one warp adds.
// Experts of up to 8 tiles, a tile per warp, skip the pipeline.  (One thread per column that also loaded walked 144 tiles in
// 13 us; with the slices of the tiles summed apart, in another order, both passes of [18432, 2048] took 11.3 us, now 11.1.)
constexpr int kFinalTiles = 64;
template <typename TO>
__global__ void __launch_bounds__(256)
ess_final_kernel(const float* partial, const int32_t* pad_offsets,
                 int64_t cols, TO* __restrict__ out, int64_t ldo) {
  wait_for_previous();
  __shared__ float rows[kFinalTiles][32];
  const int e = blockIdx.y;
  const int cx = threadIdx.x & 31, slice = threadIdx.x >> 5;
  const int64_t c = (int64_t)blockIdx.x * 32 + cx;
  const int64_t t0 = pad_offsets[e] / kRowTile, t1 = pad_offsets[e + 1] / kRowTile;
  if (t1 - t0 <= 8) {      // a tile per warp
    rows[slice][cx] = c < cols && t0 + slice < t1 ? partial[(t0 + slice) * cols + c] : 0.f;
    __syncthreads();
    if (slice == 0 && c < cols) {
      float s = 0.f;
      for (int i = 0; i < (int)(t1 - t0); ++i) s += rows[i][cx];
      out[(int64_t)e * ldo + c] = from_f32<TO>(s);
    }
    return;
  }
  float next[kFinalTiles / 8];
  auto fetch = [&](int64_t base) {
#pragma unroll
    for (int i = 0; i < kFinalTiles / 8; ++i) {
      const int64_t t = base + slice + 8 * i;
      next[i] = c < cols && t < t1 ? partial[t * cols + c] : 0.f;
    }
  };
  fetch(t0);
  float s = 0.f;
  for (int64_t base = t0; base < t1; base += kFinalTiles) {      // uniform across the block
#pragma unroll
    for (int i = 0; i < kFinalTiles / 8; ++i) rows[slice + 8 * i][cx] = next[i];
    __syncthreads();
    if (base + kFinalTiles < t1) fetch(base + kFinalTiles);
    if (slice == 0) {
      const int n = (int)min((int64_t)kFinalTiles, t1 - base);
#pragma unroll 16
      for (int i = 0; i < n; ++i) s += rows[i][cx];
    }
    __syncthreads();
  }
  if (slice == 0 && c < cols) out[(int64_t)e * ldo + c] = from_f32<TO>(s);
}

}  // namespace
}  // namespace hexa

using namespace hexa;

extern "C" int hexa_gather_rows(const void* src, int64_t src_ld, const int32_t* row_token, const int32_t* pad_offsets,
                                int E, int64_t row_cap, int64_t cols, void* dst, int64_t dst_ld, int dtype,
                                void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  HEXA_REQUIRE(row_token && pad_offsets && dst, "hexa_gather_rows: null pointer");   // src may be null when there are no tokens
  HEXA_REQUIRE(E > 0 && row_cap >= 0 && cols > 0 && src_ld >= cols && dst_ld >= cols, "hexa_gather_rows: bad sizes");
  HEXA_REQUIRE(dtype == HEXA_F32 || dtype == HEXA_F16 || dtype == HEXA_BF16, "hexa_gather_rows: bad dtype %d", dtype);
  if (row_cap == 0) return HEXA_OK;
  const int64_t es = (int64_t)dtype_size(dtype);
  const int64_t row_bytes = cols * es, sld = src_ld * es, dld = dst_ld * es;
  const bool v16 = (row_bytes % 16 == 0) && (sld % 16 == 0) && (dld % 16 == 0) && aligned16(src) && aligned16(dst);
  const int warps = 8;
  const unsigned grid = (unsigned)ceil_div(row_cap, warps);
  if (v16)
    after_previous(gather_rows_kernel<16>, grid, warps * 32, 0, stream)((const uint8_t*)src, sld, row_token, pad_offsets, E, row_bytes,
                                                            (uint8_t*)dst, dld);
  else
    after_previous(gather_rows_kernel<2>, grid, warps * 32, 0, stream)((const uint8_t*)src, sld, row_token, pad_offsets, E, row_bytes,
                                                           (uint8_t*)dst, dld);
  HEXA_LAUNCH_CHECK("gather_rows");
  return HEXA_OK;
}

extern "C" int hexa_combine_rows(const void* src, int64_t src_ld, const int32_t* token_row, int64_t T, int top_k,
                                 int64_t cols, void* dst, int64_t dst_ld, int dtype, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  HEXA_REQUIRE(T >= 0 && top_k > 0 && cols > 0 && src_ld >= cols && dst_ld >= cols, "hexa_combine_rows: bad sizes");
  if (T == 0) return HEXA_OK;
  HEXA_REQUIRE(src && token_row && dst, "hexa_combine_rows: null pointer");
  HEXA_REQUIRE(aligned16(src) && aligned16(dst), "hexa_combine_rows: pointers must be 16-byte aligned");
  if (T == 0) return HEXA_OK;
  switch (dtype) {
    case HEXA_F32: combine_launch<float>(src, src_ld, token_row, T, top_k, cols, dst, dst_ld, stream); break;
    case HEXA_F16: combine_launch<__half>(src, src_ld, token_row, T, top_k, cols, dst, dst_ld, stream); break;
    case HEXA_BF16: combine_launch<__nv_bfloat16>(src, src_ld, token_row, T, top_k, cols, dst, dst_ld, stream); break;
    default: HEXA_REQUIRE(false, "hexa_combine_rows: bad dtype %d", dtype);
  }
  HEXA_LAUNCH_CHECK("combine_rows");
  return HEXA_OK;
}

extern "C" int hexa_mask_pad_rows(void* buf, int64_t ld, const int32_t* row_token, const int32_t* pad_offsets, int E,
                                  int64_t row_cap, int64_t cols, int dtype, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  HEXA_REQUIRE(buf && row_token && pad_offsets, "hexa_mask_pad_rows: null pointer");
  HEXA_REQUIRE(E > 0 && row_cap >= 0 && cols > 0 && ld >= cols, "hexa_mask_pad_rows: bad sizes");
  HEXA_REQUIRE(dtype == HEXA_F32 || dtype == HEXA_F16 || dtype == HEXA_BF16, "hexa_mask_pad_rows: bad dtype %d", dtype);
  if (row_cap == 0) return HEXA_OK;
  const int64_t es = (int64_t)dtype_size(dtype);
  const int warps = 8;
  after_previous(mask_pad_rows_kernel, (unsigned)ceil_div(row_cap, warps), warps * 32, 0, stream)((uint8_t*)buf, ld * es, row_token,
                                                                                     pad_offsets, E, cols * es);
  HEXA_LAUNCH_CHECK("mask_pad_rows");
  return HEXA_OK;
}

extern "C" size_t hexa_ess_workspace_bytes(int64_t row_cap, int64_t cols) {
  if (row_cap < 0 || cols <= 0) return 0;
  return (size_t)ceil_div(row_cap, kRowTile) * (size_t)cols * sizeof(float);
}

namespace hexa {
int ess_finish(const float* partial, const int32_t* pad_offsets, int E, int64_t cols, void* out, int64_t ldo, int out_dtype, cudaStream_t stream);
// Shared by hexa_ess and the entry points built on it: both passes on caller-provided scratch.
int ess_launch(const void* src, int64_t src_ld, const int32_t* pad_offsets, int E, int64_t row_cap, int64_t cols,
               void* out, int64_t ldo, int out_dtype, int dtype, float* partial, cudaStream_t stream) {
  const int64_t tiles = ceil_div(row_cap, kRowTile);
  if (tiles > 0) {
    const int V = 16 / (int)dtype_size(dtype);
    dim3 grid((unsigned)ceil_div(cols, kEssCx * V), (unsigned)tiles);
    HEXA_REQUIRE(tiles <= 65535, "hexa_ess: more than 65535 row tiles (row_capacity %lld)", (long long)row_cap);
#define HEXA_ESS(T)                                                                                                          \
  after_previous(ess_partial_kernel<T, false>, grid, kEssCx * kEssRy, 0, stream)((const T*)src, src_ld, nullptr, pad_offsets, E, cols, nullptr, 0, partial)
    switch (dtype) {
      case HEXA_F32: HEXA_ESS(float); break;
      case HEXA_F16: HEXA_ESS(__half); break;
      case HEXA_BF16: HEXA_ESS(__nv_bfloat16); break;
      default: HEXA_REQUIRE(false, "hexa_ess: bad dtype %d", dtype);
    }
#undef HEXA_ESS
    HEXA_LAUNCH_CHECK("ess_partial");
  }
  return ess_finish(partial, pad_offsets, E, cols, out, ldo, out_dtype, stream);
}

int ess_finish(const float* partial, const int32_t* pad_offsets, int E, int64_t cols, void* out, int64_t ldo, int out_dtype,
               cudaStream_t stream) {
  dim3 grid2((unsigned)ceil_div(cols, 32), (unsigned)E);
  if (out_dtype == HEXA_F16) after_previous(ess_final_kernel<__half>, grid2, 256, 0, stream)(partial, pad_offsets, cols, (__half*)out, ldo);
  else if (out_dtype == HEXA_BF16) after_previous(ess_final_kernel<__nv_bfloat16>, grid2, 256, 0, stream)(partial, pad_offsets, cols, (__nv_bfloat16*)out, ldo);
  else after_previous(ess_final_kernel<float>, grid2, 256, 0, stream)(partial, pad_offsets, cols, (float*)out, ldo);
  HEXA_LAUNCH_CHECK("ess_final");
  return HEXA_OK;
}
}  // namespace hexa

extern "C" int hexa_gather_rows_ess(const void* src, int64_t src_ld, const int32_t* row_token, const int32_t* pad_offsets,
                                    int E, int64_t row_cap, int64_t cols, void* dst, int64_t dst_ld, float* sums,
                                    int64_t ld_sums, int dtype, void* workspace, size_t workspace_bytes, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  HEXA_REQUIRE(row_token && pad_offsets && dst && sums && workspace, "hexa_gather_rows_ess: null pointer");
  HEXA_REQUIRE(E > 0 && E <= 65535 && row_cap >= 0 && cols > 0 && src_ld >= cols && dst_ld >= cols && ld_sums >= cols,
               "hexa_gather_rows_ess: bad sizes");
  int flags;
  const bool dtype_ok = take_flags(dtype, HEXA_SUMS_16, flags);
  HEXA_REQUIRE(dtype_ok && (dtype == HEXA_F32 || dtype == HEXA_F16 || dtype == HEXA_BF16), "hexa_gather_rows_ess: bad dtype %d", dtype);
  const int out_dtype = flags ? dtype : HEXA_F32;
  HEXA_REQUIRE(aligned16(dst), "hexa_gather_rows_ess: dst must be 16-byte aligned");
  const size_t need = hexa_ess_workspace_bytes(row_cap, cols);
  if (workspace_bytes < need) {
    set_error("hexa_gather_rows_ess: workspace %zu bytes < required %zu", workspace_bytes, need);
    return HEXA_ERR_WORKSPACE;
  }
  const int64_t tiles = ceil_div(row_cap, kRowTile), V = 16 / (int64_t)dtype_size(dtype);
  // one pass where every row is whole 16-byte groups on both sides; otherwise the two operators one after the other
  const bool one = tiles > 0 && row_cap % kRowTile == 0 && tiles <= 65535 && cols % V == 0 && src_ld % V == 0 && dst_ld % V == 0 &&
                   aligned16(src);
  if (!one) {
    const int rc = hexa_gather_rows(src, src_ld, row_token, pad_offsets, E, row_cap, cols, dst, dst_ld, dtype, stream_);
    if (rc != HEXA_OK) return rc;
    return ess_launch(dst, dst_ld, pad_offsets, E, row_cap, cols, sums, ld_sums, out_dtype, dtype, (float*)workspace, stream);
  }
  dim3 grid((unsigned)ceil_div(cols, kEssCx * V), (unsigned)tiles);
#define HEXA_GATHER_ESS(T)                                                                                                   \
  after_previous(ess_partial_kernel<T, true>, grid, kEssCx * kEssRy, 0, stream)((const T*)src, src_ld, row_token, pad_offsets, E, cols, (T*)dst, \
                                                                    dst_ld, (float*)workspace)
  if (dtype == HEXA_F32) HEXA_GATHER_ESS(float);
  else if (dtype == HEXA_F16) HEXA_GATHER_ESS(__half);
  else HEXA_GATHER_ESS(__nv_bfloat16);
#undef HEXA_GATHER_ESS
  HEXA_LAUNCH_CHECK("gather_rows_ess");
  return ess_finish((const float*)workspace, pad_offsets, E, cols, sums, ld_sums, out_dtype, stream);
}

extern "C" int hexa_ess(const void* src, int64_t src_ld, const int32_t* pad_offsets, int E, int64_t row_cap,
                        int64_t cols, float* out, int64_t ldo, int dtype, void* workspace, size_t workspace_bytes,
                        void* stream_) {
  HEXA_REQUIRE(src && pad_offsets && out && workspace, "hexa_ess: null pointer");
  int flags;
  HEXA_REQUIRE(take_flags(dtype, HEXA_SUMS_16, flags), "hexa_ess: bad dtype %d", dtype);
  HEXA_REQUIRE(E > 0 && E <= 65535 && row_cap >= 0 && cols > 0 && src_ld >= cols && ldo >= cols, "hexa_ess: bad sizes");
  HEXA_REQUIRE(aligned16(src), "hexa_ess: src must be 16-byte aligned");
  const size_t need = hexa_ess_workspace_bytes(row_cap, cols);
  if (workspace_bytes < need) {
    set_error("hexa_ess: workspace %zu bytes < required %zu", workspace_bytes, need);
    return HEXA_ERR_WORKSPACE;
  }
  return ess_launch(src, src_ld, pad_offsets, E, row_cap, cols, out, ldo, flags ? dtype : HEXA_F32, dtype, (float*)workspace, (cudaStream_t)stream_);
}

// ---- ESS on library-owned scratch -------------------------------------------------------------------
// Pass 1 of ESS needs one fp32 partial row per 128 sorted rows.  hexa_ess takes that scratch from the
// caller; this variant keeps it in a fixed array inside the library instead, for callers that have no
// way to obtain device memory at the point of the call.
namespace hexa {
constexpr size_t kEssStaticFloats = (size_t)8 << 20;   // 8 Mi floats = 32 MiB, resident on every device that loads the library
static __device__ __align__(256) float g_ess_static_scratch[kEssStaticFloats];
}  // namespace hexa

extern "C" size_t hexa_ess_static_capacity_bytes(void) { return hexa::kEssStaticFloats * sizeof(float); }

extern "C" int hexa_ess_static(const void* src, int64_t src_ld, const int32_t* pad_offsets, int E, int64_t row_cap,
                               int64_t cols, float* out, int64_t ldo, int dtype, void* stream_) {
  HEXA_REQUIRE(src && pad_offsets && out, "hexa_ess_static: null pointer");
  HEXA_REQUIRE(E > 0 && E <= 65535 && row_cap >= 0 && cols > 0 && src_ld >= cols && ldo >= cols, "hexa_ess_static: bad sizes");
  HEXA_REQUIRE(aligned16(src), "hexa_ess_static: src must be 16-byte aligned");
  const size_t need = hexa_ess_workspace_bytes(row_cap, cols);
  if (need > kEssStaticFloats * sizeof(float)) {
    set_error("hexa_ess_static: needs %zu bytes of scratch (row_capacity/128 * cols floats) but the built-in buffer holds %zu; "
              "use hexa_ess with caller-provided workspace for this size",
              need, kEssStaticFloats * sizeof(float));
    return HEXA_ERR_WORKSPACE;
  }
  // The array's name is only a host-side handle; the kernels need its address on the current device.
  // Looked up once per device, with that device current (first call on a device: do it before any stream capture).
  static float* dev_addr[64] = {nullptr};
  int dev = 0;
  HEXA_CUDA(cudaGetDevice(&dev));
  HEXA_REQUIRE(dev >= 0 && dev < 64, "hexa_ess_static: device ordinal %d out of range", dev);
  float* scratch = __atomic_load_n(&dev_addr[dev], __ATOMIC_ACQUIRE);
  if (!scratch) {
    HEXA_CUDA(cudaGetSymbolAddress((void**)&scratch, g_ess_static_scratch));
    __atomic_store_n(&dev_addr[dev], scratch, __ATOMIC_RELEASE);
  }
  // Nothing in the scratch has to start at zero: pass 1 overwrites every partial row that pass 2 reads.
  return ess_launch(src, src_ld, pad_offsets, E, row_cap, cols, out, ldo, HEXA_F32, dtype, scratch, (cudaStream_t)stream_);
}
