// CUDA-core (FFMA) ESMM and ESTMM on the sorted-row layout, fp32 accumulation.
// These are the kernels for fp32 data (where a 16-bit tensor-core pass cannot meet a 1e-5
// tolerance) and for shapes the tcgen05 kernels do not take (leading dimensions that are not
// multiples of 16 bytes).
//
// Bound: the FP32 pipe (128 FMA/clk/SM).  A TILE x TILE output tile per block of 256 threads, 16-deep k steps in two
// shared-memory buffers: the global loads of step s+1 are issued before the FMAs of step s and stored after them, one
// barrier per step.  Both operands sit k-major in shared memory ([k][row]), so a thread's operands are 16-byte reads and
// its (TILE/16)^2 accumulators are updated as column pairs by fma.rn.f32x2 (half the issue slots of FFMA, the same
// rounding).  Every output is still one chain of FMAs in ascending k.
//   TILE = 128  8x8 accumulators per thread: 64 FMAs for 64 bytes of shared-memory reads
//   TILE = 64   4x4: a quarter of the tile, for outputs with too few 128-tiles to fill the device (see use_large_tile)
#include "gemm_launch.h"
#include "hexa_common.cuh"

namespace hexa {
namespace {

constexpr int BK = 16;
constexpr int kThreads = 256;

__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack_f32x2(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void fma_f32x2(uint64_t& d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// One operand's TILE x BK slab, four consecutive elements of global memory per load.  KMAJOR: the source's rows run along
// k (src[row * ld + k]), otherwise along the tile's own dimension (src[k * ld + row]).  VEC: fp32 with 16-byte aligned
// rows whose length is a multiple of four, so every group of four is wholly inside or outside.
template <typename T, int TILE, bool KMAJOR, bool VEC> struct Slab {
  static constexpr int kLoads = TILE * BK / 4 / kThreads;
  static constexpr int kPitch = TILE + 4;
  float4 reg[kLoads];

  __device__ __forceinline__ void load(const T* src, int64_t ld, int64_t row0, int64_t rows, int64_t k0, int64_t k_end) {
#pragma unroll
    for (int q = 0; q < kLoads; ++q) {
      const int idx = threadIdx.x + kThreads * q;
      const int64_t row = row0 + (KMAJOR ? idx / (BK / 4) : (idx % (TILE / 4)) * 4);
      const int64_t k = k0 + (KMAJOR ? (idx % (BK / 4)) * 4 : idx / (TILE / 4));
      const T* p = src + (KMAJOR ? row * ld + k : k * ld + row);
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (row < rows && k < k_end) {
        if (VEC) {
          const float4 w = *reinterpret_cast<const float4*>(p);
          v[0] = w.x; v[1] = w.y; v[2] = w.z; v[3] = w.w;
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if ((KMAJOR ? k + i < k_end : row + i < rows)) v[i] = to_f32<T>(p[i]);
        }
      }
      reg[q] = make_float4(v[0], v[1], v[2], v[3]);
    }
  }
  __device__ __forceinline__ void store(float* sm) const {
#pragma unroll
    for (int q = 0; q < kLoads; ++q) {
      const int idx = threadIdx.x + kThreads * q;
      if (KMAJOR) {
        const int row = idx / (BK / 4), k = (idx % (BK / 4)) * 4;
        sm[(k + 0) * kPitch + row] = reg[q].x;
        sm[(k + 1) * kPitch + row] = reg[q].y;
        sm[(k + 2) * kPitch + row] = reg[q].z;
        sm[(k + 3) * kPitch + row] = reg[q].w;
      } else {
        *reinterpret_cast<float4*>(sm + (idx / (TILE / 4)) * kPitch + (idx % (TILE / 4)) * 4) = reg[q];
      }
    }
  }
};

// Accumulators of one thread: QUADS x QUADS blocks of 4x4 outputs, 64 rows / columns apart.  Block (qi, qj), element (i, j)
// is output (qi * 64 + ty * 4 + i, qj * 64 + tx * 4 + j) of the tile; a warp covers 16 x 32 of every 64 x 64 quarter.
template <int TILE> struct Acc {
  static constexpr int kQuads = TILE / 64;
  uint64_t v[4 * kQuads][2 * kQuads];
  int tx, ty;
  __device__ __forceinline__ Acc() {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    tx = (lane & 7) + (warp & 1) * 8;
    ty = (lane >> 3) + (warp >> 1) * 4;
#pragma unroll
    for (int i = 0; i < 4 * kQuads; ++i)
#pragma unroll
      for (int j = 0; j < 2 * kQuads; ++j) v[i][j] = 0ull;
  }
  __device__ __forceinline__ void step(const float* a, const float* b) {
    constexpr int P = TILE + 4;
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float4 av[kQuads];
      ulonglong2 bv[kQuads];
#pragma unroll
      for (int q = 0; q < kQuads; ++q) {
        av[q] = *reinterpret_cast<const float4*>(a + k * P + q * 64 + ty * 4);
        bv[q] = *reinterpret_cast<const ulonglong2*>(b + k * P + q * 64 + tx * 4);
      }
#pragma unroll
      for (int qi = 0; qi < kQuads; ++qi) {
        const float ar[4] = {av[qi].x, av[qi].y, av[qi].z, av[qi].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint64_t aa = pack_f32x2(ar[i], ar[i]);
#pragma unroll
          for (int qj = 0; qj < kQuads; ++qj) {
            fma_f32x2(v[qi * 4 + i][qj * 2], aa, bv[qj].x);
            fma_f32x2(v[qi * 4 + i][qj * 2 + 1], aa, bv[qj].y);
          }
        }
      }
    }
  }
  __device__ __forceinline__ void row4(int qi, int i, int qj, float (&f)[4]) const {
    const float2 lo = unpack_f32x2(v[qi * 4 + i][qj * 2]), hi = unpack_f32x2(v[qi * 4 + i][qj * 2 + 1]);
    f[0] = lo.x; f[1] = lo.y; f[2] = hi.x; f[3] = hi.y;
  }
};

// The k loop shared by both operators: acc += A[k_begin .. k_end)^T-slabs of the two operands.
template <typename T, int TILE, bool A_KMAJOR, bool B_KMAJOR, bool VEC>
__device__ __forceinline__ void contract(Acc<TILE>& acc, const T* a, int64_t lda, int64_t a_row0, int64_t a_rows,
                                         const T* b, int64_t ldb, int64_t b_row0, int64_t b_rows, int64_t k_begin,
                                         int64_t k_end) {
  __shared__ __align__(16) float As[2][BK * (TILE + 4)];
  __shared__ __align__(16) float Bs[2][BK * (TILE + 4)];
  if (k_begin >= k_end) return;
  Slab<T, TILE, A_KMAJOR, VEC> sa;
  Slab<T, TILE, B_KMAJOR, VEC> sb;
  sa.load(a, lda, a_row0, a_rows, k_begin, k_end);
  sb.load(b, ldb, b_row0, b_rows, k_begin, k_end);
  sa.store(As[0]);
  sb.store(Bs[0]);
  __syncthreads();
  int buf = 0;
  for (int64_t k0 = k_begin; k0 < k_end; k0 += BK) {
    const bool more = k0 + BK < k_end;
    if (more) {
      sa.load(a, lda, a_row0, a_rows, k0 + BK, k_end);
      sb.load(b, ldb, b_row0, b_rows, k0 + BK, k_end);
    }
    acc.step(As[buf], Bs[buf]);
    if (more) {      // the other buffer was last read before the previous barrier
      sa.store(As[buf ^ 1]);
      sb.store(Bs[buf ^ 1]);
      __syncthreads();
      buf ^= 1;
    }
  }
}

// A launch with a condition does nothing unless that word is set.
__device__ __forceinline__ bool wanted(const int32_t* only_if) { return only_if == nullptr || *only_if != 0; }

template <typename T, int TILE, bool B_NK, bool VEC>
__global__ void __launch_bounds__(kThreads, TILE == 128 ? 2 : 4)
esmm_simt_kernel(const T* a, int64_t lda, const T* b, int64_t ldb,
                 int64_t b_estride, const void* bias, int64_t ldbias, T* __restrict__ aux, int64_t ldaux,
                 T* __restrict__ c, int64_t ldc, const int32_t* tile_expert,
                 const int32_t* pad_offsets, const int32_t* row_token, int E, int64_t n_out,
                 int64_t k, int epilogue, int act, int e_begin, int e_end, int bias16,
                 const int32_t* only_if) {
  wait_for_previous(false);
  if (!wanted(only_if)) return;
  const int64_t row0 = (int64_t)blockIdx.y * TILE;
  if (row0 >= pad_offsets[E]) return;
  const int e = tile_expert[row0 / kRowTile];
  if (e < e_begin || e >= e_end) return;      // also the -1 of tiles beyond the last segment
  const int64_t n0 = (int64_t)blockIdx.x * TILE;
  Acc<TILE> acc;
  contract<T, TILE, true, B_NK, VEC>(acc, a, lda, row0, row0 + TILE, b + (int64_t)e * b_estride, ldb, n0, n_out, 0, k);
#pragma unroll
  for (int qi = 0; qi < Acc<TILE>::kQuads; ++qi)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t r = row0 + qi * 64 + acc.ty * 4 + i;
      const bool live = row_token == nullptr || row_token[r] >= 0;
#pragma unroll
      for (int qj = 0; qj < Acc<TILE>::kQuads; ++qj) {
        const int64_t n = n0 + qj * 64 + acc.tx * 4;
        if (n >= n_out) continue;
        float f[4], y[4];
        acc.row4(qi, i, qj, f);
        T* cp = c + r * ldc + n;
        T* xp = aux + r * ldaux + n;
        float x[4] = {0.f, 0.f, 0.f, 0.f};
        if (epilogue == HEXA_EPI_DACT) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (VEC || n + j < n_out) x[j] = to_f32<T>(xp[j]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float v = f[j];
          if (bias && n + j < n_out) {
            const int64_t at = (int64_t)e * ldbias + n + j;
            v += bias16 ? to_f32<T>(static_cast<const T*>(bias)[at]) : static_cast<const float*>(bias)[at];
          }
          y[j] = live ? v : 0.f;
          if (epilogue == HEXA_EPI_ACT) v = act_apply(act, v);
          else if (epilogue == HEXA_EPI_DACT) v = v * act_grad(act, x[j]);
          f[j] = live ? v : 0.f;
        }
        if (VEC) {      // T is float
          if (epilogue == HEXA_EPI_ACT && aux) *reinterpret_cast<float4*>(xp) = make_float4(y[0], y[1], y[2], y[3]);
          *reinterpret_cast<float4*>(cp) = make_float4(f[0], f[1], f[2], f[3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (n + j >= n_out) continue;
            if (epilogue == HEXA_EPI_ACT && aux) xp[j] = from_f32<T>(y[j]);
            cp[j] = from_f32<T>(f[j]);
          }
        }
      }
    }
}

template <typename T, typename TO, int TILE, bool VEC>
__global__ void __launch_bounds__(kThreads, TILE == 128 ? 2 : 4)
estmm_simt_kernel(const T* p, int64_t ldp, const T* q, int64_t ldq,
                  const int32_t* pad_offsets, int64_t m, int64_t n, TO* __restrict__ out, int64_t ldo,
                  int64_t o_estride, int64_t m_split, int64_t split_stride, int beta, const int32_t* only_if) {
  wait_for_previous(false);
  if (!wanted(only_if)) return;
  const int e = blockIdx.z;
  const int64_t m0 = (int64_t)blockIdx.y * TILE, n0 = (int64_t)blockIdx.x * TILE;
  Acc<TILE> acc;
  contract<T, TILE, false, false, VEC>(acc, p, ldp, m0, m, q, ldq, n0, n, pad_offsets[e], pad_offsets[e + 1]);
  TO* oe = out + (int64_t)e * o_estride;
#pragma unroll
  for (int qi = 0; qi < Acc<TILE>::kQuads; ++qi)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t mm = m0 + qi * 64 + acc.ty * 4 + i;
      if (mm >= m) continue;
      TO* row = oe + (mm / m_split) * split_stride + (mm % m_split) * ldo;
#pragma unroll
      for (int qj = 0; qj < Acc<TILE>::kQuads; ++qj) {
        const int64_t nn = n0 + qj * 64 + acc.tx * 4;
        if (nn >= n) continue;
        float f[4];
        acc.row4(qi, i, qj, f);
        if (VEC) {      // T and TO are float
          float4* dst = reinterpret_cast<float4*>(row + nn);
          float4 w = make_float4(f[0], f[1], f[2], f[3]);
          if (beta) { const float4 o = *dst; w.x += o.x; w.y += o.y; w.z += o.z; w.w += o.w; }
          *dst = w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (nn + j >= n) continue;
            float v = f[j];
            if (beta) v += to_f32<TO>(row[nn + j]);
            row[nn + j] = from_f32<TO>(v);
          }
        }
      }
    }
}

// 128-tiles do 64 FMAs per 64 bytes of shared-memory reads against 16 per 32 bytes, but two of their blocks fill an SM:
// with fewer of them than the device holds at once, four times as many 64-tiles keep more of it busy.
bool use_large_tile(int64_t tiles128) { return tiles128 >= 2 * (int64_t)sm_count(); }

}  // namespace

int esmm_simt_launch(const void* a, int64_t lda, const void* b, int b_layout, int64_t ldb, int64_t b_estride,
                     const void* bias, int64_t ldbias, void* aux, int64_t ldaux, void* c, int64_t ldc,
                     const int32_t* tile_expert, const int32_t* pad_offsets, const int32_t* row_token, int E,
                     int64_t row_cap, int64_t n_out, int64_t k, int dtype, int epilogue, int act, cudaStream_t stream,
                     int e_begin, int e_end, int bias16, const int32_t* only_if) {
  if (row_cap == 0 || e_begin >= e_end) return HEXA_OK;
  if (e_begin < 0) e_begin = 0;
  HEXA_REQUIRE(row_cap / 64 <= 65535, "hexa_esmm (simt): row_capacity %lld too large", (long long)row_cap);
  const bool nk = b_layout == HEXA_B_NK;
  const bool vec = dtype == HEXA_F32 && aligned16(a) && aligned16(b) && aligned16(c) && (!aux || (aligned16(aux) && ldaux % 4 == 0)) &&
                   lda % 4 == 0 && ldb % 4 == 0 && b_estride % 4 == 0 && ldc % 4 == 0 && k % 4 == 0 && n_out % 4 == 0;
  const bool large = use_large_tile(ceil_div(n_out, 128) * (row_cap / 128));
  const int tile = large ? 128 : 64;
  dim3 grid((unsigned)ceil_div(n_out, tile), (unsigned)(row_cap / tile));
#define HEXA_ESMM_SIMT(T, TILE, NK, VEC)                                                                               \
  after_previous(esmm_simt_kernel<T, TILE, NK, VEC>, grid, kThreads, 0, stream, only_if != nullptr)((const T*)a, lda, (const T*)b, ldb, b_estride, bias, \
                                                                    ldbias, (T*)aux, ldaux, (T*)c, ldc, tile_expert,   \
                                                                    pad_offsets, row_token, E, n_out, k, epilogue, act, \
                                                                    e_begin, e_end, bias16, only_if)
#define HEXA_ESMM_SIMT_T(T, VEC)                              \
  do {                                                        \
    if (large && nk) HEXA_ESMM_SIMT(T, 128, true, VEC);       \
    else if (large) HEXA_ESMM_SIMT(T, 128, false, VEC);       \
    else if (nk) HEXA_ESMM_SIMT(T, 64, true, VEC);            \
    else HEXA_ESMM_SIMT(T, 64, false, VEC);                   \
  } while (0)
  switch (dtype) {
    case HEXA_F32:
      if (vec) HEXA_ESMM_SIMT_T(float, true);
      else HEXA_ESMM_SIMT_T(float, false);
      break;
    case HEXA_F16: HEXA_ESMM_SIMT_T(__half, false); break;
    case HEXA_BF16: HEXA_ESMM_SIMT_T(__nv_bfloat16, false); break;
    default: HEXA_REQUIRE(false, "hexa_esmm: bad dtype %d", dtype);
  }
#undef HEXA_ESMM_SIMT_T
#undef HEXA_ESMM_SIMT
  HEXA_LAUNCH_CHECK("esmm_simt");
  return HEXA_OK;
}

int estmm_simt_launch(const void* p, int64_t ldp, const void* q, int64_t ldq, const int32_t* pad_offsets, int E,
                      int64_t m, int64_t n, void* out, int64_t ldo, int64_t o_estride, int64_t m_split, int64_t split_stride,
                      int dtype, int out_dtype, int beta, cudaStream_t stream, const int32_t* only_if) {
  HEXA_REQUIRE(ceil_div(m, 64) <= 65535 && E <= 65535, "hexa_estmm (simt): grid too large");
  const bool vec = dtype == HEXA_F32 && aligned16(p) && aligned16(q) && aligned16(out) && ldp % 4 == 0 && ldq % 4 == 0 && ldo % 4 == 0 &&
                   o_estride % 4 == 0 && split_stride % 4 == 0 && m % 4 == 0 && n % 4 == 0;
  const bool large = use_large_tile((int64_t)E * ceil_div(m, 128) * ceil_div(n, 128));
  const int tile = large ? 128 : 64;
  dim3 grid((unsigned)ceil_div(n, tile), (unsigned)ceil_div(m, tile), (unsigned)E);
#define HEXA_ESTMM_SIMT_V(T, TO, TILE, VEC)                                                                             \
  after_previous(estmm_simt_kernel<T, TO, TILE, VEC>, grid, kThreads, 0, stream, only_if != nullptr)((const T*)p, ldp, (const T*)q, ldq, pad_offsets, m, n, \
                                                                     (TO*)out, ldo, o_estride, m_split, split_stride, beta, only_if)
#define HEXA_ESTMM_SIMT(T, TO, VEC)                    \
  do {                                                 \
    if (large) HEXA_ESTMM_SIMT_V(T, TO, 128, VEC);     \
    else HEXA_ESTMM_SIMT_V(T, TO, 64, VEC);            \
  } while (0)
  if (dtype == HEXA_F32 && out_dtype == HEXA_F32) {
    if (vec) HEXA_ESTMM_SIMT(float, float, true);
    else HEXA_ESTMM_SIMT(float, float, false);
  }
  else if (dtype == HEXA_F16 && out_dtype == HEXA_F32) HEXA_ESTMM_SIMT(__half, float, false);
  else if (dtype == HEXA_F16 && out_dtype == HEXA_F16) HEXA_ESTMM_SIMT(__half, __half, false);
  else if (dtype == HEXA_BF16 && out_dtype == HEXA_F32) HEXA_ESTMM_SIMT(__nv_bfloat16, float, false);
  else if (dtype == HEXA_BF16 && out_dtype == HEXA_BF16) HEXA_ESTMM_SIMT(__nv_bfloat16, __nv_bfloat16, false);
  else HEXA_REQUIRE(false, "hexa_estmm: unsupported dtype pair %d -> %d", dtype, out_dtype);
#undef HEXA_ESTMM_SIMT
#undef HEXA_ESTMM_SIMT_V
  HEXA_LAUNCH_CHECK("estmm_simt");
  return HEXA_OK;
}

}  // namespace hexa
