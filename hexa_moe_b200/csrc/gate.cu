// The step right before routing, as one kernel each way: softmax over the gate logits, top-k expert ids written in
// the route-major int32 layout the routing kernel reads, and the GShard auxiliary loss
//     l = (1/T) sum_e mass_e * ce_e,   mass_e = sum_t softmax(logits)[t,e],   ce_e = (E/T) #{t : top-1(t) = e}
// (reference hexa_moe/impls/cascaded_moe.py:568-598, impls/layers.py:480-489, impls/losses.py:12-19), plus the
// gradient of l with respect to the logits.  The [T,E] score matrix is never written: the backward kernel
// recomputes the softmax from the logits it has to read anyway.
//
// GShard kernels: a group of G lanes (8 up to 64 experts, 16 up to 128, else 32) per token, lane g holding columns
// g, g + G, ...: a warp works on 32 / G tokens at once and a reduction over a token is log2(G) shuffles; the next token's
// row is loaded while this one is worked on.  Sums over a token are added in the order of a 32-lane xor tree over columns
// modulo 32 whatever G is.  Column sums stay in registers across the tokens of a group, meet in shared memory once per
// block and leave the block as one partial row (and one row of top-1 counts) in the workspace; gate_finish_kernel adds the
// rows in a fixed order with all its threads.  A single block finishes by itself.  Nothing has to start at zero and every
// float sum has a fixed order: mass and loss are bit-identical from run to run.
// Bound: latency (a token is ~30 dependent shuffles) up to some 10^4 tokens, then the reading of the logits.
// [131072, 64] top-2: 102 us at first, then 26 + 10 with parallel partial rows, 21 + 5 with products for the quotients, a tree
// for each lane's maximum and a third of the partial rows; the gradient 23, 17, 15 us.
// Load-importance kernels: one warp per token; the block that finishes last adds the partial rows (in block order).
// Ties: the lowest expert id wins, and the k ids of a token come out in descending score order.  The selection is
// total: a score that is NaN ranks below every number, so a row of NaN / inf logits (an overflowed fp16 step) still
// yields k distinct ids in [0, E) - the lowest free columns - and only the loss carries the NaN, as it does through
// F.softmax -> torch.topk in the reference.
#include <float.h>

#include "hexa_common.cuh"

namespace hexa {
namespace {

constexpr int kGateThreads = 256;
constexpr int kGateWarps = kGateThreads / 32;
constexpr int kGateMaxExperts = 512;
constexpr int kGateMaxBlocks = 1024;   // partial rows of kGateMaxExperts 32-bit words the workspace holds
constexpr size_t kGateTicketBytes = 256;

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// softmax of one token's logits, spread over the warp; columns >= E come out as 0
template <int VPT>
__device__ __forceinline__ void warp_softmax(const float* row, int E, int lane, float (&s)[VPT]) {
  float m = -FLT_MAX;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = lane + 32 * i;
    s[i] = c < E ? row[c] : -FLT_MAX;
    m = fmaxf(m, s[i]);
  }
  m = warp_max(m);
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    s[i] = (lane + 32 * i) < E ? expf(s[i] - m) : 0.f;
    sum += s[i];
  }
  sum = warp_sum(sum);
#pragma unroll
  for (int i = 0; i < VPT; ++i) s[i] = s[i] / sum;
}

// ---- groups of G lanes per token, PER columns per lane ----------------------------------------------------------------
// Sum over a token's columns in the order of warp_sum over lanes c mod 32 (the columns of one such lane added first).
template <int G, int PER>
__device__ __forceinline__ float group_sum(const float (&v)[PER]) {
  constexpr int R = 32 / G;
  float cls[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    cls[r] = 0.f;
#pragma unroll
    for (int j = r; j < PER; j += R) cls[r] += v[j];
  }
#pragma unroll
  for (int o = R / 2; o > 0; o >>= 1)
#pragma unroll
    for (int r = 0; r < o; ++r) cls[r] += cls[r + o];
  float x = cls[0];
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

template <int G, int PER>
__device__ __forceinline__ void group_load(const float* row, int E, int g, bool valid, float (&v)[PER]) {
#pragma unroll
  for (int j = 0; j < PER; ++j) v[j] = (valid && g + G * j < E) ? row[g + G * j] : -FLT_MAX;
}

// s / sum for a token's exponentials (0 <= s <= 1 <= sum <= E, both NaN-free), bit for bit the IEEE quotient: one correctly
// rounded reciprocal per lane and Markstein's remainder correction per element (P. Markstein, Computation of elementary
// functions on the IBM RISC System/6000, 1990) are three instructions where a division is a dozen.  The remainder has to be exact, so a
// lane with a non-zero exponential below 2^-90, or with a sum that is no such number, takes the division.  Lanes of one token may
// go different ways: equal exponentials are equal scores all the same, and the lowest id wins, because both give the quotient.
template <int PER>
__device__ __forceinline__ void normalise(float sum, float (&s)[PER]) {
  uint32_t least = 0xffffffffu;
#pragma unroll
  for (int j = 0; j < PER; ++j) least = min(least, __float_as_uint(s[j]) - 1u);      // zero wraps to the top
  if (sum >= 1.f && sum <= 1024.f && least >= ((127u - 90u) << 23)) {
    const float r = __frcp_rn(sum);
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const float q = s[j] * r;
      s[j] = fmaf(fmaf(-q, sum, s[j]), r, q);
    }
  } else {
#pragma unroll
    for (int j = 0; j < PER; ++j) s[j] = s[j] / sum;
  }
}

// logits -> softmax in place; columns >= E come out as 0
template <int G, int PER>
__device__ __forceinline__ void group_softmax(int E, int g, float (&s)[PER]) {
  float m = -FLT_MAX;
#pragma unroll
  for (int j = 0; j < PER; ++j) m = fmaxf(m, s[j]);
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
#pragma unroll
  for (int j = 0; j < PER; ++j) s[j] = g + G * j < E ? expf(s[j] - m) : 0.f;
  normalise<PER>(group_sum<G, PER>(s), s);
}

__device__ __forceinline__ void fold_loss(float part, float* red, int64_t T, int E, float* __restrict__ loss) {
  // fixed-order block reduction: lanes by xor tree, warps in index order
  part = warp_sum(part);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tot = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
    loss[0] = tot * ((float)E / (float)T) / (float)T;
  }
}

// partial: per block E float column sums, then E int top-1 counts
template <int G, int PER, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
gate_topk_kernel(const float* logits, int64_t ld, int64_t T, int E, int k, int32_t* __restrict__ ids,
                 float* __restrict__ mass, int32_t* __restrict__ first_count, float* __restrict__ loss,
                 float* __restrict__ partial) {
  wait_for_previous();
  constexpr int kGroups = 32 / G;
  __shared__ float mass_w[WARPS][G * PER];
  __shared__ int cnt_s[G * PER];
  __shared__ float red_s[WARPS];
  for (int e = threadIdx.x; e < G * PER; e += blockDim.x) cnt_s[e] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane & (G - 1);
  const int64_t first = ((int64_t)blockIdx.x * WARPS + warp) * kGroups;     // this warp's first token of a sweep
  const int64_t step = (int64_t)gridDim.x * WARPS * kGroups;
  const int grp = lane / G;
  float acc[PER], next[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) acc[j] = 0.f;
  group_load<G, PER>(logits + (first + grp) * ld, E, g, first + grp < T, next);
  for (int64_t t0 = first; t0 < T; t0 += step) {      // uniform across the warp; groups past T carry no token
    const int64_t t = t0 + grp;
    const bool live = t < T;
    float s[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) s[j] = next[j];
    group_load<G, PER>(logits + (t + step) * ld, E, g, t + step < T, next);
    group_softmax<G, PER>(E, g, s);
    if (live) {
#pragma unroll
      for (int j = 0; j < PER; ++j) acc[j] += s[j];
    }
    // candidates: scores are not negative, so a column that is taken or does not exist counts as -1 and some lane always
    // has one at 0 or more while fewer than E are taken (k <= E is checked by the host); a NaN counts as 0: it makes the
    // whole row NaN, whose lowest columns are then taken
#pragma unroll
    for (int j = 0; j < PER; ++j) s[j] = g + G * j < E ? fmaxf(s[j], 0.f) : -1.f;      // fmaxf(NaN, 0) is 0
    for (int i = 0; i < k; ++i) {
      // this lane's maximum, neighbours first, so that the lower columns are always on the left; of equal scores they stay
      float v[PER];
      int at[PER];
#pragma unroll
      for (int j = 0; j < PER; ++j) { v[j] = s[j]; at[j] = j; }
#pragma unroll
      for (int w = 1; w < PER; w *= 2)
#pragma unroll
        for (int j = 0; j + w < PER; j += 2 * w)
          if (v[j + w] > v[j]) { v[j] = v[j + w]; at[j] = at[j + w]; }
      float best = v[0];
      int bi = g + G * at[0];
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
      }
      const bool valid = (unsigned)bi < (unsigned)E;     // always true; kept so that no index derived from data is trusted
#pragma unroll
      for (int j = 0; j < PER; ++j)
        if (bi == g + G * j) s[j] = -1.f;
      if (g == 0 && live) {
        ids[(int64_t)i * T + t] = valid ? bi : -1;         // -1 is a row the routing kernel skips
        if (i == 0 && valid) atomicAdd(&cnt_s[bi], 1);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < PER; ++j) {
#pragma unroll
    for (int o = G; o < 32; o <<= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
    if (grp == 0) mass_w[warp][g + G * j] = acc[j];
  }
  __syncthreads();
  const bool only = gridDim.x == 1;
  int32_t* counts = reinterpret_cast<int32_t*>(partial) + (int64_t)blockIdx.x * 2 * E + E;
  float part = 0.f;
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    float m = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) m += mass_w[w][e];
    if (only) {
      mass[e] = m;
      first_count[e] = cnt_s[e];
      part += m * (float)cnt_s[e];
    } else {
      partial[(int64_t)blockIdx.x * 2 * E + e] = m;
      counts[e] = cnt_s[e];
    }
  }
  if (only) fold_loss(part, red_s, T, E, loss);
}

// Adds the blocks' rows: 1024 / E threads per expert take every (1024 / E)-th block, their sums meet in index order.
constexpr int kFinishThreads = 1024;
__global__ void __launch_bounds__(kFinishThreads)
gate_finish_kernel(const float* partial, int blocks, int64_t T, int E, float* __restrict__ mass,
                   int32_t* __restrict__ first_count, float* __restrict__ loss) {
  wait_for_previous();
  __shared__ float m_s[kFinishThreads];
  __shared__ int c_s[kFinishThreads];
  __shared__ float red_s[kFinishThreads / 32];
  const int slices = kFinishThreads / E;
  const int e = threadIdx.x % E, slice = threadIdx.x / E;
  if (slice < slices) {
    float m = 0.f;
    int c = 0;
#pragma unroll 16
    for (int b = slice; b < blocks; b += slices) {      // in the order of b; 16 rows are on their way at a time
      const float* row = partial + (int64_t)b * 2 * E;
      m += row[e];
      c += reinterpret_cast<const int32_t*>(row)[E + e];
    }
    m_s[threadIdx.x] = m;
    c_s[threadIdx.x] = c;
  }
  __syncthreads();
  float part = 0.f;
  if (threadIdx.x < E) {
    float m = 0.f;
    int c = 0;
    for (int i = 0; i < slices; ++i) { m += m_s[i * E + threadIdx.x]; c += c_s[i * E + threadIdx.x]; }
    mass[threadIdx.x] = m;
    first_count[threadIdx.x] = c;
    part = m * (float)c;
  }
  fold_loss(part, red_s, T, E, loss);
}

// dlogits[t,e] = s[t,e] * (g_e - sum_e' s[t,e'] g_e') with g_e = dloss * ce_e / T: the chain rule through
// mass = column sums of the softmax (ce counts top-1 choices and carries no gradient)
template <int G, int PER>
__global__ void __launch_bounds__(kGateThreads)
gate_loss_grad_kernel(const float* logits, int64_t ld, int64_t T, int E, const int32_t* first_count,
                      const float* dloss, float* __restrict__ dlogits, int64_t ldd) {
  wait_for_previous();
  constexpr int kGroups = 32 / G;
  const int lane = threadIdx.x & 31, g = lane & (G - 1), grp = lane / G;
  const int64_t first = ((int64_t)blockIdx.x * kGateWarps + (threadIdx.x >> 5)) * kGroups;
  const int64_t step = (int64_t)gridDim.x * kGateWarps * kGroups;
  const float scale = *dloss * ((float)E / (float)T) / (float)T;
  float ge[PER], next[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int c = g + G * j;
    ge[j] = c < E ? scale * (float)first_count[c] : 0.f;
  }
  group_load<G, PER>(logits + (first + grp) * ld, E, g, first + grp < T, next);
  for (int64_t t0 = first; t0 < T; t0 += step) {
    const int64_t t = t0 + grp;
    float s[PER], sg[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) s[j] = next[j];
    group_load<G, PER>(logits + (t + step) * ld, E, g, t + step < T, next);
    group_softmax<G, PER>(E, g, s);
#pragma unroll
    for (int j = 0; j < PER; ++j) sg[j] = s[j] * ge[j];
    const float dot = group_sum<G, PER>(sg);
    if (t < T) {
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        const int c = g + G * j;
        if (c < E) dlogits[t * ldd + c] = s[j] * (ge[j] - dot);
      }
    }
  }
}

// ---- the gate projection's operands in 16-bit terms -----------------------------------------------------------------
// x = hi + mid + lo exactly to fp32's 24 bits, each term the bf16 rounding of what the previous ones left over.
__device__ __forceinline__ void split_terms(float x, __nv_bfloat16 (&t)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    t[i] = __float2bfloat16_rn(x);
    x -= __bfloat162float(t[i]);
  }
}

template <int V> struct Vec;
template <> struct Vec<4> { using F = float4; using H = uint2; };
template <> struct Vec<1> { using F = float; using H = uint16_t; };

// out[r, q * cols + c] = term `order[q]` of src[r, c], four blocks of columns per row: (hi, hi, mid, lo) or, with
// by_rows, four blocks of rows (lo, mid, hi, hi): src is then one row of rows * cols elements.
template <int V>
__global__ void __launch_bounds__(256)
split_terms_kernel(const float* src, int64_t ld, int64_t rows, int64_t cols, int lo_first, __nv_bfloat16* __restrict__ out) {
  wait_for_previous();
  const int64_t per_row = cols / V;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < rows * per_row; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / per_row, c = (i - r * per_row) * V;
    const typename Vec<V>::F x = *reinterpret_cast<const typename Vec<V>::F*>(src + r * ld + c);
    __align__(8) __nv_bfloat16 t[3][V];
#pragma unroll
    for (int j = 0; j < V; ++j) {
      __nv_bfloat16 one[3];
      split_terms(reinterpret_cast<const float*>(&x)[j], one);
#pragma unroll
      for (int q = 0; q < 3; ++q) t[q][j] = one[q];
    }
    __nv_bfloat16* o = out + r * 4 * cols + c;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int fwd = q == 0 ? 0 : q - 1, rev = q == 3 ? 0 : 2 - q;      // (hi, hi, mid, lo) / (lo, mid, hi, hi)
      const typename Vec<V>::H a = *reinterpret_cast<const typename Vec<V>::H*>(t[fwd]);
      const typename Vec<V>::H b = *reinterpret_cast<const typename Vec<V>::H*>(t[rev]);
      *reinterpret_cast<typename Vec<V>::H*>(o + q * cols) = lo_first ? b : a;
    }
  }
}

// out[r, c] = (hi + mid) + lo of a row's three blocks of columns, stored in that order or, with lo_first, reversed
template <int V>
__global__ void __launch_bounds__(256)
sum_terms_kernel(const float* part, int64_t rows, int64_t cols, int lo_first, float* __restrict__ out) {
  wait_for_previous();
  using F = typename Vec<V>::F;
  const int64_t per_row = cols / V;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < rows * per_row; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / per_row, c = (i - r * per_row) * V;
    const float* p = part + r * 3 * cols + c;
    const F a = *reinterpret_cast<const F*>(p + (lo_first ? 2 * cols : 0));
    const F b = *reinterpret_cast<const F*>(p + cols);
    const F d = *reinterpret_cast<const F*>(p + (lo_first ? 0 : 2 * cols));
    F o;
#pragma unroll
    for (int j = 0; j < V; ++j)
      reinterpret_cast<float*>(&o)[j] = (reinterpret_cast<const float*>(&a)[j] + reinterpret_cast<const float*>(&b)[j]) +
                                        reinterpret_cast<const float*>(&d)[j];
    *reinterpret_cast<F*>(out + r * cols + c) = o;
  }
}

// ---- the gate projection of few tokens, straight on the CUDA cores -----------------------------------------------------
// logits = x W^T with x [T, d], W fp32 [E, d] and fp32 FMAs: for small T the split operands' three launches (or, for fp16
// and fp32 tokens, an fp32 GEMM with too few blocks) cost more than the products.  A warp takes 4 tokens x 4 experts,
// its lanes 8 consecutive elements of every 256 of d, so an operand value loaded once meets four of the other side, and the 16
// sums meet in 16 shuffles.  Bound: the latency of d / 256 rounds of loads.  [2048, 768], 8 experts: 4 us (fp16 with a
// cast and a GEMM 22, bf16 in split terms 7 in three launches); [16, 1024], 32 experts: 4 us (split terms 7).
template <typename T>
__device__ __forceinline__ void load8(const T* p, bool live, float (&v)[8]) {
  uint4 raw = make_uint4(0, 0, 0, 0);
  if (live) raw = *reinterpret_cast<const uint4*>(p);
  const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = to_f32<T>(e[i]);
}

template <>
__device__ __forceinline__ void load8<float>(const float* p, bool live, float (&v)[8]) {
  float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
  if (live) { lo = *reinterpret_cast<const float4*>(p); hi = reinterpret_cast<const float4*>(p)[1]; }
  v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w; v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
}

template <typename T>
__global__ void __launch_bounds__(128)
gate_project_kernel(const T* x, int64_t ldx, const float* w, int64_t tokens, int E, int64_t d, float* __restrict__ logits) {
  wait_for_previous();
  const int lane = threadIdx.x & 31;
  const int64_t groups = (E + 3) / 4;
  const int64_t tile = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int64_t t0 = tile / groups * 4;
  const int e0 = (int)(tile % groups) * 4;
  if (t0 >= tokens) return;      // uniform across the warp
  float acc[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) acc[i] = 0.f;
  for (int64_t c = lane * 8; c < d; c += 256) {
    float xv[4][8];
#pragma unroll
    for (int a = 0; a < 4; ++a) load8<T>(x + (t0 + a) * ldx + c, t0 + a < tokens, xv[a]);
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
      if (e0 + b < E) {
        lo = *reinterpret_cast<const float4*>(w + (int64_t)(e0 + b) * d + c);
        hi = *reinterpret_cast<const float4*>(w + (int64_t)(e0 + b) * d + c + 4);
      }
      const float wv[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[a * 4 + b] = fmaf(xv[a][i], wv[i], acc[a * 4 + b]);
    }
  }
  // sums over the lanes, halving the values a lane is responsible for: lane l ends with value l / 2
#pragma unroll
  for (int o = 16; o >= 2; o >>= 1) {
    const bool upper = lane & o;
#pragma unroll
    for (int i = 0; i < o / 2; ++i) {
      const float mine = upper ? acc[i + o / 2] : acc[i], theirs = upper ? acc[i] : acc[i + o / 2];
      acc[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, o);
    }
  }
  const float sum = acc[0] + __shfl_xor_sync(0xffffffffu, acc[0], 1);
  const int v = lane >> 1;
  const int64_t t = t0 + (v >> 2);
  const int e = e0 + (v & 3);
  if ((lane & 1) == 0 && t < tokens && e < E) logits[t * E + e] = sum;
}

// dx = g W, [T, d]: a thread owns 8 columns of 4 tokens
template <typename T>
__global__ void __launch_bounds__(128)
gate_project_dx_kernel(const float* g, const float* w, int64_t tokens, int E, int64_t d, T* __restrict__ dx) {
  wait_for_previous();
  const int64_t chunks = d / 8;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t t0 = i / chunks * 4, c = (i % chunks) * 8;
  if (t0 >= tokens) return;
  float acc[4][8];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[a][j] = 0.f;
#pragma unroll 2
  for (int e = 0; e < E; ++e) {
    const float4 lo = *reinterpret_cast<const float4*>(w + (int64_t)e * d + c), hi = *reinterpret_cast<const float4*>(w + (int64_t)e * d + c + 4);
    const float wv[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const float gv = t0 + a < tokens ? g[(t0 + a) * E + e] : 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[a][j] = fmaf(gv, wv[j], acc[a][j]);
    }
  }
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    if (t0 + a >= tokens) break;
    __align__(16) T o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = from_f32<T>(acc[a][j]);
#pragma unroll
    for (int j = 0; j < (int)(8 * sizeof(T) / 16); ++j)
      reinterpret_cast<uint4*>(dx + (t0 + a) * d + c)[j] = reinterpret_cast<const uint4*>(o)[j];
  }
}

// dW = g^T x, fp32 [E, d]: a block owns 32 columns of 4 experts; 64 token slices of 4 column lanes, added in slice order
template <typename T>
__global__ void __launch_bounds__(256)
gate_project_dw_kernel(const float* g, const T* x, int64_t ldx, int64_t tokens, int E, int64_t d, float* __restrict__ dw) {
  wait_for_previous();
  __shared__ float red[64][33];
  const int cl = threadIdx.x & 3, slice = threadIdx.x >> 2;
  const int64_t c = (int64_t)blockIdx.x * 32 + cl * 8;
  const int e0 = blockIdx.y * 4;
  float acc[4][8];
#pragma unroll
  for (int b = 0; b < 4; ++b)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[b][j] = 0.f;
#pragma unroll 4
  for (int64_t t = slice; t < tokens; t += 64) {
    float xv[8];
    load8<T>(x + t * ldx + c, c < d, xv);
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const float gv = e0 + b < E ? g[t * E + e0 + b] : 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[b][j] = fmaf(gv, xv[j], acc[b][j]);
    }
  }
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; ++j) red[slice][cl * 8 + j] = acc[b][j];
    __syncthreads();
    // eight threads per column add eight slices each, then meet by shuffles
    const int col = threadIdx.x >> 3, part = threadIdx.x & 7;
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += red[part * 8 + i][col];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const int64_t oc = (int64_t)blockIdx.x * 32 + col;
    if (part == 0 && e0 + b < E && oc < d) dw[(int64_t)(e0 + b) * d + oc] = s;
  }
}

unsigned elementwise_grid(int64_t items) {
  const int64_t want = ceil_div(items, 256), cap = (int64_t)sm_count() * 8;
  return (unsigned)(want < cap ? (want > 0 ? want : 1) : cap);
}


// ---- the load-importance loss (reference impls/losses.py:21-43) -------------------------------------------------------
//   importance_e = sum_t softmax(logits)[t,e]                          (clean logits)
//   load_e       = sum_t Phi((softmax(logits)[t,e] - thr_t) / sigma)   thr_t = the k-th largest NOISY logit of token t,
//                                                                      sigma = gate_noise / E  (the reference compares a
//                                                                      score with a logit: kept as it is)
//   loss         = (cv2(importance) + cv2(load)) / 2,   cv2(v) = var(v) / (mean(v)^2 + 1e-10), var unbiased
// The top-k ids are those of the noisy logits (softmax is monotonic, so they equal torch.topk of softmax(noisy)).
__device__ __forceinline__ float normal_cdf(float z) { return 0.5f * (1.f + erff(z * 0.70710678118654752f)); }

// k-th pick of one token's noisy logits held as v[VPT] per lane; writes the ids, returns the last picked value.
template <int VPT>
__device__ __forceinline__ float warp_topk(const float (&v)[VPT], int E, int k, int lane, int32_t* __restrict__ ids, int64_t T,
                                           int64_t t, int* last_id) {
  unsigned int taken = 0;
  float thr = 0.f;
  int bi_last = 0;
  for (int j = 0; j < k; ++j) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c = lane + 32 * i;
      if (c < E && !((taken >> i) & 1u)) {
        const float x = v[i] == v[i] ? v[i] : -INFINITY;
        if (bi == 0x7fffffff || x > best) { best = x; bi = c; }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    const bool valid = (unsigned)bi < (unsigned)E;
    if (valid && (bi & 31) == lane) taken |= 1u << (bi >> 5);
    if (lane == 0 && ids) ids[(int64_t)j * T + t] = valid ? bi : -1;
    thr = best;
    bi_last = valid ? bi : -1;
  }
  *last_id = bi_last;
  return thr;
}

// cv2 of an [E] vector and its gradient factors, computed by one warp (every warp that needs them recomputes them:
// E <= 512 values).  Returns mean and var through references.
__device__ __forceinline__ void warp_mean_var(const float* v, int E, int lane, float& mean, float& var) {
  float s = 0.f;
  for (int e = lane; e < E; e += 32) s += v[e];
  mean = warp_sum(s) / (float)E;
  float q = 0.f;
  for (int e = lane; e < E; e += 32) { const float d = v[e] - mean; q += d * d; }
  var = warp_sum(q) / (float)(E - 1);
}

template <int VPT>
__global__ void __launch_bounds__(kGateThreads)
gate_topk_li_kernel(const float* logits, const float* noisy, int64_t ld, int64_t T, int E, int k,
                    float inv_sigma, int32_t* __restrict__ ids, float* __restrict__ importance, float* __restrict__ load,
                    float* __restrict__ loss, unsigned int* __restrict__ ticket, float* __restrict__ partial) {
  wait_for_previous();
  __shared__ float sum_w[kGateWarps][2 * 32 * VPT];
  __shared__ bool last_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t warp0 = (int64_t)blockIdx.x * kGateWarps + warp;
  const int64_t nwarps = (int64_t)gridDim.x * kGateWarps;
  float imp[VPT], ld_acc[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) { imp[i] = 0.f; ld_acc[i] = 0.f; }
  for (int64_t t = warp0; t < T; t += nwarps) {
    float s[VPT], v[VPT];
    warp_softmax<VPT>(logits + t * ld, E, lane, s);
#pragma unroll
    for (int i = 0; i < VPT; ++i) { const int c = lane + 32 * i; v[i] = c < E ? noisy[t * ld + c] : -INFINITY; }
    int last_id;
    const float thr = warp_topk<VPT>(v, E, k, lane, ids, T, t, &last_id);
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      if (lane + 32 * i < E) { imp[i] += s[i]; ld_acc[i] += normal_cdf((s[i] - thr) * inv_sigma); }
    }
  }
#pragma unroll
  for (int i = 0; i < VPT; ++i) { sum_w[warp][lane + 32 * i] = imp[i]; sum_w[warp][32 * VPT + lane + 32 * i] = ld_acc[i]; }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {       // per-block partial rows, warps added in index order
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int w = 0; w < kGateWarps; ++w) { a += sum_w[w][e]; b += sum_w[w][32 * VPT + e]; }
    partial[(int64_t)blockIdx.x * 2 * E + e] = a;
    partial[(int64_t)blockIdx.x * 2 * E + E + e] = b;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last_s = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last_s) return;
  __threadfence();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {       // blocks added in index order
    float a = 0.f, b = 0.f;
    for (unsigned blk = 0; blk < gridDim.x; ++blk) {
      a += __ldcg(partial + (int64_t)blk * 2 * E + e);
      b += __ldcg(partial + (int64_t)blk * 2 * E + E + e);
    }
    importance[e] = a;
    load[e] = b;
  }
  __threadfence();
  __syncthreads();
  if (warp == 0) {
    float mi, vi, ml, vl;
    warp_mean_var(importance, E, lane, mi, vi);
    warp_mean_var(load, E, lane, ml, vl);
    if (lane == 0) loss[0] = 0.5f * (vi / (mi * mi + 1e-10f) + vl / (ml * ml + 1e-10f));
  }
}

// d loss / d logits for gate_topk_li_kernel's loss, times dloss[0].  With g_i = d loss / d importance and g_l = d loss /
// d load (from the forward's totals), pdf_e = phi(z_e) / sigma:
//   d s_e = g_i[e] + g_l[e] pdf_e ;  d thr = - sum_e g_l[e] pdf_e  (reaches the clean logit of the k-th choice: the noise is a constant)
//   d logits_e = s_e (d s_e - sum_e' s_e' d s_e') + [e = k-th choice] d thr
template <int VPT>
__global__ void __launch_bounds__(kGateThreads)
gate_li_grad_kernel(const float* logits, const float* noisy, int64_t ld, int64_t T, int E, int k,
                    float inv_sigma, const float* importance, const float* load,
                    const float* dloss, float* __restrict__ dlogits, int64_t ldd) {
  wait_for_previous();
  const int lane = threadIdx.x & 31;
  const int64_t warp0 = (int64_t)blockIdx.x * kGateWarps + (threadIdx.x >> 5);
  const int64_t nwarps = (int64_t)gridDim.x * kGateWarps;
  float mi, vi, ml, vl;
  warp_mean_var(importance, E, lane, mi, vi);
  warp_mean_var(load, E, lane, ml, vl);
  const float up = 0.5f * *dloss;
  const float di = mi * mi + 1e-10f, dl = ml * ml + 1e-10f;
  float gi[VPT], gl[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = lane + 32 * i;
    // d cv2 / d v_e = 2 (v_e - mean) / ((E-1) den) - var * 2 mean / (E den^2)
    gi[i] = c < E ? up * (2.f * (importance[c] - mi) / ((float)(E - 1) * di) - vi * 2.f * mi / ((float)E * di * di)) : 0.f;
    gl[i] = c < E ? up * (2.f * (load[c] - ml) / ((float)(E - 1) * dl) - vl * 2.f * ml / ((float)E * dl * dl)) : 0.f;
  }
  for (int64_t t = warp0; t < T; t += nwarps) {
    float s[VPT], v[VPT];
    warp_softmax<VPT>(logits + t * ld, E, lane, s);
#pragma unroll
    for (int i = 0; i < VPT; ++i) { const int c = lane + 32 * i; v[i] = c < E ? noisy[t * ld + c] : -INFINITY; }
    int last_id;
    const float thr = warp_topk<VPT>(v, E, k, lane, nullptr, T, t, &last_id);
    float ds[VPT];
    float dthr = 0.f, dot = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const float z = (s[i] - thr) * inv_sigma;
      const float pdf = (lane + 32 * i) < E ? 0.3989422804014327f * expf(-0.5f * z * z) * inv_sigma : 0.f;
      ds[i] = gi[i] + gl[i] * pdf;
      dthr -= gl[i] * pdf;
      dot += s[i] * ds[i];
    }
    dthr = warp_sum(dthr);
    dot = warp_sum(dot);
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c = lane + 32 * i;
      if (c < E) dlogits[t * ldd + c] = s[i] * (ds[i] - dot) + (c == last_id ? dthr : 0.f);
    }
  }
}

// Blocks of the group kernels: one sweep of a block covers warps * 32 / G tokens, 24 or 32 warps per SM at most.  Blocks of
// 32 warps where their column sums fit in shared memory: 148 partial rows instead of 444 for gate_finish_kernel to add.
int gate_group_grid(int64_t T, int G, int warps) {
  int64_t cap = (int64_t)sm_count() * (warps == 32 ? 1 : 3);
  if (cap > kGateMaxBlocks / 2) cap = kGateMaxBlocks / 2;      // a block leaves two rows of words
  const int64_t want = ceil_div(T, warps * (32 / G));
  return (int)(want < cap ? want : cap);
}
// Tokens that one block takes by itself, saving the second launch (~3 us): four sweeps at ~1 us each, of 32 warps where
// their column sums fit in shared memory.
constexpr int lone_warps(int G) { return G < 32 ? 32 : kGateWarps; }
constexpr int64_t lone_tokens(int G) { return 4 * lone_warps(G) * (32 / G); }

#define HEXA_GATE_DISPATCH(E, LAUNCH)  \
  do {                                 \
    if ((E) <= 8) { LAUNCH(8, 1); }    \
    else if ((E) <= 16) { LAUNCH(8, 2); }  \
    else if ((E) <= 32) { LAUNCH(8, 4); }  \
    else if ((E) <= 64) { LAUNCH(8, 8); }  \
    else if ((E) <= 128) { LAUNCH(16, 8); } \
    else if ((E) <= 256) { LAUNCH(32, 8); } \
    else { LAUNCH(32, 16); }           \
  } while (0);

int gate_grid(int64_t T) {
  const int64_t want = ceil_div(T, kGateThreads / 32);
  int64_t cap = (int64_t)sm_count() * 4;
  if (cap > kGateMaxBlocks) cap = kGateMaxBlocks;
  return (int)(want < cap ? (want > 0 ? want : 1) : cap);
}

}  // namespace
}  // namespace hexa

using namespace hexa;

extern "C" int hexa_gate_max_experts(void) { return kGateMaxExperts; }

extern "C" size_t hexa_gate_workspace_bytes(void) {
  return kGateTicketBytes + (size_t)kGateMaxBlocks * kGateMaxExperts * sizeof(float);   // ticket + partial-mass rows (2 MiB)
}

extern "C" int hexa_gate_topk(const float* logits, int64_t ld, int64_t num_tokens, int num_experts, int top_k, int32_t* ids,
                              float* mass, int32_t* first_count, float* loss, void* workspace, size_t workspace_bytes,
                              void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  HEXA_REQUIRE(num_tokens >= 0 && num_experts >= 1 && num_experts <= kGateMaxExperts, "hexa_gate_topk: needs 1 <= experts <= %d (got %d)",
               kGateMaxExperts, num_experts);
  HEXA_REQUIRE(top_k >= 1 && top_k <= num_experts, "hexa_gate_topk: top_k %d out of range for %d experts", top_k, num_experts);
  HEXA_REQUIRE(mass && first_count && loss && workspace && workspace_bytes >= hexa_gate_workspace_bytes(),
               "hexa_gate_topk: null output or workspace smaller than hexa_gate_workspace_bytes()");
  HEXA_REQUIRE(num_tokens == 0 || (logits && ids && ld >= num_experts), "hexa_gate_topk: null logits/ids or ld < experts");
  HEXA_REQUIRE(aligned16(workspace), "hexa_gate_topk: workspace must be 16-byte aligned");
  if (num_tokens == 0) {
    HEXA_CUDA(cudaMemsetAsync(mass, 0, sizeof(float) * num_experts, stream));
    HEXA_CUDA(cudaMemsetAsync(first_count, 0, sizeof(int32_t) * num_experts, stream));
    HEXA_CUDA(cudaMemsetAsync(loss, 0, sizeof(float), stream));
    return HEXA_OK;
  }
  float* partial = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + kGateTicketBytes);
  int grid = 1;
#define HEXA_GATE_FWD(G, PER)                                                                                              \
  if (num_tokens <= lone_tokens(G)) {                                                                                      \
    after_previous(gate_topk_kernel<G, PER, lone_warps(G)>, 1, lone_warps(G) * 32, 0, stream)(logits, ld, num_tokens, num_experts,     \
                                                                                  top_k, ids, mass, first_count, loss,     \
                                                                                  partial);                                \
  } else {                                                                                                                 \
    grid = gate_group_grid(num_tokens, G, lone_warps(G));                                                                  \
    after_previous(gate_topk_kernel<G, PER, lone_warps(G)>, grid, lone_warps(G) * 32, 0, stream)(logits, ld, num_tokens, num_experts,  \
                                                                                     top_k, ids, mass, first_count, loss,  \
                                                                                     partial);                             \
  }
  HEXA_GATE_DISPATCH(num_experts, HEXA_GATE_FWD)
#undef HEXA_GATE_FWD
  HEXA_LAUNCH_CHECK("gate_topk_kernel");
  if (grid > 1) {
    after_previous(gate_finish_kernel, 1, kFinishThreads, 0, stream)(partial, grid, num_tokens, num_experts, mass, first_count, loss);
    HEXA_LAUNCH_CHECK("gate_finish_kernel");
  }
  return HEXA_OK;
}

extern "C" int hexa_gate_loss_grad(const float* logits, int64_t ld, int64_t num_tokens, int num_experts,
                                   const int32_t* first_count, const float* dloss, float* dlogits, int64_t ldd, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  HEXA_REQUIRE(num_tokens >= 0 && num_experts >= 1 && num_experts <= kGateMaxExperts, "hexa_gate_loss_grad: needs 1 <= experts <= %d (got %d)",
               kGateMaxExperts, num_experts);
  if (num_tokens == 0) return HEXA_OK;
  HEXA_REQUIRE(logits && first_count && dloss && dlogits && ld >= num_experts && ldd >= num_experts,
               "hexa_gate_loss_grad: null pointer or leading dimension < experts");
  int grid = 1;
#define HEXA_GATE_BWD(G, PER)                                                                                             \
  grid = gate_group_grid(num_tokens, G, kGateWarps);                                                                      \
  after_previous(gate_loss_grad_kernel<G, PER>, grid, kGateThreads, 0, stream)(logits, ld, num_tokens, num_experts, first_count, dloss, \
                                                                   dlogits, ldd)
  HEXA_GATE_DISPATCH(num_experts, HEXA_GATE_BWD)
#undef HEXA_GATE_BWD
  HEXA_LAUNCH_CHECK("gate_loss_grad_kernel");
  return HEXA_OK;
}

extern "C" int hexa_gate_split_terms(const float* src, int64_t ld, int64_t rows, int64_t cols, int by_rows, void* out, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  HEXA_REQUIRE(rows >= 0 && cols >= 0 && ld >= cols, "hexa_gate_split_terms: bad sizes");
  if (rows == 0 || cols == 0) return HEXA_OK;
  HEXA_REQUIRE(src && out, "hexa_gate_split_terms: null pointer");
  if (by_rows) {      // blocks of rows: the same as blocks of columns of one long row
    HEXA_REQUIRE(ld == cols, "hexa_gate_split_terms: blocks of rows need a contiguous source");
    cols *= rows;
    ld = cols;
    rows = 1;
  }
  __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out);
  const bool v4 = cols % 4 == 0 && ld % 4 == 0 && aligned16(src) && aligned16(out);
  if (v4) after_previous(split_terms_kernel<4>, elementwise_grid(rows * cols / 4), 256, 0, stream)(src, ld, rows, cols, by_rows, o);
  else after_previous(split_terms_kernel<1>, elementwise_grid(rows * cols), 256, 0, stream)(src, ld, rows, cols, by_rows, o);
  HEXA_LAUNCH_CHECK("split_terms_kernel");
  return HEXA_OK;
}

extern "C" int hexa_gate_sum_terms(const float* part, int64_t rows, int64_t cols, int lo_first, float* out, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  HEXA_REQUIRE(rows >= 0 && cols >= 0, "hexa_gate_sum_terms: bad sizes");
  if (rows == 0 || cols == 0) return HEXA_OK;
  HEXA_REQUIRE(part && out, "hexa_gate_sum_terms: null pointer");
  const bool v4 = cols % 4 == 0 && aligned16(part) && aligned16(out);
  if (v4) after_previous(sum_terms_kernel<4>, elementwise_grid(rows * cols / 4), 256, 0, stream)(part, rows, cols, lo_first, out);
  else after_previous(sum_terms_kernel<1>, elementwise_grid(rows * cols), 256, 0, stream)(part, rows, cols, lo_first, out);
  HEXA_LAUNCH_CHECK("sum_terms_kernel");
  return HEXA_OK;
}

extern "C" int hexa_gate_topk_load_importance(const float* logits, const float* logits_w_noise, int64_t ld, int64_t num_tokens,
                                              int num_experts, int top_k, float sigma, int32_t* ids, float* importance,
                                              float* load, float* loss, void* workspace, size_t workspace_bytes, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  HEXA_REQUIRE(num_tokens >= 0 && num_experts >= 1 && num_experts <= kGateMaxExperts,
               "hexa_gate_topk_load_importance: needs 1 <= experts <= %d (got %d)", kGateMaxExperts, num_experts);
  HEXA_REQUIRE(top_k >= 1 && top_k <= num_experts, "hexa_gate_topk_load_importance: top_k %d out of range for %d experts", top_k, num_experts);
  HEXA_REQUIRE(sigma > 0.f, "hexa_gate_topk_load_importance: sigma (gate_noise / experts) must be > 0");
  HEXA_REQUIRE(importance && load && loss && workspace && workspace_bytes >= hexa_gate_workspace_bytes() && aligned16(workspace),
               "hexa_gate_topk_load_importance: null output, or workspace smaller than hexa_gate_workspace_bytes() or not 16-byte aligned");
  HEXA_REQUIRE(num_tokens == 0 || (logits && logits_w_noise && ids && ld >= num_experts),
               "hexa_gate_topk_load_importance: null logits/ids or ld < experts");
  HEXA_CUDA(cudaMemsetAsync(importance, 0, sizeof(float) * num_experts, stream));
  HEXA_CUDA(cudaMemsetAsync(load, 0, sizeof(float) * num_experts, stream));
  HEXA_CUDA(cudaMemsetAsync(loss, 0, sizeof(float), stream));
  HEXA_CUDA(cudaMemsetAsync(workspace, 0, 16, stream));
  if (num_tokens == 0) return HEXA_OK;
  unsigned int* ticket = static_cast<unsigned int*>(workspace);
  float* partial = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + kGateTicketBytes);
  int grid = gate_grid(num_tokens);
  if (grid > kGateMaxBlocks / 2) grid = kGateMaxBlocks / 2;      // two partial rows per block
  const float inv_sigma = 1.f / sigma;
#define HEXA_GATE_LI(V)                                                                                                     \
  after_previous(gate_topk_li_kernel<V>, grid, kGateThreads, 0, stream)(logits, logits_w_noise, ld, num_tokens, num_experts, top_k, inv_sigma, \
                                                            ids, importance, load, loss, ticket, partial)
  const int vpt = (num_experts + 31) / 32;
  if (vpt <= 1) HEXA_GATE_LI(1);
  else if (vpt <= 2) HEXA_GATE_LI(2);
  else if (vpt <= 4) HEXA_GATE_LI(4);
  else if (vpt <= 8) HEXA_GATE_LI(8);
  else HEXA_GATE_LI(16);
#undef HEXA_GATE_LI
  HEXA_LAUNCH_CHECK("gate_topk_li_kernel");
  return HEXA_OK;
}

extern "C" int hexa_gate_load_importance_grad(const float* logits, const float* logits_w_noise, int64_t ld, int64_t num_tokens,
                                              int num_experts, int top_k, float sigma, const float* importance, const float* load,
                                              const float* dloss, float* dlogits, int64_t ldd, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  HEXA_REQUIRE(num_tokens >= 0 && num_experts >= 1 && num_experts <= kGateMaxExperts,
               "hexa_gate_load_importance_grad: needs 1 <= experts <= %d (got %d)", kGateMaxExperts, num_experts);
  HEXA_REQUIRE(top_k >= 1 && top_k <= num_experts && sigma > 0.f, "hexa_gate_load_importance_grad: bad top_k or sigma");
  if (num_tokens == 0) return HEXA_OK;
  HEXA_REQUIRE(logits && logits_w_noise && importance && load && dloss && dlogits && ld >= num_experts && ldd >= num_experts,
               "hexa_gate_load_importance_grad: null pointer or leading dimension < experts");
  const int grid = gate_grid(num_tokens);
  const float inv_sigma = 1.f / sigma;
#define HEXA_GATE_LIG(V)                                                                                                     \
  after_previous(gate_li_grad_kernel<V>, grid, kGateThreads, 0, stream)(logits, logits_w_noise, ld, num_tokens, num_experts, top_k, inv_sigma, \
                                                            importance, load, dloss, dlogits, ldd)
  const int vpt = (num_experts + 31) / 32;
  if (vpt <= 1) HEXA_GATE_LIG(1);
  else if (vpt <= 2) HEXA_GATE_LIG(2);
  else if (vpt <= 4) HEXA_GATE_LIG(4);
  else if (vpt <= 8) HEXA_GATE_LIG(8);
  else HEXA_GATE_LIG(16);
#undef HEXA_GATE_LIG
  HEXA_LAUNCH_CHECK("gate_li_grad_kernel");
  return HEXA_OK;
}

extern "C" int hexa_gate_project(const void* x, int64_t ldx, const float* w, int64_t tokens, int num_experts, int64_t d, int dtype,
                                 float* logits, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  HEXA_REQUIRE(tokens >= 0 && num_experts >= 1 && d >= 8 && d % 8 == 0 && ldx >= d && ldx % 8 == 0, "hexa_gate_project: bad sizes (d and ldx must be multiples of 8)");
  HEXA_REQUIRE(dtype == HEXA_F32 || dtype == HEXA_F16 || dtype == HEXA_BF16, "hexa_gate_project: bad dtype %d", dtype);
  if (tokens == 0) return HEXA_OK;
  HEXA_REQUIRE(x && w && logits && aligned16(x) && aligned16(w), "hexa_gate_project: null or unaligned pointer");
  const int64_t tiles = ceil_div(tokens, 4) * ceil_div(num_experts, 4);
  HEXA_REQUIRE(ceil_div(tiles, 4) < INT32_MAX, "hexa_gate_project: too many tokens");
  const unsigned grid = (unsigned)ceil_div(tiles, 4);
  if (dtype == HEXA_F32) after_previous(gate_project_kernel<float>, grid, 128, 0, stream)((const float*)x, ldx, w, tokens, num_experts, d, logits);
  else if (dtype == HEXA_F16) after_previous(gate_project_kernel<__half>, grid, 128, 0, stream)((const __half*)x, ldx, w, tokens, num_experts, d, logits);
  else after_previous(gate_project_kernel<__nv_bfloat16>, grid, 128, 0, stream)((const __nv_bfloat16*)x, ldx, w, tokens, num_experts, d, logits);
  HEXA_LAUNCH_CHECK("gate_project_kernel");
  return HEXA_OK;
}

extern "C" int hexa_gate_project_grad(const float* g, const void* x, int64_t ldx, const float* w, int64_t tokens, int num_experts,
                                      int64_t d, int dtype, void* dx, float* dw, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  HEXA_REQUIRE(tokens >= 1 && num_experts >= 1 && d >= 8 && d % 8 == 0 && ldx >= d && ldx % 8 == 0, "hexa_gate_project_grad: bad sizes (d and ldx must be multiples of 8)");
  HEXA_REQUIRE(dtype == HEXA_F32 || dtype == HEXA_F16 || dtype == HEXA_BF16, "hexa_gate_project_grad: bad dtype %d", dtype);
  HEXA_REQUIRE(g && (!dx || (w && aligned16(w) && aligned16(dx))) && (!dw || (x && aligned16(x))), "hexa_gate_project_grad: null or unaligned pointer");
  const int64_t blocks = ceil_div(ceil_div(tokens, 4) * (d / 8), 128);
  HEXA_REQUIRE(blocks < INT32_MAX && ceil_div(num_experts, 4) <= 65535, "hexa_gate_project_grad: too many tokens or experts");
  if (dx) {
    if (dtype == HEXA_F32) after_previous(gate_project_dx_kernel<float>, (unsigned)blocks, 128, 0, stream)(g, w, tokens, num_experts, d, (float*)dx);
    else if (dtype == HEXA_F16) after_previous(gate_project_dx_kernel<__half>, (unsigned)blocks, 128, 0, stream)(g, w, tokens, num_experts, d, (__half*)dx);
    else after_previous(gate_project_dx_kernel<__nv_bfloat16>, (unsigned)blocks, 128, 0, stream)(g, w, tokens, num_experts, d, (__nv_bfloat16*)dx);
    HEXA_LAUNCH_CHECK("gate_project_dx_kernel");
  }
  if (dw) {
    const dim3 grid((unsigned)ceil_div(d, 32), (unsigned)ceil_div(num_experts, 4));
    if (dtype == HEXA_F32) after_previous(gate_project_dw_kernel<float>, grid, 256, 0, stream)(g, (const float*)x, ldx, tokens, num_experts, d, dw);
    else if (dtype == HEXA_F16) after_previous(gate_project_dw_kernel<__half>, grid, 256, 0, stream)(g, (const __half*)x, ldx, tokens, num_experts, d, dw);
    else after_previous(gate_project_dw_kernel<__nv_bfloat16>, grid, 256, 0, stream)(g, (const __nv_bfloat16*)x, ldx, tokens, num_experts, d, dw);
    HEXA_LAUNCH_CHECK("gate_project_dw_kernel");
  }
  return HEXA_OK;
}
