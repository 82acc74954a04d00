// Launchers of the GEMM-shaped operators, one set per kernel family (defined in gemm_tc.cu and gemm_simt.cu,
// selected by the C-ABI entry points in ops_api.cu).  Argument order follows hexa_esmm / hexa_estmm.
#pragma once

#include <cuda.h>

#include "hexa_common.cuh"

namespace hexa {
// gemm_tc.cu: cuTensorMapEncodeTiled with zero fill out of bounds, rank up to 4
int encode_tensor_map(CUtensorMap* tm, const void* base, CUtensorMapDataType type, int rank, const uint64_t* dims,
                      const uint64_t* strides_bytes, const uint32_t* box, CUtensorMapSwizzle swizzle);
// gemm_f32.cu: fp32 operands as three bf16 planes on the tensor cores.  *_workspace_bytes: 0 where it does not pay or apply.
size_t esmm_f32_workspace_bytes(int E, int64_t row_cap, int64_t n_out, int64_t k);
size_t estmm_f32_workspace_bytes(int E, int64_t row_cap, int64_t m, int64_t n);
int esmm_f32_launch(const void* a, int64_t lda, const void* b, int b_layout, int64_t ldb, int64_t b_estride, const float* bias,
                    int64_t ldbias, void* aux, int64_t ldaux, void* c, int64_t ldc, const int32_t* tile_expert,
                    const int32_t* pad_offsets, const int32_t* row_token, const int32_t* pair_block, int E, int64_t row_cap,
                    int64_t n_out, int64_t k, int epilogue, int act, cudaStream_t stream, void* workspace);
int estmm_f32_launch(const void* p, int64_t ldp, const void* q, int64_t ldq, const int32_t* pad_offsets, int E, int64_t row_cap,
                     int64_t m, int64_t n, void* out, int64_t ldo, int64_t o_estride, cudaStream_t stream, void* workspace);
// The CUDA-core launchers below can be told to do nothing unless a device word is set (`only_if`; null: always run).
// (their bias, and that of esmm_tc_launch, is fp32 or, with bias16, of the data's 16-bit type)
int esmm_simt_launch(const void*, int64_t, const void*, int, int64_t, int64_t, const void*, int64_t, void*, int64_t, void*,
                     int64_t, const int32_t*, const int32_t*, const int32_t*, int, int64_t, int64_t, int64_t, int, int, int,
                     cudaStream_t, int e_begin, int e_end, int bias16 = 0, const int32_t* only_if = nullptr);
int estmm_simt_launch(const void*, int64_t, const void*, int64_t, const int32_t*, int, int64_t, int64_t, void*, int64_t,
                      int64_t, int64_t, int64_t, int, int, int, cudaStream_t, const int32_t* only_if = nullptr);
bool esmm_tc_supported(const void*, int64_t, const void*, int64_t, int64_t, const void*, int64_t, const void*, int64_t,
                       const float*, int64_t, int64_t, int);
int esmm_tc_launch(const void*, int64_t, const void*, int, int64_t, int64_t, const void*, int64_t, void*, int64_t, void*,
                   int64_t, const int32_t*, const int32_t*, const int32_t*, const int32_t*, int, int64_t, int64_t, int64_t, int,
                   int, int, cudaStream_t, int e_begin, int e_end, int bias16, float* colsum = nullptr);
bool estmm_tc_supported(const void*, int64_t, const void*, int64_t, const void*, int64_t, int64_t, int64_t, int64_t, int, int);
int estmm_tc_launch(const void*, int64_t, const void*, int64_t, const int32_t*, int, int64_t, int64_t, int64_t, void*, int64_t,
                    int64_t, int64_t, int64_t, int, int, int, cudaStream_t, void* const* split_out = nullptr, int n_split = 0,
                    void* workspace = nullptr, size_t workspace_bytes = 0);
size_t estmm_tc_workspace_bytes(int E, int64_t row_cap, int64_t m, int64_t n);
// rows.cu: both passes of ESS, and its second pass alone (per expert, the partial rows of its 128-row blocks added in order)
int ess_launch(const void* src, int64_t src_ld, const int32_t* pad_offsets, int E, int64_t row_cap, int64_t cols, void* out,
               int64_t ldo, int out_dtype, int dtype, float* partial, cudaStream_t stream);
int ess_finish(const float* partial, const int32_t* pad_offsets, int E, int64_t cols, void* out, int64_t ldo, int out_dtype,
               cudaStream_t stream);
}  // namespace hexa
