// float32 products on the tensor cores (gemm_f32.cu), called from ptj_gemm.
#pragma once
#include "gemm_epilogue.cuh"

namespace ptj {
// Floats of workspace with which a float32 product of this shape runs on the tensor cores; 0: it stays on the
// fused-multiply-add kernel.
size_t gemm_f32_workspace_floats(int64_t M, int64_t N, int64_t K, bool a_kmajor, bool b_kmajor);
// The product, arguments already validated; workspace: at least that many floats, 256-byte aligned planes inside it need
// a 16-byte aligned base.
int gemm_f32_tc(const float* a, const float* b, const EpilogueParams& ep, int64_t M, int64_t N, int64_t K, int64_t lda,
                int64_t ldb, bool a_kmajor, bool b_kmajor, float* workspace, cudaStream_t st);
}  // namespace ptj
