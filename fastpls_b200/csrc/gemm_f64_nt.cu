// FP64 tensor-core GEMM tiles, op(A) = A, op(B) = B^T.
#include "gemm_f64.cuh"

FPLS_GEMM64_INSTANTIATE(false, true)
