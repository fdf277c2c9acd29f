// Products of float32 operands on the tensor cores (gemm_f32.cu), called by the entry points of gemm_ref.cu.
#pragma once
#include "common.cuh"

struct F32Args {
    const float *A, *W, *W2, *bias;  // A [M, K] with rows of lda, W and W2 (SwiGLU; else null) [N, K]
    float* C;                        // [M, N] with rows of ldc
    int M, N, K, lda, ldc, epilogue;
    int* status;
    int width, rows;  // tokens and weight rows of a CTA's tile (chosen by the launcher)
    int whole;        // rows of A, W and W2 are whole 16-byte pieces at 16-byte bases
};

int gemm_f32_run(F32Args p, cudaStream_t stream);
