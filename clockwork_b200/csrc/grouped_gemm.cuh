// What the kernels of the products in groups share: the epilogues, and the entry of the tcgen05 form.
#pragma once
#include "common.cuh"

#define GG_EPI_STORE 0        // C (T) = acc
#define GG_EPI_STORE_F32 1    // C (float) = acc
#define GG_EPI_SILU_MUL 2     // C (T) = silu(acc) * acc2, acc2 from B2; with a positive `glu_limit` the clamped form below
#define GG_EPI_SIGMOID_GATE 3 // C (T) = acc * sigmoid(gate[dst, c_group_off*g + n])
#define GG_EPI_RELU2 4        // C (T) = max(acc, 0)^2
#define GG_EPI_GROUP_GATE 5   // C (T) = acc * sigmoid(gate[dst, g]), `gate` float32: one number per row and group

// The gated activation of the two-product form: silu(a) b, or, with a positive limit,
//   a' = min(a, limit), b' = clamp(b, -limit, limit):  a' sigmoid(1.702 a') (b' + 1)
__device__ __forceinline__ float gg_glu(float a, float b, float limit) {
    if (limit > 0.f) {
        a = fminf(a, limit);
        b = fminf(fmaxf(b, -limit), limit);
        return a / (1.f + expf(-1.702f * a)) * (b + 1.f);
    }
    return a / (1.f + expf(-a)) * b;
}

// The arguments of cw_grouped_gemm (see there), bfloat16 operands.
struct GroupedArgs {
    const bf16 *A, *B, *B2;
    int lda, a_group_off;
    long long b_stride;
    void* C;
    int ldc, c_group_off;
    const int *offsets, *a_index;
    int a_div;
    const int* c_index;
    const void* gate;  // bfloat16 (GG_EPI_SIGMOID_GATE) or float32 (GG_EPI_GROUP_GATE)
    int ldg, M, Nout, K, G;
    float glu_limit;
    int* status;
};
// Whether the tcgen05 kernels take these sizes, strides and pointers; and the launch.
bool grouped_tc_takes(const GroupedArgs& p, int epilogue);
int grouped_tc_run(const GroupedArgs& p, int epilogue, cudaStream_t stream);
