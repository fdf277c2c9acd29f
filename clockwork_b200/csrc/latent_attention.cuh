// What the kernels of the attention over a cached latent share.
#pragma once
#include "request_tiles.cuh"

struct LatentArgs {
    const bf16* qa;           // [N*H, D]
    bf16* out;                // [N*H, rank]
    const bf16* cache;        // [slots, D]
    const int* block_tables;  // [S, max_blocks]
    const int* tok_seq;       // [N], < 0: padding
    const int* positions;     // [N]
    const int* q_start;       // [S + 1]
    const float* sink;        // [H] or null
    int N, S, H, rank, rot, page_size, max_blocks, num_pages;
    float scale;
    int parts;
    float* partial;           // parts > 1: [parts, N*H, rank] sums, then [parts, N*H, 2] running maxima and denominators
    int* status;
};

// Whether the tcgen05 kernel takes these sizes (uncut keys); and the launch.
bool latent_tc_takes(const LatentArgs& a);
int latent_tc_run(const LatentArgs& a, cudaStream_t stream);
