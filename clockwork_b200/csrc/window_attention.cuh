// What the kernels of the windowed attention share.
#pragma once
#include "request_tiles.cuh"

struct WindowAttentionArgs {
    const void* q;            // [N, ldq]: head h's query at columns h*dk ..
    int ldq;
    const void* cache;        // [rows, G, dk + dv]
    const int* block_tables;  // [S, max_blocks]
    int max_blocks, page_size, num_pages;
    const int* positions;     // [N]
    const int* tok_seq;       // [N], < 0: padding
    int H, G, dk, dv, window;
    float scale;
    const float* head_scale;  // [H] or null: multiplied into the score
    const float* talk;        // [H, H] or null: score_h <- sum_g talk[h, g] score_g
    const float* head_bias;   // [H] or null: added to the mixed score
    int sigmoid_weights;      // 0: softmax over the visible keys; 1: sigmoid of each score, not normalised
    int blocked;              // 0: p sees the last `window` positions; 1: p sees its own block of `window` positions up to itself
    const float* sink;        // [H] or null: a logit per head that counts once in the softmax's denominator
    void* out;                // [N, H*dv]
    int tile;                 // keys per tile (<= 32)
    int parts, part_keys;     // a token's window in `parts` pieces of `part_keys` keys (a multiple of tile)
    float* partial;           // parts > 1: [N, parts, H*dv + 2H] sums, running maxima and denominators
    int* status;
    // further switches (all off when zero or null)
    float softcap;            // > 0: score <- softcap tanh(score / softcap)
    const float* slopes;      // [H] or null: slopes[h] * (p - j) is taken off the score
    float temp_coef;          // with temp_every > 0: the score of a query at position p is multiplied by
    int temp_every;           //   1 + temp_coef ln(floor((p + 1) / temp_every) + 1)
    const float* gate;        // [N, ldg] or null: head h's output is multiplied by sigmoid(gate[n * ldg + h])
    int ldg;
    int pool;                 // > 0: blocks of `pool` positions that end at or before p - window are seen as one row each
    const void* pool_cache;   // [rows, G, dk + dv]: row b of a request is the mean of its positions b*pool .. b*pool + pool - 1
    const int* pool_tables;   // [S, pool_max_blocks]
    int pool_max_blocks, pool_pages;
    int keep;                 // the sequence's first `keep` positions are seen by every later one
    int voff;                 // where a head's value begins in its row (row width voff + dv; below dk: key and value overlap)
    int gate_entries;         // 1: the gate has a number per output entry ([N, ldg], ldg >= H*dv) instead of one per head
};

__device__ __forceinline__ float wa_query_temperature(int p, float coef, int every) {
    return every > 0 ? 1.f + coef * logf((float)((p + 1) / every + 1)) : 1.f;
}

// Whether the tcgen05 kernel takes these switches, sizes and addresses; whether it is faster than the mma.sync kernel for a step of N
// rows of S requests; and the launch (a.parts is not looked at there: rows are not cut).
#define WC_MAX_PARTS 4
bool window_tc_takes(const WindowAttentionArgs& a);
bool window_tc_pays(const WindowAttentionArgs& a, int N, int S);
int window_tc_run(const WindowAttentionArgs& a, const int* q_start, int S, int N, cudaStream_t stream);
