// Paged causal attention, general form: any mixture of prompt portions and single decoded
// tokens, any head count / group size / head size, optional window.  One thread block per
// (token, query head); float32 scores, softmax and accumulation in both run precisions.
//
// Reference: clockwork/kernels/attention.py:45-65 (scores = q.k * scale with the scale applied
// after the dot product, key j visible to the query at absolute position p iff j <= p,
// softmax, P.V), :35-42 (query head h reads KV head h // (nh/nkv)), :68-96 and :113-134 (keys
// and values gathered through the request's block table).  A token's keys are those of its own
// request at positions [max(0, p+1-window), p]; they are read from the cache, where this step's
// tokens were written before (clockwork/engine/model.py:100-127).
//
// Keys are processed in chunks of 128 starting at the first visible key; the chunking depends
// on the token's position and the window only, never on the rest of the batch.
//
// Two kernels with the same operations in the same order per row, so the same bits: attn_rows_kernel for float32 portions of a few
// rows or more, without a window; attn_ref_kernel for everything else.
#include "attention_mma.cuh"
#include "request_tiles.cuh"

#define CH 128

template <typename T>
__global__ void __launch_bounds__(CH)
attn_ref_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out,
                const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                const int* __restrict__ block_tables, const int* __restrict__ tok_seq,
                const int* __restrict__ positions, int nh, int nkv, int hd, int page_size,
                int max_blocks, int num_pages, float scale, int window, const int* __restrict__ q_start, int S,
                int below, int* status) {
    extern __shared__ float q_s[];  // [hd]
    __shared__ float p_s[CH];
    __shared__ int slot_s[CH];
    __shared__ float scratch[33];
    __shared__ int row_s;
    const int h = blockIdx.y, tid = threadIdx.x;
    int t = blockIdx.x;
    if (below > 0) {  // the rows of short requests one after the other (attn_rows_kernel has the others, and padding)
        if (tid < 32) {
            const RowTile tile = find_row_tile(blockIdx.x, false, q_start, tok_seq, S, 1, 1, 1, below);
            if (tid == 0) row_s = tile.seq >= 0 ? tile.row0 : -1;
        }
        __syncthreads();
        t = row_s;
        if (t < 0) return;
    }
    const int kvh = h / (nh / nkv);
    const int seq = tok_seq[t];
    T* o = out + ((size_t)t * nh + h) * hd;
    if (seq < 0) {  // padding row of a fixed-shape batch
        for (int d = tid; d < hd; d += CH) o[d] = from_f<T>(0.f);
        return;
    }
    const int kv_end = positions[t] + 1;
    const int kv_begin = window > 0 ? max(0, kv_end - window) : 0;
    const T* qrow = q + (size_t)t * q_stride + (size_t)h * hd;
    for (int d = tid; d < hd; d += CH) q_s[d] = to_f(qrow[d]);
    __syncthreads();
    const int* table = block_tables + (size_t)seq * max_blocks;
    float m = -INFINITY, l = 0.f;
    float acc0 = 0.f, acc1 = 0.f;  // output dims tid and tid + CH (hd <= 256)
    for (int c0 = kv_begin; c0 < kv_end; c0 += CH) {
        const int j = c0 + tid;
        float s = -INFINITY;
        int slot = -1;
        if (j < kv_end) {
            const int blk = j / page_size;
            const int page = blk < max_blocks ? table[blk] : -1;
            if (page < 0 || page >= num_pages) {
                cw_report(status, CW_ST_PAGE_RANGE, t, page);
            } else {
                slot = page * page_size + j % page_size;
                const T* kp = k_cache + ((size_t)slot * nkv + kvh) * hd;
                float dot = 0.f;
                for (int d = 0; d < hd; ++d) dot = fmaf(q_s[d], to_f(kp[d]), dot);
                s = dot * scale;
            }
        }
        slot_s[tid] = slot;
        const float m_new = fmaxf(m, block_max(s, scratch));
        const float p = (slot >= 0) ? expf(s - m_new) : 0.f;
        p_s[tid] = p;
        const float csum = block_sum(p, scratch);  // also orders p_s/slot_s writes before reads
        const float alpha = (m == -INFINITY) ? 0.f : expf(m - m_new);
        l = l * alpha + csum;
        acc0 *= alpha;
        acc1 *= alpha;
        const int n = min(CH, kv_end - c0);
        if (m_new != -INFINITY) {
            for (int jj = 0; jj < n; ++jj) {
                const int sl = slot_s[jj];
                if (sl < 0) continue;
                const T* vp = v_cache + ((size_t)sl * nkv + kvh) * hd;
                const float pj = p_s[jj];
                if (tid < hd) acc0 = fmaf(pj, to_f(vp[tid]), acc0);
                if (tid + CH < hd) acc1 = fmaf(pj, to_f(vp[tid + CH]), acc1);
            }
            m = m_new;
        }
        __syncthreads();
    }
    const float inv = l > 0.f ? 1.0f / l : 0.f;
    if (tid < hd) o[tid] = from_f<T>(acc0 * inv);
    if (tid + CH < hd) o[tid + CH] = from_f<T>(acc1 * inv);
}

// The same for float32 rows of a portion: a block takes up to 16 consecutive rows of one request and one head (four a warp), so that
// a chunk's keys and values are fetched once for 16 rows and read from shared memory; the next chunk's keys are on their way while
// the weights and the weighted sum are formed, its values while its scores are.  attn_ref_kernel fetches every key and value from L2 for
// every row, a row of the cache per thread: bound by those reads.  A row's chunks, its dot products (ascending entries), the
// trees of its sums and its weighted sum (ascending keys) are those of attn_ref_kernel.
// Measured (B200, 12 heads of 128 on 2; a block per row and this): 100 rows behind 300 299 -> 77 us, behind 2,000 1,616 -> 345; 8
// requests of 6 rows behind 2,000 923 -> 382.
#define ROWS_PER_WARP 4
#define ROWS_PER_BLOCK 16

struct AttnRowsArgs {
    const float* q;
    int q_stride;
    float* out;
    const float *k_cache, *v_cache;
    const int *block_tables, *tok_seq, *positions, *q_start;
    int N, S, from;  // requests of fewer than `from` rows are left to attn_ref_kernel
    int nh, nkv, hd, page_size, max_blocks, num_pages;
    float scale;
    int* status;
};

__global__ void __launch_bounds__(128) attn_rows_kernel(const AttnRowsArgs a) {
    extern __shared__ __align__(16) float shared[];
    const int hd = a.hd, ld = hd + 4, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* k_s = shared;                      // [CH][ld]
    float* v_s = k_s + CH * ld;               // [CH][hd]
    float* q_s = v_s + CH * hd;               // [ROWS_PER_BLOCK][hd]
    float* p_s = q_s + ROWS_PER_BLOCK * hd;   // [4 warps][CH][ROWS_PER_WARP]
    int* slot_s = (int*)(p_s + ROWS_PER_BLOCK * CH);  // [2][CH]
    __shared__ int tile_s[3];  // request, first row, rows
    const int h = blockIdx.y, kvh = h / (a.nh / a.nkv);
    for (int r = blockIdx.x * ROWS_PER_BLOCK; r < min(a.N, ((int)blockIdx.x + 1) * ROWS_PER_BLOCK); ++r)
        if (a.tok_seq[r] < 0)  // padding rows, which belong to no request: zeros
            for (int d = threadIdx.x; d < hd; d += 128) a.out[((size_t)r * a.nh + h) * hd + d] = 0.f;
    if (warp == 0) {
        const RowTile tile = find_row_tile(blockIdx.x, true, a.q_start, a.tok_seq, a.S, 1, ROWS_PER_BLOCK, a.from);
        if (lane == 0) {
            tile_s[0] = tile.seq;
            tile_s[1] = tile.row0;
            tile_s[2] = tile.rows;
        }
    }
    __syncthreads();
    const int seq = tile_s[0], row0 = tile_s[1], rows = tile_s[2];
    if (seq < 0) return;
    for (int e = threadIdx.x; e < ROWS_PER_BLOCK * hd; e += 128)
        q_s[e] = e < rows * hd ? a.q[(size_t)(row0 + e / hd) * a.q_stride + (size_t)h * hd + e % hd] : 0.f;
    float* p_w = p_s + warp * CH * ROWS_PER_WARP;

    int ends[ROWS_PER_WARP];  // how many keys this warp's rows see (0: no row)
#pragma unroll
    for (int i = 0; i < ROWS_PER_WARP; ++i) {
        const int r = warp * ROWS_PER_WARP + i;
        ends[i] = r < rows ? a.positions[row0 + r] + 1 : 0;
    }
    int longest = 0;
    for (int r = 0; r < rows; ++r) longest = max(longest, a.positions[row0 + r] + 1);
    const int* table = a.block_tables + (size_t)seq * a.max_blocks;
    const int chunks = (longest + CH - 1) / CH;

    auto find_slots = [&](int c) {  // of chunk c's keys, one a thread
        const int j = c * CH + threadIdx.x;
        int slot = -1;
        if (j < longest) {
            const int blk = j / a.page_size;
            const int page = blk < a.max_blocks ? table[blk] : -1;
            if (page < 0 || page >= a.num_pages)
                cw_report(a.status, CW_ST_PAGE_RANGE, row0, page);
            else
                slot = page * a.page_size + j % a.page_size;
        }
        slot_s[(c & 1) * CH + threadIdx.x] = slot;
    };
    auto fetch = [&](const float* cache, float* to, int row, int c) {
        const int pieces = hd / 4, n = min(CH, longest - c * CH);
        for (int e = threadIdx.x; e < n * pieces; e += 128) {
            const int j = e / pieces, d = (e - j * pieces) * 4, slot = slot_s[(c & 1) * CH + j];
            if (slot >= 0) cp_async16(to + j * row + d, cache + ((size_t)slot * a.nkv + kvh) * hd + d);
        }
        cp_async_commit();
    };

    float m[ROWS_PER_WARP], l[ROWS_PER_WARP], acc[ROWS_PER_WARP][4];
#pragma unroll
    for (int i = 0; i < ROWS_PER_WARP; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[i][x] = 0.f;
    }
    if (chunks > 0) {
        find_slots(0);
        __syncthreads();
        fetch(a.k_cache, k_s, ld, 0);
        fetch(a.v_cache, v_s, hd, 0);
    }
    for (int c = 0; c < chunks; ++c) {
        if (c + 1 < chunks) find_slots(c + 1);
        cp_async_wait<1>();  // chunk c's keys (its values may be on their way)
        __syncthreads();
        // scores: lane = key, four keys a lane
        float s[ROWS_PER_WARP][4];
#pragma unroll
        for (int i = 0; i < ROWS_PER_WARP; ++i)
#pragma unroll
            for (int x = 0; x < 4; ++x) s[i][x] = 0.f;
        const float* qw = q_s + warp * ROWS_PER_WARP * hd;
        const int* slots = slot_s + (c & 1) * CH;
        int slot[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) slot[x] = slots[x * 32 + lane];
        if (c * CH < max(max(ends[0], ends[1]), max(ends[2], ends[3]))) {
#pragma unroll 2
            for (int d = 0; d < hd; d += 4) {
                float4 kv[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) kv[x] = *reinterpret_cast<const float4*>(k_s + (x * 32 + lane) * ld + d);
#pragma unroll
                for (int i = 0; i < ROWS_PER_WARP; ++i) {
                    const float4 qv = *reinterpret_cast<const float4*>(qw + i * hd + d);
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        s[i][x] = fmaf(qv.x, kv[x].x, s[i][x]);
                        s[i][x] = fmaf(qv.y, kv[x].y, s[i][x]);
                        s[i][x] = fmaf(qv.z, kv[x].z, s[i][x]);
                        s[i][x] = fmaf(qv.w, kv[x].w, s[i][x]);
                    }
                }
            }
        }
        __syncthreads();  // the keys have been read
        if (c + 1 < chunks) fetch(a.k_cache, k_s, ld, c + 1);
        else cp_async_commit();
#pragma unroll
        for (int i = 0; i < ROWS_PER_WARP; ++i) {
            const bool live = c * CH < ends[i];
            float top = -INFINITY, p[4], w[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const bool seen = slot[x] >= 0 && c * CH + x * 32 + lane < ends[i];
                s[i][x] = seen ? s[i][x] * a.scale : -INFINITY;
                top = fmaxf(top, s[i][x]);
            }
            const float m_new = fmaxf(m[i], warp_max(top));
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const bool seen = slot[x] >= 0 && c * CH + x * 32 + lane < ends[i];
                p[x] = seen ? expf(s[i][x] - m_new) : 0.f;
                w[x] = warp_sum(p[x]);
            }
            if (live) {
                const float alpha = m[i] == -INFINITY ? 0.f : expf(m[i] - m_new);
                // (the tree over four warps' sums that a block-wide sum of 128 threads takes)
                l[i] = l[i] * alpha + ((w[0] + w[2]) + (w[1] + w[3]));
#pragma unroll
                for (int x = 0; x < 4; ++x) acc[i][x] *= alpha;
                if (m_new != -INFINITY) m[i] = m_new;
            }
#pragma unroll
            for (int x = 0; x < 4; ++x) p_w[(x * 32 + lane) * ROWS_PER_WARP + i] = p[x];
        }
        cp_async_wait<1>();  // chunk c's values (the next keys may be on their way)
        __syncthreads();
        const int d = lane * 4, base = c * CH;
        int common = CH, most = 0;  // keys that all of the warp's rows see, that any of them sees
#pragma unroll
        for (int i = 0; i < ROWS_PER_WARP; ++i) {
            const int n = min(CH, max(ends[i] - base, 0));
            common = min(common, n);
            most = max(most, n);
        }
        if (d < hd) {
            int j = 0;
#pragma unroll 4
            for (; j < common; ++j) {
                if (slots[j] < 0) continue;
                const float4 v = *reinterpret_cast<const float4*>(v_s + j * hd + d);
                const float4 p = *reinterpret_cast<const float4*>(p_w + j * ROWS_PER_WARP);
                const float pr[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
                for (int i = 0; i < ROWS_PER_WARP; ++i) {
                    acc[i][0] = fmaf(pr[i], v.x, acc[i][0]);
                    acc[i][1] = fmaf(pr[i], v.y, acc[i][1]);
                    acc[i][2] = fmaf(pr[i], v.z, acc[i][2]);
                    acc[i][3] = fmaf(pr[i], v.w, acc[i][3]);
                }
            }
            for (; j < most; ++j) {  // (a key is left out for rows that do not see it, whatever its value holds)
                if (slots[j] < 0) continue;
                const float4 v = *reinterpret_cast<const float4*>(v_s + j * hd + d);
#pragma unroll
                for (int i = 0; i < ROWS_PER_WARP; ++i) {
                    if (base + j >= ends[i]) continue;
                    const float pr = p_w[j * ROWS_PER_WARP + i];
                    acc[i][0] = fmaf(pr, v.x, acc[i][0]);
                    acc[i][1] = fmaf(pr, v.y, acc[i][1]);
                    acc[i][2] = fmaf(pr, v.z, acc[i][2]);
                    acc[i][3] = fmaf(pr, v.w, acc[i][3]);
                }
            }
        }
        __syncthreads();  // the values and the chunk's slots have been read
        if (c + 1 < chunks) fetch(a.v_cache, v_s, hd, c + 1);
    }
    cp_async_wait<0>();
#pragma unroll
    for (int i = 0; i < ROWS_PER_WARP; ++i) {
        const int r = warp * ROWS_PER_WARP + i;
        if (r >= rows || lane * 4 >= hd) continue;
        const float inv = l[i] > 0.f ? 1.0f / l[i] : 0.f;
        *reinterpret_cast<float4*>(a.out + ((size_t)(row0 + r) * a.nh + h) * hd + lane * 4) =
            make_float4(acc[i][0] * inv, acc[i][1] * inv, acc[i][2] * inv, acc[i][3] * inv);
    }
}

// cw_attention_ref for the requests of at least `from` rows (and padding rows): float32, no window, heads of up to 128 entries in
// whole 16-byte pieces, all pointers 16-byte aligned (CW_ERR_UNSUPPORTED otherwise).  q_start [S + 1].  tiles: how many tiles of 16 rows
// these requests have (0: not known; padding rows are then among the N rows).
extern "C" int cw_attention_rows(const void* q, int q_stride, void* out, const void* k_cache, const void* v_cache,
                                 const int* block_tables, const int* tok_seq, const int* positions, const int* q_start, int S, int from,
                                 int tiles, int N, int nh, int nkv, int hd, int page_size, int max_blocks, int num_pages, float scale, int* status,
                                 cudaStream_t stream) {
    if (N == 0) return CW_OK;
    if (N < 0 || S < 0 || q_start == nullptr || nh <= 0 || nkv <= 0 || nh % nkv != 0 || hd <= 0 || page_size <= 0 || max_blocks <= 0) return CW_ERR_BAD_SIZE;
    if (hd > 128 || hd % 4 || q_stride % 4 || nh > 65535 || ((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_cache | (uintptr_t)v_cache) % 16)
        return CW_ERR_UNSUPPORTED;
    auto bytes = [](int size) { return sizeof(float) * (size_t)(CH * (2 * size + 4) + ROWS_PER_BLOCK * (size + CH)) + sizeof(int) * 2 * CH; };
    const size_t smem = bytes(hd);
    const cudaError_t err = cudaFuncSetAttribute(attn_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes(128));
    if (err != cudaSuccess) return (int)err;
    const AttnRowsArgs args = {(const float*)q, q_stride, (float*)out, (const float*)k_cache, (const float*)v_cache, block_tables, tok_seq,
                               positions, q_start, N, S, from, nh, nkv, hd, page_size, max_blocks, num_pages, scale, status};
    attn_rows_kernel<<<dim3(tiles > 0 ? tiles : (N + ROWS_PER_BLOCK - 1) / ROWS_PER_BLOCK + S, nh), 128, smem, stream>>>(args);
    return CW_LAUNCH_CHECK();
}

// below > 0 (with q_start [S + 1]): only the requests of fewer rows than that; rows: how many they have (0: not known).
extern "C" int cw_attention_ref(const void* q, int q_stride, void* out, const void* k_cache,
                                const void* v_cache, const int* block_tables, const int* tok_seq,
                                const int* positions, int N, int nh, int nkv, int hd,
                                int page_size, int max_blocks, int num_pages, float scale,
                                int window, const int* q_start, int S, int below, int rows, int dtype, int* status,
                                cudaStream_t stream) {
    if (N == 0) return CW_OK;
    if (N < 0 || nh <= 0 || nkv <= 0 || nh % nkv != 0 || hd <= 0 || page_size <= 0 || max_blocks <= 0)
        return CW_ERR_BAD_SIZE;
    if (below > 0 && (q_start == nullptr || S < 0)) return CW_ERR_BAD_SIZE;
    if (hd > 2 * CH || nh > 65535) return CW_ERR_UNSUPPORTED;
    dim3 grid(below > 0 && rows > 0 ? rows : N, nh);
    const size_t smem = (size_t)hd * sizeof(float);
    if (dtype == 0)
        attn_ref_kernel<float><<<grid, CH, smem, stream>>>(
            (const float*)q, q_stride, (float*)out, (const float*)k_cache, (const float*)v_cache,
            block_tables, tok_seq, positions, nh, nkv, hd, page_size, max_blocks, num_pages, scale,
            window, q_start, S, below, status);
    else if (dtype == 1)
        attn_ref_kernel<bf16><<<grid, CH, smem, stream>>>(
            (const bf16*)q, q_stride, (bf16*)out, (const bf16*)k_cache, (const bf16*)v_cache,
            block_tables, tok_seq, positions, nh, nkv, hd, page_size, max_blocks, num_pages, scale,
            window, q_start, S, below, status);
    else
        return CW_ERR_BAD_DTYPE;
    return CW_LAUNCH_CHECK();
}

CW_TRACE_TU(attention_ref)
