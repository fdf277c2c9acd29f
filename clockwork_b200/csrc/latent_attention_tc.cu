// Attention over a cached latent (latent_attention.cu) for prompt portions on the 5th-generation tensor cores.
//
// The rows of a request's (token, head) pairs, consecutive in qa, are the 128 lanes of tensor memory.  The sums of 128 rows of 512
// latents would fill it (512 columns of float32), so a CTA keeps 256 columns of them and there are as many CTAs per row tile as
// the latent has pieces of 256 columns, each forming the scores for itself (576 multiply-adds per row and key, beside 2 x 256 of
// its own sums: half again as many as without the repetition, which costs less than handing scores from SM to SM).
//   S  = Q C^T         Q [128][rank + rot] stays on chip: of wide rows the first 256 columns in tensor memory, as the A operand of
//                      their MMAs, the rest in shared memory; the cached rows of 64 keys come page by page by TMA, two stages or more
//   P  = 2^(S c - m)   four warps, a thread per row: float32 statistics, the maximum moved lazily as in attention_prefill_tc.cu;
//                      the weights as two bfloat16 halves (P = hi + lo: 16 bits of mantissa) over S in tensor memory
//   O += hi C + lo C   A in tensor memory, the same cached tile as it lies (MN-major B)
// S of the next tile is formed while the warps work on this one, before this one's sums if its keys have come, else behind.  Rows of the last tile behind the context are set to zero in
// shared memory, whatever the cache holds there.  CTAs of a request's last rows, which see the most keys, come first.
// What bounds it: the latency of a tile's chain of loads, scores (36 MMAs of 128 x 64 x 16 for 576 columns), weights and sums, with the two
// stages that 147 KB hold: the tensor pipe was 28 % busy, the issue slots 15 %, L2 7 % at 261 us.  With tiles of 32 keys it ran 332 us, with all of Q in shared memory as well (two stages of 32 keys) 446.
// Measured (B200, 2,048 tokens of 16 heads over 512 + 64): the mma.sync kernel it replaced for uncut keys 494 us, this one 199 us (261 before the issuing threads were elected).
#include "latent_attention.cuh"
#include "tc_attention.cuh"

#define LC_ROWS 128
#define LC_KEYS 64
#define LC_COLS 256                          // latent columns of a CTA
#define LC_THREADS 192                       // producer warp, MMA warp, four softmax warps
#define LC_MAX_STAGES 4
#define LC_Q_BLOCK (LC_ROWS * 128)           // 64 columns of all rows
#define LC_K_BLOCK (LC_KEYS * 128)
#define LC_LAZY 8.0f                         // log2 of how far a tile's maximum may exceed the one in use
#define LC_SMEM (226 * 1024)
#define LC_HELD 4                            // blocks of Q in tensor memory, at most
#define LC_S_COL LC_COLS                     // tensor memory: O, two S buffers, Q
#define LC_Q_COL (LC_S_COL + 2 * LC_KEYS)

// Whether a phase is complete, without waiting for it (mbarrier.try_wait may hold the thread for as long as it likes, here on a
// barrier that only completes when this thread goes on).
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

struct LatentTc {
    LatentArgs a;
    int blocks;      // of 64 columns in a row of rank + rot
    int held;        // how many of them, the first ones, Q keeps in tensor memory
    int stages, splits;
    int box, boxes;  // rows of a TMA box (within a page), boxes of a tile
};

__global__ void __launch_bounds__(LC_THREADS, 1)
latent_attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_c, const LatentTc p) {
    extern __shared__ uint8_t lc_smem[];
    const LatentArgs& a = p.a;
    uint8_t* q_s = (uint8_t*)(((uintptr_t)lc_smem + 1023) & ~(uintptr_t)1023);
    uint8_t* k_s = q_s + (p.blocks - p.held) * LC_Q_BLOCK;
    const int stage_bytes = p.blocks * LC_K_BLOCK;
    uint64_t* bars = (uint64_t*)(k_s + p.stages * stage_bytes);
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * LC_MAX_STAGES, q_full = empty0 + 8 * LC_MAX_STAGES, aux = q_full + 8;
    const uint32_t s_full0 = aux + 8, p_full0 = s_full0 + 16, o_done0 = p_full0 + 16, q_held = o_done0 + 16;
    uint32_t* tmem_slot = (uint32_t*)(bars + 2 * LC_MAX_STAGES + 9);
    volatile int* give_up = (volatile int*)(tmem_slot + 1);
    int* tile_s = (int*)(tmem_slot + 2);  // request, first row, rows
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, H = a.H, rank = a.rank;
    const int split = blockIdx.x % p.splits, block = blockIdx.x / p.splits;
    const long long total_rows = (long long)a.N * H;

    pdl_wait();
    if (split == 0) {  // rows of no request (padding of a fixed-shape step) come out as zeros
        const long long first = (long long)block * LC_ROWS, last = min(total_rows, first + LC_ROWS);
        for (long long t = first / H; t * H < last; ++t)
            if (a.tok_seq[t] < 0)
                for (long long i = max(first, t * H) * rank + tid; i < min(last, (t + 1) * H) * rank; i += LC_THREADS) a.out[i] = __float2bfloat16_rn(0.f);
    }
    if (warp == 0) {
        const RowTile tile = find_row_tile(block, true, a.q_start, a.tok_seq, a.S, H, LC_ROWS);
        if (lane == 0) {
            tile_s[0] = tile.seq;
            tile_s[1] = tile.row0;
            tile_s[2] = tile.rows;
            for (int s = 0; s < LC_MAX_STAGES; ++s) {
                mbar_init(full0 + 8 * s, 1);
                mbar_init(empty0 + 8 * s, 1);
            }
            mbar_init(q_full, 1);
            mbar_init(aux, 1);
            for (int b = 0; b < 2; ++b) {
                mbar_init(s_full0 + 8 * b, 1);
                mbar_init(p_full0 + 8 * b, 4);
                mbar_init(o_done0 + 8 * b, 1);
            }
            mbar_init(q_held, 4);
            *give_up = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
    }
    __syncthreads();
    const int seq = tile_s[0], row0 = tile_s[1], rows = tile_s[2];
    if (seq < 0) return;
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    pdl_release();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot, s_col = tmem + LC_S_COL;
    const int tok0 = row0 / H, head0 = row0 - tok0 * H, p0 = a.positions[tok0];
    const int kv_end = p0 + (head0 + rows - 1) / H + 1, tiles = (kv_end + LC_KEYS - 1) / LC_KEYS;
    const int cols = min(LC_COLS, rank - split * LC_COLS);

    if (warp == 0) {
        // ---- producer warp: a lane looks up the row of a box, one issues the copies --------------------------------------------
        if (lane == 0) {
            mbar_expect_tx(q_full, (p.blocks - p.held) * LC_Q_BLOCK);
            for (int b = p.held; b < p.blocks; ++b) tma_load_2d(smem_u32(q_s + (b - p.held) * LC_Q_BLOCK), &map_q, b * 64, row0, q_full);
        }
        const int* table = a.block_tables + (size_t)seq * a.max_blocks;
        auto find_row = [&](int t) {  // lane x: the cache row where box x of tile t begins
            const int j = t * LC_KEYS + lane * p.box, blk = j / a.page_size;
            if (lane >= p.boxes || j >= kv_end) return 0;
            int page = blk < a.max_blocks ? table[blk] : -1;
            if (page < 0 || page >= a.num_pages) {
                cw_report(a.status, CW_ST_PAGE_RANGE, tok0, page);
                page = 0;
            }
            return page * a.page_size + j % a.page_size;
        };
        int next_row = find_row(0);
        bool ok = true;
        int t = 0;
        for (; t < tiles; ++t) {
            const int s = t % p.stages, valid = min(LC_KEYS, kv_end - t * LC_KEYS), live = (valid + p.box - 1) / p.box;
            const int this_row = next_row;
            if (t + 1 < tiles) next_row = find_row(t + 1);  // (looked up while this tile's stage empties)
            ok = mbar_wait(empty0 + 8 * s, ((t / p.stages) & 1) ^ 1, give_up);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            uint8_t* stage = k_s + s * stage_bytes;
            const uint32_t bar = valid == LC_KEYS ? full0 + 8 * s : aux;
            if (lane == 0) mbar_expect_tx(bar, live * p.box * 128 * p.blocks);
            __syncwarp();
            // (one lane issues them: a lane each for 36 boxes took the prompt below 205 us, so 199)
            for (int x = 0; x < live; ++x) {
                const int from = __shfl_sync(0xffffffffu, this_row, x);
                if (elect_one())
                    for (int b = 0; b < p.blocks; ++b) tma_load_2d(smem_u32(stage + b * LC_K_BLOCK + x * p.box * 128), &map_c, b * 64, from, bar);
            }
            if (valid < LC_KEYS) {  // (the last tile only) rows behind the context: zeros
                ok = mbar_wait(aux, 0, give_up);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                const int pieces = (LC_KEYS - valid) * 8;
                for (int e = lane; e < pieces * p.blocks; e += 32) {
                    const int b = e / pieces, i = e - b * pieces;
                    *(uint4*)(stage + b * LC_K_BLOCK + valid * 128 + i * 16) = make_uint4(0, 0, 0, 0);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(full0 + 8 * s) : "memory");
            }
        }
        if (*give_up && lane == 0) {  // the copies in flight, bounded
            const long long t0 = clock64();
            while (!mbar_try_wait(q_full, 0) && clock64() - t0 < WAIT_CYCLES) {
            }
            for (int k = max(0, t - p.stages); k < t; ++k) {
                const long long t1 = clock64();
                while (!mbar_try_wait(full0 + 8 * (k % p.stages), (k / p.stages) & 1) && clock64() - t1 < WAIT_CYCLES) {
                }
            }
            if (t < tiles && kv_end - t * LC_KEYS < LC_KEYS) {
                const long long t1 = clock64();
                while (!mbar_try_wait(aux, 0) && clock64() - t1 < WAIT_CYCLES) {
                }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            // ---- MMA issuer ---------------------------------------------------------------------------------------
            constexpr uint32_t idesc_s = instr_desc(LC_ROWS, LC_KEYS);
            const uint32_t idesc_o = instr_desc(LC_ROWS, cols) | (1u << 16);  // B is MN-major
            const int ksteps = (rank + a.rot) / 16;
            bool ok = mbar_wait(q_full, 0, give_up) && mbar_wait(q_held, 0, give_up);
            tc_fence_after();
            auto scores = [&](int t) {
                const int s = t % p.stages;
                if (!mbar_wait(full0 + 8 * s, (t / p.stages) & 1, give_up)) return false;
                tc_fence_after();
                const uint32_t q_addr = smem_u32(q_s), k_addr = smem_u32(k_s + s * stage_bytes);
                const uint32_t to = s_col + (t & 1) * LC_KEYS;
                int k = 0;
                for (; k < 4 * p.held; ++k)
                    umma_bf16_a_tmem(to, tmem + LC_Q_COL + 8 * k, smem_desc_sw128(k_addr + (k >> 2) * LC_K_BLOCK) + 2 * (k & 3), idesc_s, k > 0 ? 1u : 0u);
                for (; k < ksteps; ++k)
                    umma_bf16(to, smem_desc_sw128(q_addr + ((k >> 2) - p.held) * LC_Q_BLOCK) + 2 * (k & 3),
                              smem_desc_sw128(k_addr + (k >> 2) * LC_K_BLOCK) + 2 * (k & 3), idesc_s, k > 0 ? 1u : 0u);
                umma_commit(s_full0 + 8 * (t & 1));
                return true;
            };
            if (ok) ok = scores(0);
            int formed = 1;  // tiles whose scores have been issued
            for (int t = 0; t < tiles && ok; ++t) {
                // the next tile's scores go first if its keys are there (its buffer's weights were read by the sums of tile t - 1,
                // issued before); otherwise this tile's sums, which free the stage that the loads wait for
                const long long t0 = clock64();
                while (!mbar_test(p_full0 + 8 * (t & 1), (t >> 1) & 1)) {
                    if (formed == t + 1 && formed < tiles && mbar_test(full0 + 8 * (formed % p.stages), (formed / p.stages) & 1)) ok = scores(formed++);
                    if (*give_up || clock64() - t0 > WAIT_CYCLES) {
                        *give_up = 1;
                        ok = false;
                    }
                    if (!ok) break;
                }
                if (!ok) break;
                tc_fence_after();
                const uint32_t v_addr = smem_u32(k_s + (t % p.stages) * stage_bytes + split * (LC_COLS / 64) * LC_K_BLOCK);
#pragma unroll
                for (int kk = 0; kk < LC_KEYS / 16; ++kk)
#pragma unroll
                    for (int part = 0; part < 2; ++part)  // hi, lo
                        umma_bf16_a_tmem(tmem, s_col + (t & 1) * LC_KEYS + part * (LC_KEYS / 2) + kk * 8,
                                         smem_desc_mn_sw128(v_addr + kk * 2048, LC_K_BLOCK, 1024), idesc_o, t > 0 || kk > 0 || part > 0 ? 1u : 0u);
                umma_commit(empty0 + 8 * (t % p.stages));
                umma_commit(o_done0 + 8 * (t & 1));
                if (formed == t + 1 && formed < tiles) ok = scores(formed++);
            }
        }
    } else {
        // ---- softmax: a thread per row ---------------------------------------------------------------------------
        const int quarter = warp & 3, row = quarter * 32 + lane;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        const int pos = p0 + (head0 + row) / H;  // (rows past the tile's end are computed and not stored)
        const float scale2 = a.scale * 1.4426950408889634f;
        {  // the first blocks of the row's Q: 32 words, 64 columns, at a time
            const uint4* from = (const uint4*)(a.qa + (size_t)(row0 + min(row, rows - 1)) * (rank + a.rot));
            for (int b = 0; b < p.held; ++b) {
                float w[32];
#pragma unroll
                for (int i = 0; i < 8; ++i) *(uint4*)&w[4 * i] = from[8 * b + i];
                tmem_st16(tmem + lanes + LC_Q_COL + 32 * b, w);
                tmem_st16(tmem + lanes + LC_Q_COL + 32 * b + 16, w + 16);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(q_held) : "memory");
        }
        float m = -INFINITY, l = 0.f;  // the maximum that the row's exponentials are taken against (base 2), their sum
        bool ok = true;
        for (int t = 0; t < tiles; ++t) {
            ok = mbar_wait(s_full0 + 8 * (t & 1), (t >> 1) & 1, give_up);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            if (t >= 2) {  // the sums of tile t - 2 (their barrier's next phase, those of tile t, needs this warp's weights)
                ok = mbar_wait(o_done0 + 8 * (t & 1), ((t >> 1) - 1) & 1, give_up);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
            }
            tc_fence_after();
            const uint32_t s_addr = s_col + (t & 1) * LC_KEYS + lanes;
            float v[LC_KEYS];
            tmem_ld32(s_addr, v);
            tmem_ld32(s_addr + 32, v + 32);
            if (t * LC_KEYS + LC_KEYS - 1 > p0) {
#pragma unroll
                for (int i = 0; i < LC_KEYS; ++i) v[i] = t * LC_KEYS + i <= pos ? v[i] : -INFINITY;
            }
            float mx[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
            for (int i = 4; i < LC_KEYS; ++i) mx[i & 3] = fmaxf(mx[i & 3], v[i]);
            const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale2;
            float alpha = 1.f;
            bool moved = false;
            if (top > m + LC_LAZY) {  // (never for a tile without a visible key)
                if (m != -INFINITY) {
                    alpha = ex2(m - top);
                    moved = true;
                }
                m = top;
            }
            const float base = m == -INFINITY ? 0.f : m;
            if (__any_sync(0xffffffffu, moved)) {  // O so far times alpha, at rest once the sums of the tile before are done
                ok = mbar_wait(o_done0 + 8 * ((t - 1) & 1), ((t - 1) >> 1) & 1, give_up);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                rescale_o<LC_COLS>(tmem + lanes, alpha);
            }
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < LC_KEYS; ++i) v[i] = ex2(fmaf(v[i], scale2, -base));
#pragma unroll
            for (int i = 0; i < LC_KEYS; ++i) sum[i & 3] += v[i];
            l = l * alpha + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float hi[16], low[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float x = v[32 * half + 2 * i], y = v[32 * half + 2 * i + 1];
                    const uint32_t w = pack2(x, y);
                    hi[i] = __uint_as_float(w);
                    low[i] = __uint_as_float(pack2(x - __uint_as_float(w << 16), y - __uint_as_float(w & 0xffff0000u)));
                }
                tmem_st16(s_addr + 16 * half, hi);
                tmem_st16(s_addr + LC_KEYS / 2 + 16 * half, low);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(p_full0 + 8 * (t & 1)) : "memory");
        }
        for (int t = max(0, tiles - 2); t < tiles && ok; ++t) {
            ok = mbar_wait(o_done0 + 8 * (t & 1), (t >> 1) & 1, give_up);
            ok = __all_sync(0xffffffffu, ok);
        }
        if (ok) {
            tc_fence_after();
            // the sink joins the denominator only
            const float sk = a.sink != nullptr ? a.sink[(head0 + row) % H] * 1.4426950408889634f : -INFINITY;
            const float top = fmaxf(m, sk), keep = m == -INFINITY ? 0.f : exp2f(m - top);
            const float denom = l * keep + (sk == -INFINITY ? 0.f : exp2f(sk - top));
            const float inv = denom > 0.f ? keep / denom : 0.f;
            bf16* out = a.out + (size_t)(row0 + row) * rank + split * LC_COLS;
            for (int c = 0; c < cols; c += 16) {
                float v[16];
                tmem_ld16(tmem + lanes + c, v);
                if (row < rows) {
                    uint4 w[2];
                    w[0] = make_uint4(pack2(v[0] * inv, v[1] * inv), pack2(v[2] * inv, v[3] * inv), pack2(v[4] * inv, v[5] * inv), pack2(v[6] * inv, v[7] * inv));
                    w[1] = make_uint4(pack2(v[8] * inv, v[9] * inv), pack2(v[10] * inv, v[11] * inv), pack2(v[12] * inv, v[13] * inv), pack2(v[14] * inv, v[15] * inv));
                    *(uint4*)(out + c) = w[0];
                    *(uint4*)(out + c + 8) = w[1];
                }
            }
        }
    }
    __syncwarp();
    if (*give_up && tid == 0) cw_report(a.status, CW_ST_WAIT_TIMEOUT, blockIdx.x, -3);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

// ---- host side ---------------------------------------------------------------------------------------------------
static int lc_map(CUtensorMap* map, const void* ptr, long long rows, int columns, int box_rows) {
    const cuuint64_t dims[2] = {(cuuint64_t)columns, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)columns * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elem,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : -1;
}

// Q keeps its first blocks in tensor memory where all of it in shared memory would leave less than two stages.
static int lc_held(int blocks) { return blocks > 6 ? LC_HELD : 0; }
static int lc_stages(int blocks) {
    const int room = (LC_SMEM - 2048 - (blocks - lc_held(blocks)) * LC_Q_BLOCK) / (blocks * LC_K_BLOCK);
    return room > LC_MAX_STAGES ? LC_MAX_STAGES : room;
}

// Rows of whole steps of 16 columns; pages of 8, 16 or 32 tokens or a multiple of 64 (a box of keys lies in one page).
bool latent_tc_takes(const LatentArgs& a) {
    const int D = a.rank + a.rot, blocks = (D + 63) / 64;
    if (!(a.scale > 0.f)) return false;  // (the maximum is taken before the factor)
    if (D % 16 || a.rank % 16 || a.rank > 2 * LC_COLS || lc_stages(blocks) < 2) return false;
    if (a.page_size != 8 && a.page_size != 16 && a.page_size != 32 && a.page_size % LC_KEYS) return false;
    return ((uintptr_t)a.qa | (uintptr_t)a.cache | (uintptr_t)a.out) % 16 == 0 && (long long)a.num_pages * a.page_size <= 0x7fffffffLL;
}

int latent_tc_run(const LatentArgs& a, cudaStream_t stream) {
    if (load_encode() != 0) return CW_ERR_UNSUPPORTED;
    const int D = a.rank + a.rot;
    LatentTc p = {a, (D + 63) / 64, lc_held((D + 63) / 64), lc_stages((D + 63) / 64), (a.rank + LC_COLS - 1) / LC_COLS, a.page_size < LC_KEYS ? a.page_size : LC_KEYS, 0};
    p.boxes = LC_KEYS / p.box;
    const long long rows = (long long)a.N * a.H, blocks = ((rows + LC_ROWS - 1) / LC_ROWS + a.S) * p.splits;
    if (blocks > 0x7fffffffLL) return CW_ERR_UNSUPPORTED;
    CUtensorMap q, c;
    if (lc_map(&q, a.qa, rows, D, LC_ROWS) != 0 || lc_map(&c, a.cache, (long long)a.num_pages * a.page_size, D, p.box) != 0) return CW_ERR_UNSUPPORTED;
    const size_t smem = (size_t)(p.blocks - p.held) * LC_Q_BLOCK + (size_t)p.blocks * p.stages * LC_K_BLOCK + 2048;
    const cudaError_t e = cudaFuncSetAttribute(latent_attention_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LC_SMEM);
    if (e != cudaSuccess) return (int)e;
    return cw_launch(latent_attention_tc_kernel, dim3((unsigned)blocks), dim3(LC_THREADS), smem, stream, 1, q, c, p);
}

CW_TRACE_TU(latent_attention_tc)
