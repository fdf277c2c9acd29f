// Windowed attention (window_attention.cu) for prompt portions on the 5th-generation tensor cores: softmax weights over a sliding
// window (with kept first positions) or a block of positions, keys and values in one cache row.
//
// The 128 lanes of tensor memory are 128 / per consecutive tokens of one request times the `per` query heads of a key/value head,
// so that a key is read once for all of them.  Keys in tiles of 64, the key's and the value's columns of a row fetched page by page
// by TMA into rings of their own (a key's stage is free when its scores are formed, a value's when its sums are):
//   S  = Q K^T         both K-major in shared memory
//   P  = 2^(S c - m)   four warps, a thread per row: float32 statistics, the maximum moved lazily as in attention_prefill_tc.cu;
//                      the weights as two bfloat16 halves (P = hi + lo: 16 bits of mantissa) over S in tensor memory
//   O += hi V + lo V   A in tensor memory, the values as they lie (MN-major B)
// Two CTAs share an SM, one's loads and exponentials beside the other's products.  A tile's pages that no row sees (given back,
// or between the kept positions and the window) are not read; rows of a value tile that were not fetched, or lie behind the
// context, are set to zero in shared memory.  Switches that change a score by more than a factor and an addend per row (mixed
// heads, sigmoid weights, a cap, a distance bias, pooled blocks) stay with the mma.sync kernel, and so do the steps that it is
// faster for (window_tc_pays).
// What bounds it: the latency of a tile's chain (scores, 64 exponentials and their split in halves a thread, sums): the issue slots are 23 %
// busy, the tensor pipe 17 % (33 % on the SM with the longest rows), L2 8 %.
// Measured (B200, prompts of 1,500, 421 and 127 tokens, 16 heads of 128 on 4, window 1,024): mma.sync kernel and merge 223 us, this
// one 55 us.
#include "tc_attention.cuh"
#include "window_attention.cuh"

#define WC_ROWS 128
#define WC_KEYS 64
#define WC_THREADS 192                // producer warp, MMA warp, four softmax warps
#define WC_MAX_STAGES 4
#define WC_Q_BLOCK (WC_ROWS * 128)    // 64 columns of all rows
#define WC_BLOCK (WC_KEYS * 128)      // 64 columns of a tile's keys
#define WC_MAX_DIM 128
#define WC_LAZY 8.0f                  // log2 of how far a tile's maximum may exceed the one in use
#define WC_TMEM 256                   // O in columns 0 .. 127, two S buffers
#define WC_SMEM (112 * 1024)          // two CTAs to an SM
#define WC_MIN_TILES 64               // row tiles from which keys cut in more than WC_MAX_PARTS parts run here as well
#define WC_AT_ONCE 296                // CTAs that run side by side on 148 SMs

struct WindowTc {
    WindowAttentionArgs a;
    const int* q_start;
    int S, N, per, tokens;  // heads of a key/value head, tokens of a row tile
    int kb, vb, stages;     // blocks of 64 columns of a key and of a value
    int box, boxes;         // rows of a TMA box (within a page), boxes of a tile
};

__global__ void __launch_bounds__(WC_THREADS, 2)
window_attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_c, const WindowTc p) {
    extern __shared__ uint8_t wc_smem[];
    const WindowAttentionArgs& a = p.a;
    uint8_t* q_s = (uint8_t*)(((uintptr_t)wc_smem + 1023) & ~(uintptr_t)1023);
    uint8_t* k_s = q_s + p.kb * WC_Q_BLOCK;
    uint8_t* v_s = k_s + p.stages * p.kb * WC_BLOCK;
    uint64_t* bars = (uint64_t*)(v_s + p.stages * p.vb * WC_BLOCK);
    const uint32_t k_full = smem_u32(bars), k_empty = k_full + 8 * WC_MAX_STAGES, v_full = k_empty + 8 * WC_MAX_STAGES;
    const uint32_t v_empty = v_full + 8 * WC_MAX_STAGES, q_full = v_empty + 8 * WC_MAX_STAGES, aux = q_full + 8;
    const uint32_t s_full = aux + 8, p_full = s_full + 16, o_done0 = p_full + 16;
    uint32_t* tmem_slot = (uint32_t*)(bars + 4 * WC_MAX_STAGES + 8);
    volatile int* give_up = (volatile int*)(tmem_slot + 1);
    int* tile_s = (int*)(tmem_slot + 2);  // request, first token, tokens
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = blockIdx.x % a.G, block = blockIdx.x / a.G, per = p.per, dv = a.dv, HV = a.H * dv;
    bf16* const all_out = (bf16*)a.out;

    // rows of no request (padding of a fixed-shape step) come out as zeros: every block has its share of the tokens
    for (int n = block * p.tokens; n < min(p.N, (block + 1) * p.tokens); ++n)
        if (a.tok_seq[n] < 0)
            for (int i = tid; i < per * dv; i += WC_THREADS) all_out[(size_t)n * HV + (size_t)g * per * dv + i] = __float2bfloat16_rn(0.f);
    if (warp == 0) {
        const RowTile tile = find_row_tile(block, true, p.q_start, a.tok_seq, p.S, 1, p.tokens);
        if (lane == 0) {
            tile_s[0] = tile.seq;
            tile_s[1] = tile.row0;
            tile_s[2] = tile.rows;
            for (int s = 0; s < WC_MAX_STAGES; ++s) {
                mbar_init(k_full + 8 * s, 1);
                mbar_init(k_empty + 8 * s, 1);
                mbar_init(v_full + 8 * s, 1);
                mbar_init(v_empty + 8 * s, 1);
            }
            mbar_init(q_full, 1);
            mbar_init(aux, 1);
            for (int b = 0; b < 2; ++b) {
                mbar_init(s_full + 8 * b, 1);
                mbar_init(p_full + 8 * b, 4);
                mbar_init(o_done0 + 8 * b, 1);
            }
            *give_up = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
    }
    __syncthreads();
    const int seq = tile_s[0], n0 = tile_s[1], tokens = tile_s[2];
    if (seq < 0) return;
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), WC_TMEM);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot, s_col = tmem + WC_MAX_DIM;
    // the keys: those of the kept positions before the window's first tile, then from that tile to the last token
    const int p0 = a.positions[n0], kv_end = p0 + tokens;
    auto first_of = [&](int pos) { return a.blocked ? pos - pos % a.window : max(0, pos - a.window + 1); };
    const int start = first_of(p0), t_first = start / WC_KEYS, kept = min((a.keep + WC_KEYS - 1) / WC_KEYS, t_first);
    const int tiles = kept + (kv_end + WC_KEYS - 1) / WC_KEYS - t_first;
    auto key_of = [&](int t) { return (t < kept ? t : t_first + t - kept) * WC_KEYS; };

    if (warp == 0) {
        // ---- producer warp: a lane per box of rows and block of columns --------------------------------------------
        const int row_width = a.voff + dv;
        if (lane == 0) {
            mbar_expect_tx(q_full, p.kb * WC_Q_BLOCK);
            for (int b = 0; b < p.kb; ++b)
                asm volatile(
                    "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                    ::"r"(smem_u32(q_s + b * WC_Q_BLOCK)), "l"(&map_q), "r"(q_full), "r"(b * 64), "r"(g * per), "r"(n0)
                    : "memory");
        }
        const int* table = a.block_tables + (size_t)seq * a.max_blocks;
        auto find_row = [&](int t) {  // lane x: the cache row where box x of tile t begins (-1: no row of the tile sees it)
            const int j = key_of(t) + lane * p.box, blk = j / a.page_size;
            if (lane >= p.boxes || j >= kv_end || (j + p.box <= start && j >= a.keep)) return -1;
            int page = blk < a.max_blocks ? table[blk] : -1;
            if (page < 0 || page >= a.num_pages) {
                if (g == 0) cw_report(a.status, CW_ST_PAGE_RANGE, n0, page);
                page = 0;
            }
            return page * a.page_size + j % a.page_size;
        };
        int next_row = find_row(0), partial = 0, t = 0;
        bool ok = true;
        auto copy = [&](uint8_t* stage, int blocks, int column, int row, uint32_t bar, unsigned live) {
            for (int e0 = 0; e0 < p.boxes * blocks; e0 += 32) {
                const int e = e0 + lane, x = e / blocks, b = e - x * blocks;
                const int from = __shfl_sync(0xffffffffu, row, x & 31);
                if (e < p.boxes * blocks && (live >> x & 1)) tma_load_2d(smem_u32(stage + b * WC_BLOCK + x * p.box * 128), &map_c, column + b * 64, from, bar);
            }
        };
        for (; t < tiles; ++t) {
            const int s = t % p.stages, row = next_row, valid = min(WC_KEYS, kv_end - key_of(t));
            const unsigned live = __ballot_sync(0xffffffffu, row >= 0);
            const int bytes = __popc(live) * p.box * 128;
            if (t + 1 < tiles) next_row = find_row(t + 1);  // (looked up while this tile's stages empty)
            const uint32_t phase = ((t / p.stages) & 1) ^ 1;
            ok = mbar_wait(k_empty + 8 * s, phase, give_up);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            if (lane == 0) mbar_expect_tx(k_full + 8 * s, bytes * p.kb);
            __syncwarp();
            copy(k_s + s * p.kb * WC_BLOCK, p.kb, g * row_width, row, k_full + 8 * s, live);
            ok = mbar_wait(v_empty + 8 * s, phase, give_up);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            uint8_t* stage = v_s + s * p.vb * WC_BLOCK;
            const bool whole = valid == WC_KEYS && __popc(live) == p.boxes;
            const uint32_t bar = whole ? v_full + 8 * s : aux;
            if (lane == 0) mbar_expect_tx(bar, bytes * p.vb);
            __syncwarp();
            copy(stage, p.vb, g * row_width + a.voff, row, bar, live);
            if (!whole) {  // rows that were not fetched, or lie behind the context: zeros
                ok = mbar_wait(aux, partial & 1, give_up);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                ++partial;
                for (int e = lane; e < WC_KEYS * 8 * p.vb; e += 32) {
                    const int b = e / (WC_KEYS * 8), i = e - b * (WC_KEYS * 8), r = i >> 3;
                    if (r >= valid || !(live >> (r / p.box) & 1)) *(uint4*)(stage + b * WC_BLOCK + i * 16) = make_uint4(0, 0, 0, 0);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(v_full + 8 * s) : "memory");
            }
        }
        if (*give_up && lane == 0) {  // the copies in flight, bounded
            auto settle = [&](uint32_t bar, uint32_t parity) {
                const long long t0 = clock64();
                while (!mbar_try_wait(bar, parity) && clock64() - t0 < WAIT_CYCLES) {
                }
            };
            settle(q_full, 0);
            for (int k = max(0, t - p.stages); k <= min(t, tiles - 1); ++k) {
                settle(k_full + 8 * (k % p.stages), (k / p.stages) & 1);
                settle(v_full + 8 * (k % p.stages), (k / p.stages) & 1);
            }
            settle(aux, partial & 1);
        }
    } else if (warp == 1) {
        if (elect_one()) {
            // ---- MMA issuer ---------------------------------------------------------------------------------------
            constexpr uint32_t idesc_s = instr_desc(WC_ROWS, WC_KEYS);
            const uint32_t idesc_o = instr_desc(WC_ROWS, dv) | (1u << 16);  // B is MN-major
            const int ksteps = a.dk / 16;
            bool ok = mbar_wait(q_full, 0, give_up);
            auto scores = [&](int t) {
                const int s = t % p.stages;
                if (!mbar_wait(k_full + 8 * s, (t / p.stages) & 1, give_up)) return false;
                tc_fence_after();
                const uint32_t q_addr = smem_u32(q_s), k_addr = smem_u32(k_s + s * p.kb * WC_BLOCK);
                for (int k = 0; k < ksteps; ++k)
                    umma_bf16(s_col + (t & 1) * WC_KEYS, smem_desc_sw128(q_addr + (k >> 2) * WC_Q_BLOCK) + 2 * (k & 3),
                              smem_desc_sw128(k_addr + (k >> 2) * WC_BLOCK) + 2 * (k & 3), idesc_s, k > 0 ? 1u : 0u);
                umma_commit(k_empty + 8 * s);
                umma_commit(s_full + 8 * (t & 1));
                return true;
            };
            if (ok) ok = scores(0);
            for (int t = 0; t < tiles && ok; ++t) {
                if (t + 1 < tiles) ok = scores(t + 1);  // (its buffer's weights were read by the sums of tile t - 1, issued before)
                if (!ok) break;
                const int s = t % p.stages;
                ok = mbar_wait(v_full + 8 * s, (t / p.stages) & 1, give_up) && mbar_wait(p_full + 8 * (t & 1), (t >> 1) & 1, give_up);
                if (!ok) break;
                tc_fence_after();
                const uint32_t v_addr = smem_u32(v_s + s * p.vb * WC_BLOCK);
#pragma unroll
                for (int kk = 0; kk < WC_KEYS / 16; ++kk)
#pragma unroll
                    for (int part = 0; part < 2; ++part)  // hi, lo
                        umma_bf16_a_tmem(tmem, s_col + (t & 1) * WC_KEYS + part * (WC_KEYS / 2) + kk * 8,
                                         smem_desc_mn_sw128(v_addr + kk * 2048, WC_BLOCK, 1024), idesc_o, t > 0 || kk > 0 || part > 0 ? 1u : 0u);
                umma_commit(v_empty + 8 * s);
                umma_commit(o_done0 + 8 * (t & 1));
            }
        }
    } else {
        // ---- softmax: a thread per row ---------------------------------------------------------------------------
        const int quarter = warp & 3, row = quarter * 32 + lane;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        const int n = n0 + row / per, h = g * per + row % per, pos = p0 + row / per;  // (rows past the tile's end are not stored)
        const int lo = first_of(pos);
        // whole tiles between these are seen by every row
        const int seen_from = first_of(kv_end - 1), seen_to = p0;
        float scale2 = a.scale * 1.4426950408889634f * wa_query_temperature(pos, a.temp_coef, a.temp_every);
        if (a.head_scale != nullptr) scale2 *= a.head_scale[h];
        const bool negative = scale2 < 0.f;  // (then it is -S whose largest value counts)
        scale2 = scale2 == 0.f ? 1e-37f : fabsf(scale2);  // (a hidden key's -infinity must stay that under a factor of nothing)
        const float shift = a.head_bias != nullptr ? a.head_bias[h] * 1.4426950408889634f : 0.f;
        float m = -INFINITY, l = 0.f;  // the maximum that the row's exponentials are taken against (base 2), their sum
        bool ok = true;
        for (int t = 0; t < tiles; ++t) {
            ok = mbar_wait(s_full + 8 * (t & 1), (t >> 1) & 1, give_up);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            if (t >= 2) {  // the sums of tile t - 2 (their barrier's next phase, those of tile t, needs this warp's weights)
                ok = mbar_wait(o_done0 + 8 * (t & 1), ((t >> 1) - 1) & 1, give_up);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
            }
            tc_fence_after();
            const uint32_t s_addr = s_col + (t & 1) * WC_KEYS + lanes;
            float v[WC_KEYS];
            tmem_ld32(s_addr, v);
            tmem_ld32(s_addr + 32, v + 32);
            if (negative) {
#pragma unroll
                for (int i = 0; i < WC_KEYS; ++i) v[i] = -v[i];
            }
            const int key = key_of(t);
            if (key < seen_from || key + WC_KEYS - 1 > seen_to) {
#pragma unroll
                for (int i = 0; i < WC_KEYS; ++i) {
                    const int j = key + i;
                    v[i] = j <= pos && (j >= lo || j < a.keep) ? v[i] : -INFINITY;
                }
            }
            float mx[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
            for (int i = 4; i < WC_KEYS; ++i) mx[i & 3] = fmaxf(mx[i & 3], v[i]);
            const float top = fmaf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), scale2, shift);
            float alpha = 1.f;
            bool moved = false;
            if (top > m + WC_LAZY) {  // (never for a tile without a visible key)
                if (m != -INFINITY) {
                    alpha = ex2(m - top);
                    moved = true;
                }
                m = top;
            }
            const float base = m == -INFINITY ? INFINITY : m - shift;  // (no visible key so far: weights of 0, also where the addend is -infinity)
            if (__any_sync(0xffffffffu, moved)) {  // O so far times alpha, at rest once the sums of the tile before are done
                ok = mbar_wait(o_done0 + 8 * ((t - 1) & 1), ((t - 1) >> 1) & 1, give_up);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                for (int c = 0; c < dv; c += 16) rescale_o<16>(tmem + lanes + c, alpha);
            }
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < WC_KEYS; ++i) v[i] = ex2(fmaf(v[i], scale2, -base));
#pragma unroll
            for (int i = 0; i < WC_KEYS; ++i) sum[i & 3] += v[i];
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
                tmem_st16(s_addr + WC_KEYS / 2 + 16 * half, low);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(p_full + 8 * (t & 1)) : "memory");
        }
        for (int t = max(0, tiles - 2); t < tiles && ok; ++t) {
            ok = mbar_wait(o_done0 + 8 * (t & 1), (t >> 1) & 1, give_up);
            ok = __all_sync(0xffffffffu, ok);
        }
        if (ok) {
            tc_fence_after();
            const float sk = a.sink != nullptr ? a.sink[h] * 1.4426950408889634f : -INFINITY;  // joins the denominator only
            const float top = fmaxf(m, sk), keep = m == -INFINITY ? 0.f : exp2f(m - top);
            const float denom = l * keep + (sk == -INFINITY ? 0.f : exp2f(sk - top));
            const bool stored = row < tokens * per;
            float inv = denom > 0.f ? keep / denom : 0.f;
            const float* gate = a.gate != nullptr && stored ? a.gate + (size_t)n * a.ldg + (a.gate_entries ? h * dv : h) : nullptr;
            if (gate != nullptr && !a.gate_entries) inv /= 1.f + expf(-*gate);
            bf16* out = all_out + (size_t)n * HV + (size_t)h * dv;
            for (int c = 0; c < dv; c += 16) {
                float v[16];
                tmem_ld16(tmem + lanes + c, v);
                if (!stored) continue;
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] *= inv;
                if (gate != nullptr && a.gate_entries) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] /= 1.f + expf(-gate[c + i]);
                }
                *(uint4*)(out + c) = make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
                *(uint4*)(out + c + 8) = make_uint4(pack2(v[8], v[9]), pack2(v[10], v[11]), pack2(v[12], v[13]), pack2(v[14], v[15]));
            }
        }
    }
    __syncwarp();
    if (*give_up && tid == 0) cw_report(a.status, CW_ST_WAIT_TIMEOUT, blockIdx.x, -4);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, WC_TMEM);
}

// ---- host side ---------------------------------------------------------------------------------------------------
static int wc_stages(int kb, int vb) {
    const int room = (WC_SMEM - 2048 - kb * WC_Q_BLOCK) / ((kb + vb) * WC_BLOCK);
    return room > WC_MAX_STAGES ? WC_MAX_STAGES : room;
}

// Whether this kernel is the faster one.  Its time is that of a row tile's chain, about 13 us and 1.5 to 1.8 for 64 keys, times the
// rounds of WC_AT_ONCE CTAs; single tokens fill a row tile with `per` rows of 128, so many of them take several rounds.  The
// mma.sync kernel takes 4 to 5 us and 6 to 11 for 64 keys (24 with one head per key/value head of 128 + 128), in blocks of 16
// rows of which four to eight share an SM, and cuts the keys of few rows in parts.  Measured there and here (us, B200):
//   cut keys: 64 tokens behind 8,000 on an open window, 15 parts, 134 and 236; 32 of them, 4 parts, 316 and 238; 512, 16 parts on 64
//   row tiles, 481 and 258; 8 behind 1,000 in a window of 1,024, 8 parts, 39 and 43; 4 parts of 512 keys, 32 heads of 64 + 64 on 8:
//   8 single tokens 22 and 24, a portion of 32 24 and 27, 24 single tokens 41 and 28; with heads of 128 + 128 equal or faster here;
//   uncut, 16 heads of 128 + 128 on 4: 64 single tokens in a window of 64 17 and 22, of 128 28 and 23; 256 of them, four rounds, 43 and
//   80, 72 and 92, of 192 104 and 101; 32 heads of 64 + 64 on 8, 128 single tokens: 27 and 59, 44 and 67, 61 and 74, of 256 77 and 81;
//   a portion of 300 in a window of 16 13 and 21, of 64 23 and 21 (heads of 64 + 64: 16 and 18).
bool window_tc_pays(const WindowAttentionArgs& a, int N, int S) {
    const int per = a.H / a.G, width = a.dk + a.dv;
    const long long keys = (long long)a.window + a.keep;
    const bool singles = N < 2LL * S;  // (fewer than two tokens a request: as good as all of them)
    if (a.parts > WC_MAX_PARTS) return ((long long)N * per + WC_ROWS - 1) / WC_ROWS * a.G >= WC_MIN_TILES;
    if (a.parts > 1) return !(a.parts == WC_MAX_PARTS && width <= 128 && per > 1 && N <= 32 && (N <= 8 || !singles));
    if (!singles) return keys * width > (N >= 32 ? 8192 : 4096);
    if ((long long)min(N, S) * a.G <= WC_AT_ONCE) return keys > (per > 1 ? 64 : 16);
    return keys > (per >= 8 || (per == 1 && width > 128) ? 64 : 32768 / width);
}

// Key and value sizes of whole steps of 16 up to 128; query heads per key/value head that divide the 128 rows; rows, strides and
// bases of whole 16-byte pieces; pages of 8, 16 or 32 tokens or a multiple of 64 (a box of keys lies in one page).
bool window_tc_takes(const WindowAttentionArgs& a) {
    if (a.talk != nullptr || a.sigmoid_weights || a.softcap > 0.f || a.slopes != nullptr || a.pool > 0) return false;
    if (a.dk % 16 || a.dv % 16 || a.dk > WC_MAX_DIM || a.dv > WC_MAX_DIM) return false;
    const int per = a.H / a.G, width = a.voff + a.dv;
    if (per > WC_ROWS || (per & (per - 1)) || width % 8 || a.voff % 8 || a.ldq % 8) return false;
    if (a.page_size != 8 && a.page_size != 16 && a.page_size != 32 && a.page_size % WC_KEYS) return false;
    return ((uintptr_t)a.q | (uintptr_t)a.cache | (uintptr_t)a.out) % 16 == 0 && (long long)a.num_pages * a.page_size <= 0x7fffffffLL;
}

int window_tc_run(const WindowAttentionArgs& a, const int* q_start, int S, int N, cudaStream_t stream) {
    if (load_encode() != 0) return CW_ERR_UNSUPPORTED;
    const int per = a.H / a.G, kb = (a.dk + 63) / 64, vb = (a.dv + 63) / 64, box = a.page_size < WC_KEYS ? a.page_size : WC_KEYS;
    const WindowTc p = {a, q_start, S, N, per, WC_ROWS / per, kb, vb, wc_stages(kb, vb), box, WC_KEYS / box};
    const long long blocks = (((long long)N + p.tokens - 1) / p.tokens + S) * a.G;
    if (blocks > 0x7fffffffLL) return CW_ERR_UNSUPPORTED;
    CUtensorMap q, c;
    {
        const cuuint64_t dims[3] = {(cuuint64_t)a.dk, (cuuint64_t)a.H, (cuuint64_t)N};
        const cuuint64_t strides[2] = {(cuuint64_t)a.dk * 2, (cuuint64_t)a.ldq * 2};
        const cuuint32_t shape[3] = {64, (cuuint32_t)per, (cuuint32_t)p.tokens}, elem[3] = {1, 1, 1};
        if (g_encode(&q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(a.q), dims, strides, shape, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return CW_ERR_UNSUPPORTED;
    }
    {
        const int width = a.G * (a.voff + a.dv);
        const cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)a.num_pages * a.page_size};
        const cuuint64_t strides[1] = {(cuuint64_t)width * 2};
        const cuuint32_t shape[2] = {64, (cuuint32_t)box}, elem[2] = {1, 1};
        if (g_encode(&c, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(a.cache), dims, strides, shape, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return CW_ERR_UNSUPPORTED;
    }
    const size_t smem = (size_t)kb * WC_Q_BLOCK + (size_t)p.stages * (kb + vb) * WC_BLOCK + 2048;
    const cudaError_t e = cudaFuncSetAttribute(window_attention_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WC_SMEM);
    if (e != cudaSuccess) return (int)e;
    return cw_launch_ordered(window_attention_tc_kernel, dim3((unsigned)blocks), dim3(WC_THREADS), smem, stream, q, c, p);
}

CW_TRACE_TU(window_attention_tc)
