// The matrix product for prompt portions on CTA pairs (tcgen05 cta_group::2).
//
// Two CTAs of a cluster, on neighbouring SMs, share one tile of 256 output features x bn tokens:
// each loads its own 128 rows of W and only half of the token tile, and the leader's one thread
// issues MMAs of M = 256 that run on both SMs' tensor cores and read the token tile from both
// shared memories.  Against two independent 128 x bn tiles that halves the token-operand traffic
// per SM (TMA writes and tensor-core reads of shared memory), which is what bounds the single-CTA
// kernel.  Each CTA keeps the accumulator of its own 128 features in its own tensor memory (two
// buffers: the epilogue of one tile overlaps the MMAs of the next) and stores it itself.
//
// Barriers: `full[s]` lives in the leader and counts one arrive.expect_tx per CTA plus the bytes
// of both CTAs' copies (the peer's copies signal it through the cluster's shared-memory window);
// `empty[s]` and `acc_full[b]` are signalled in both CTAs at once by a multicast tcgen05.commit;
// `acc_empty[b]` lives in the leader and counts one arrival per epilogue warp.  Every wait is
// bounded; a CTA that gives up records CW_ST_WAIT_TIMEOUT, and both CTAs meet at the cluster
// barrier before tensor memory is freed.
//
// Few tiles and a long inner dimension (a few hundred tokens against K = 8960): a k-block takes a pair
// at least 180 ns, a stage's round trip over the stages in flight (wide tiles 1.3 ns a token), so with
// fewer tiles than pairs the product's time is K's, whatever the tile's width.  The products that add
// into the residual are then split over K (p.splits > 1): a unit of work is (tile, split), every split
// adds its partial tile into the residual with the same reductions, and the splits of a tile add in
// split order: split k waits, before its first store, until split k - 1 has published (its word of
// p.split_flags == k) that its adds are complete.  Units are handed out in the order (tile, split) to
// pairs that all run at once and take their units in ascending order, so the unit waited for is always
// running or done.
#pragma once
#include "tc_common.cuh"

#define PAIR_EPI_WARPS 8
#define PAIR_THREADS (64 + 32 * PAIR_EPI_WARPS)
#define PAIR_CHUNK 32            // tokens per round of an epilogue warp
#define PAIR_MAX_STAGES 12
#define PAIR_MAX_SMEM (226 * 1024)  // (a few bytes of the 227 KB are static)

// SWIGLU: two weight matrices (gate and up) against the same token tile, two accumulators per tile, and
// silu(gate) * up in the epilogue; token tiles are then at most 128 wide (tensor memory holds two
// buffers of two accumulators).
template <bool SWIGLU>
struct PairCfgT {
    static constexpr int BN_MAX = SWIGLU ? 128 : 256;            // BM = 128 and BK = 64 as in the single-CTA kernels
    static constexpr int ACC_STRIDE = 256;                       // tensor-memory columns per buffer (SWIGLU: gate at 0, up at 128)
    static constexpr int A_BYTES = BM * BK * 2;                  // this CTA's 128 rows of W (of each W)
    static constexpr int SMEM_BYTES = PAIR_MAX_SMEM;
    static constexpr int TMEM_COLS = 512;                        // two buffers of up to 256 columns
    // A stage holds the weight rows and half of a token tile of bn, so that narrow tiles have more stages (11 at 64 tokens, 7 at
    // 256; SwiGLU 6 and, at 128, 5): what bounds the products of few tiles and a long K is the latency of a stage's round trip over
    // the stages in flight.
    __host__ __device__ static constexpr int stage_bytes(int bn) { return (SWIGLU ? 2 : 1) * A_BYTES + bn / 2 * BK * 2; }
    __host__ __device__ static constexpr int stages(int bn) {
        const int n = (SMEM_BYTES - 2048) / stage_bytes(bn);
        return n < PAIR_MAX_STAGES ? n : PAIR_MAX_STAGES;
    }
    static_assert(stages(BN_MAX) >= 4, "too few operand stages");
};
using PairCfg = PairCfgT<false>;

__device__ __forceinline__ void tmem_alloc_pair(uint32_t result_slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(result_slot), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                               uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrives, when the MMAs issued so far are complete, on the barrier at this offset in both CTAs.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
        ::"r"(bar), "h"((uint16_t)3)
        : "memory");
}
// A tile copy whose completion bytes go to a barrier that may lie in the other CTA of the pair.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t cluster_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(cluster_bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void mbar_expect_tx_cluster(uint32_t cluster_bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cluster.b64 _, [%0], %1;" ::"r"(cluster_bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}

// Tiles: 256 features x p.bn tokens per pair; p.bn is a multiple of 16 (each CTA holds p.bn / 2 token
// rows, whole swizzle atoms of 8).  map_x's box is p.bn / 2 rows.
template <bool SWIGLU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_w2,
                    const __grid_constant__ CUtensorMap map_x, const GemmParams p) {
    using C = PairCfgT<SWIGLU>;
    constexpr int B_OFF = (SWIGLU ? 2 : 1) * C::A_BYTES;  // the token rows' place in a stage
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int bn = p.bn, half_bn = bn >> 1;
    const int stages = C::stages(bn), stage_bytes = C::stage_bytes(bn);
    uint64_t* bars = (uint64_t*)(smem + stages * stage_bytes);
    // bars: full[S], empty[S], acc_full[2], acc_empty[2]
    uint32_t* tmem_slot = (uint32_t*)(bars + 2 * PAIR_MAX_STAGES + 4);
    volatile int* give_up = (volatile int*)(tmem_slot + 1);

    // Only the activations come from the preceding kernel, and only the producer threads read them
    // (everything else follows from their copies): they alone wait for it, after the set-up and after
    // the weight tiles of the first stages have gone out.
    cw_trace(0);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank();  // 0: the leader, which issues the MMAs
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + PAIR_MAX_STAGES);
    const uint32_t accf0 = smem_u32(bars + 2 * PAIR_MAX_STAGES), acce0 = smem_u32(bars + 2 * PAIR_MAX_STAGES + 2);
    const int m_tiles = (p.N + 2 * BM - 1) / (2 * BM), n_tiles = (p.T + bn - 1) / bn;
    const int splits = p.splits, nkb = p.kb_per_split;  // splits * nkb == p.num_kb
    const int tiles = m_tiles * n_tiles * splits;       // units of work: unit u is split u % splits of tile u / splits
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(full0 + 8 * s, 2);   // one arrive.expect_tx per CTA (used in the leader only)
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(accf0 + 8 * b, 1);
            mbar_init(acce0 + 8 * b, 2 * PAIR_EPI_WARPS);   // one arrival per epilogue warp of both CTAs (used in the leader only)
        }
        *give_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) tmem_alloc_pair(smem_u32(tmem_slot), C::TMEM_COLS);
    tc_fence_before();
    cluster_sync();  // both CTAs' barriers are initialised before either signals the other's
    pdl_release();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0 && elect_one()) {
        // ---- TMA producer (both CTAs): own rows of W, own half of the token tile ------------------------
        const uint32_t stage_tx = B_OFF + half_bn * BK * 2;
        const int my_tiles = pair < tiles ? (tiles - pair + pairs - 1) / pairs : 0;
        const int total = my_tiles * nkb;  // k-blocks of all this pair's units, in order
        const int early = min(total, stages);
        bool ok = true;
        // the first stages: weight tiles before the wait, their activation tiles after it
        for (int phase = 0; phase < 2; ++phase) {
            if (phase == 1) pdl_wait();
            for (int i = 0; i < early; ++i) {
                const int ts = i / nkb, unit = pair + ts * pairs, tile = unit / splits;
                const int kb = (unit - tile * splits) * nkb + (i - ts * nkb);  // k-block within K
                const int m0 = (tile % m_tiles) * 2 * BM + (int)rank * BM;
                const int n0 = (tile / m_tiles) * bn + (int)rank * half_bn;
                const uint32_t a_dst = smem_u32(smem + i * stage_bytes);
                const uint32_t bar = dsmem_addr(full0 + 8 * i, 0);  // the leader's barrier
                if (phase == 0) {
                    mbar_expect_tx_cluster(bar, stage_tx);
                    tma_load_2d_pair(a_dst, &map_w, kb * BK, m0, bar);
                    if (SWIGLU) tma_load_2d_pair(a_dst + C::A_BYTES, &map_w2, kb * BK, m0, bar);
                } else {
                    tma_load_2d_pair(a_dst + B_OFF, &map_x, kb * BK, n0, bar);
                }
            }
        }
        // the rest runs ahead over tiles, bounded by the ring only; the stage and its phase are counted along
        int kb = early % nkb, s = early == stages ? 0 : early;
        uint32_t parity = early < stages ? 1 : 0;
        const uint32_t smem0 = smem_u32(smem), leader_full0 = dsmem_addr(full0, 0);
        for (int unit = pair + (early / nkb) * pairs; unit < tiles && ok; unit += pairs, kb = 0) {
            const int tile = unit / splits, kb0 = (unit - tile * splits) * nkb;
            const int m0 = (tile % m_tiles) * 2 * BM + (int)rank * BM;
            const int n0 = (tile / m_tiles) * bn + (int)rank * half_bn;
            for (; kb < nkb; ++kb) {
                ok = mbar_wait(empty0 + 8 * s, parity, give_up);
                if (!ok) break;
                const uint32_t a_dst = smem0 + s * stage_bytes;
                const uint32_t bar = leader_full0 + 8 * s;
                mbar_expect_tx_cluster(bar, stage_tx);
                tma_load_2d_pair(a_dst, &map_w, (kb0 + kb) * BK, m0, bar);
                if (SWIGLU) tma_load_2d_pair(a_dst + C::A_BYTES, &map_w2, (kb0 + kb) * BK, m0, bar);
                tma_load_2d_pair(a_dst + B_OFF, &map_x, (kb0 + kb) * BK, n0, bar);
                if (++s == stages) {
                    s = 0;
                    parity ^= 1;
                }
            }
        }
        if (*give_up) {
            // copies may still be in flight into this CTA's shared memory, and their barrier lies in the
            // leader: let them land before the CTA goes on to the final barrier and leaves
            const long long t0 = clock64();
            while (clock64() - t0 < 2000000LL) {
            }
        }
    } else if (warp == 1 && rank == 0 && elect_one()) {
        // ---- MMA issuer (leader only): tile `it` accumulates into TMEM buffer it & 1 of both CTAs ---------
        pdl_wait();  // (parked here a thread polls no barrier)
        const uint32_t idesc = instr_desc(2 * BM, bn);
        const uint64_t desc0 = smem_desc_sw128(smem_u32(smem));
        uint64_t adesc = desc0;  // (16-byte units: a stage further is stage_bytes / 16)
        int it = 0, s = 0;
        uint32_t parity = 0;
        bool ok = true;
        for (int tile = pair; tile < tiles && ok; tile += pairs, ++it) {
            const int buf = it & 1;
            ok = mbar_wait(acce0 + 8 * buf, ((it >> 1) & 1) ^ 1, give_up);  // both epilogues have drained it
            if (!ok) break;
            tc_fence_after();
            const uint32_t acc = tmem_base + buf * C::ACC_STRIDE;
            for (int kb = 0; kb < nkb; ++kb) {
                ok = mbar_wait(full0 + 8 * s, parity, give_up);
                if (!ok) break;
                tc_fence_after();
                const uint64_t udesc = adesc + C::A_BYTES / 16, bdesc = adesc + B_OFF / 16;
#pragma unroll
                for (int k = 0; k < BK / 16; ++k)
                    umma_bf16_pair(acc, adesc + 2 * k, bdesc + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                if (SWIGLU) {
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k)
                        umma_bf16_pair(acc + C::ACC_STRIDE / 2, udesc + 2 * k, bdesc + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                }
                umma_commit_pair(empty0 + 8 * s);  // the stage is free in both CTAs
                adesc += stage_bytes / 16;
                if (++s == stages) {
                    s = 0;
                    parity ^= 1;
                    adesc = desc0;
                }
            }
            if (ok) umma_commit_pair(accf0 + 8 * buf);
        }
    } else if (warp >= 2) {
        // ---- epilogue warps (both CTAs): warp w reads TMEM lanes 32 (w % 4) .. +31 of its own CTA, every other 32 tokens ---------
        // Straight from tensor memory to global memory: a warp's 32 features of a token are one line in float32, half of one in
        // bfloat16.  Where a pair has one or two tiles the epilogue is not hidden, and the way through shared memory and TMA cost
        // about 1,200 cycles per 32 tokens (stores into shared memory 440, two TMA stores 400, the proxy fence and waits for the
        // staging buffer 270).  Measured (B200): 2,048 tokens, N x K of 2048 x 1536
        // stored 16.9 -> 14.3 us, 1536 x 1536 added 16.4 -> 15.4; a tile of 256 tokens per pair and one k-block 8.0 -> 5.1 us.
        pdl_wait();
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        const bool wide = !SWIGLU && p.epilogue != 0;
        const uint32_t acce_leader = dsmem_addr(acce0, 0);
        int it = 0;
        bool ok = true;
        for (int unit = pair; unit < tiles && ok; unit += pairs, ++it) {
            const int buf = it & 1;
            const int tile = unit / splits, ks = unit - tile * splits;
            const int f = (tile % m_tiles) * 2 * BM + (int)rank * BM + quarter * 32 + lane;
            const int n0 = (tile / m_tiles) * bn;
            int* const flag = p.split_flags + (2 * tile + rank) * PAIR_EPI_WARPS + (warp - 2);
            // (a split's adds come after those of the split before it; splits that are kept apart, epilogue
            // 3, store into slabs of their own and wait for nobody)
            const bool apart = p.epilogue == 3;
            const int y0 = (apart ? ks * p.part_rows : 0) + n0;  // the tile's first row in C
            ok = __all_sync(0xffffffffu, mbar_wait(accf0 + 8 * buf, (it >> 1) & 1, give_up));
            if (!ok) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + buf * C::ACC_STRIDE + ((uint32_t)(quarter * 32) << 16);
            const float bias = (p.bias != nullptr && f < p.N && ks == 0) ? p.bias[f] : 0.f;
            if (ks > 0 && !apart) {  // (every epilogue warp of the tile waits for itself: its features and tokens are its own)
                if (lane == 0) {
                    const long long t0 = clock64();
                    int seen;
                    do {
                        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(flag) : "memory");
                    } while (seen != ks && clock64() - t0 < WAIT_CYCLES);
                    if (seen != ks) *give_up = 1;
                }
                __syncwarp();
            }
            const int c_end = min(bn, p.T - n0);
            for (int c = half * PAIR_CHUNK; c < c_end; c += 2 * PAIR_CHUNK) {
                const int rows = f < p.N ? c_end - c : 0;  // of this round's 32 tokens, those that this lane stores
                uint32_t r[PAIR_CHUNK];
                tmem_ld16_begin(taddr + c, r);
                tmem_ld16_begin(taddr + min(c + 16, bn - 16), r + 16);  // (a tile may end behind 16 tokens of a round)
                tmem_landed(r);
                tmem_landed(r + 16);
                float v[PAIR_CHUNK];
#pragma unroll
                for (int j = 0; j < PAIR_CHUNK; ++j) v[j] = __uint_as_float(r[j]) + bias;
                if (SWIGLU) {
                    tmem_ld16_begin(taddr + C::ACC_STRIDE / 2 + c, r);
                    tmem_ld16_begin(taddr + C::ACC_STRIDE / 2 + min(c + 16, bn - 16), r + 16);
                    tmem_landed(r);
                    tmem_landed(r + 16);
#pragma unroll
                    for (int j = 0; j < PAIR_CHUNK; ++j) v[j] = gated_act(v[j], __uint_as_float(r[j]), p.act_limit);
                } else if (p.squared_relu) {
#pragma unroll
                    for (int j = 0; j < PAIR_CHUNK; ++j) v[j] = squared_relu(v[j]);
                }
                const size_t at = (size_t)(y0 + c) * p.ldc + f;
                if (!wide) {
                    bf16* to = (bf16*)p.C + at;
#pragma unroll
                    for (int j = 0; j < PAIR_CHUNK; ++j, to += p.ldc)
                        if (j < rows) *to = __float2bfloat16_rn(v[j]);
                } else if (p.epilogue == 1) {
                    float* to = (float*)p.C + at;
#pragma unroll
                    for (int j = 0; j < PAIR_CHUNK; ++j, to += p.ldc)
                        if (j < rows) asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" ::"l"(to), "f"(v[j]) : "memory");
                } else {
                    float* to = (float*)p.C + at;
#pragma unroll
                    for (int j = 0; j < PAIR_CHUNK; ++j, to += p.ldc)
                        if (j < rows) *to = v[j];
                }
            }
            tc_fence_before();
            if (splits > 1 && !apart) __threadfence();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive_cluster(acce_leader + 8 * buf);  // this warp's part of the accumulator has been read out
                if (splits > 1 && !apart) {
                    // this split's adds are complete: the next split of the tile may add (the last one leaves
                    // the flag at zero for the next launch)
                    const int next = ks + 1 == splits ? 0 : ks + 1;
                    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(flag), "r"(next) : "memory");
                }
            }
        }
    }
    __syncwarp();
    if (*give_up && tid == 0) cw_report(p.status, CW_ST_WAIT_TIMEOUT, blockIdx.x, -2);
    // Neither CTA leaves, or frees tensor memory, while the other may still signal its barriers or
    // while MMAs that read its shared memory may be in flight.
    tc_fence_before();
    cluster_sync();
    if (warp == 1) tmem_dealloc_pair(tmem_base, C::TMEM_COLS);
}
