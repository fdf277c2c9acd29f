// Float32 products on the 5th-generation tensor cores, as exact as on the CUDA cores.
//
// A float32 number is the sum of three bfloat16 numbers of 8 bits each: w = w0 + w1 + w2, x = x0 + x1 + x2, the first cut off (so
// that it does not overflow), the second rounded (so that the third has either sign and what is left out below has no
// direction).  The tensor cores form w0 x0 and the six products w1 x0, w0 x1, w1 x1, w2 x0, w0 x2 and w2 x1 exactly and add
// them up in float32, cutting off what falls below the last bit; w1 x2 and w2 x2, at most 2^-24 of w0 x0, are left out.  So that little falls off, w0 x0 has an
// accumulator of its own for every 16 k, the small products two for 64 k; per 64 k the six are read out of tensor memory,
// added, and their sum is added into a running sum that carries its rounding errors along (Kahan).  Measured against float64
// (B200, K 1,536 and 8,960, this kernel and the chains of 16 fmaf with the same running sum that it replaced): normal operands
// 6.8e-8 and 7.3e-8, chains 8.1e-8 and 8.6e-8; sizes spread over e^3 8.5e-8 and 8.1e-8, chains 7.8e-8; operands of one sign 3.1e-8
// and 2.8e-8, chains 2.3e-8.  With one accumulator for all products of 64 k 8.6e-8 to 1.5e-7.
//
// Every output's sum has the same order whatever M, N or the tile it falls in, so a row's result does not depend on the rest of
// the batch: 64 k at a time, a long K cut into segments of about F32_SEGMENT by K alone, each segment on a CTA of a cluster;
// the CTAs leave sums and what they lost in shared memory, share the outputs among them and add the segments up in order.
//
// A CTA: up to 128 weight rows (the MMA's M) by up to 64 tokens (its N).  Eight warps copy the operands' next 64 k into
// shared memory, cut them in three and store them there as the MMAs read them (K-major, 128-byte swizzle), two stages;
// a thread of another issues the MMAs.  The parts of the token rows follow one another, so that one MMA of twice the width forms
// w1 [x0 | x1], w0 [x1 | x2] or w2 [x0 | x1]: 16 MMAs per 64 k, none of which takes less than about 64 cycles however narrow.
// Eight other warps read out and add up what has been formed.  What bounds it: few rows, the 16 MMAs in a row (about 1,600 cycles per
// 64 k); many, the issue slots (60 % busy: the cutting in three, then the sums) beside them.  Measured (B200, us, chains of fmaf
// -> this): 200 rows, [gate, up] 2 x 8,960 by 1,536 370 -> 200, 1,536 by 8,960 217 -> 125, 2,048 by 1,536 62 -> 38; 64 rows
// 168 -> 56, 105 -> 44, 32 -> 29; 1 row 36 -> 35, 34 -> 39, 27 -> 25.  Tried: the same eight warps for both jobs, one after the
// other (207 us for [gate, up] of 200 rows: every step's latency in a row), sixteen (199).
//
// Every wait on an mbarrier is bounded.
#include "cluster_places.cuh"
#include "gemm_f32.cuh"
#include "tc_common.cuh"

#define F32_ADDERS 8       // warps that read out and add up (two for every quarter of tensor memory)
#define F32_CONVERTERS 8   // warps that bring the operands
#define F32_THREADS 640    // (and a warpgroup whose first warp issues the MMAs)
#define F32_BK 64
#define F32_ROWS 128
#define F32_MAX_TOKENS 64
#define F32_SEGMENT 1792
#define F32_MAX_SEGMENTS 8

// sum += x with the rounding error of earlier additions carried along in `lost` (Kahan's summation;
// the order of the operations matters and the compiler keeps it: no fast-math flags are used)
__device__ __forceinline__ void f32_add(float& sum, float& lost, float x) {
    const float y = __fsub_rn(x, lost);
    const float t = __fadd_rn(sum, y);
    lost = __fsub_rn(__fsub_rn(t, sum), y);
    sum = t;
}

// The first 8 of a float's 24 bits as a float; of two such floats, the upper halves side by side.
__device__ __forceinline__ float first8(float x) { return __uint_as_float(__float_as_uint(x) & 0xffff0000u); }
__device__ __forceinline__ uint32_t upper2(float x, float y) { return __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632); }

__device__ __forceinline__ uint32_t rounded2(float x, float y) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
    return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ void f32_cluster_barrier() {
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ float2 load_of_rank(const void* mine, int rank) {  // the same place in another CTA of the cluster
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(dsmem_addr(smem_u32(mine), rank)) : "memory");
    return v;
}

template <bool SWIGLU>
__device__ __forceinline__ void f32_store(const F32Args& p, int m, int n, float v, float up) {
    if (p.bias) v += p.bias[n];
    float* to = p.C + (size_t)m * p.ldc + n;
    if (SWIGLU) {
        *to = v / (1.0f + expf(-v)) * up;
    } else if (p.epilogue == 4) {  // the square of what is positive
        v = fmaxf(v, 0.f);
        *to = v * v;
    } else if (p.epilogue == 1) {
        *to += v;
    } else {
        *to = v;
    }
}

// Tiles of up to BN tokens and up to ROWS weight rows.
template <int BN, int ROWS>
struct F32Cfg {
    static constexpr int W_PART = F32_ROWS * F32_BK * 2, X_PART = BN * F32_BK * 2;  // one of the three parts of an operand (rows: at most)
    static constexpr int STAGE = 3 * (W_PART + X_PART);
    static constexpr int MINE = BN / 32;                          // groups of 16 tokens of an adding warp
    // Tensor memory: four accumulators of w0 x0 (twice where there is room), two of the small products twice, so that the next
    // 64 k's are formed while these are read out.
    static constexpr int SETS = BN <= 32 ? 2 : 1, SMALL = SETS * 4 * BN, TMEM_COLS = 512;
    // Pieces of eight numbers of 64 k that a converting thread brings, and how many times 64 k it has on their way: as many as there
    // is room for (few rows per CTA are bound by the latency of these copies).
    static constexpr int W_PIECES = ROWS * 8 / (32 * F32_CONVERTERS), PIECES = W_PIECES + (BN * 8 + 32 * F32_CONVERTERS - 1) / (32 * F32_CONVERTERS);
    static constexpr int ROOM = (226 * 1024 - 1280 - 2 * STAGE) / (PIECES * 1024 * F32_CONVERTERS);
    static constexpr int AHEAD = ROOM < 6 ? ROOM : 6;
    static constexpr int RAW = AHEAD * PIECES * 32 * F32_CONVERTERS * 32;
    static constexpr int SMEM = 2 * STAGE + RAW + 1024 + 256;
    static_assert(SMALL + 4 * BN <= TMEM_COLS && BN % 32 == 0, "accumulators");
    static_assert(BN * F32_ROWS * 8 <= 2 * STAGE, "sums and what they lost fit where the operands were");
    static_assert(AHEAD >= 1 && SMEM <= 226 * 1024, "shared memory");
};

// Copies into shared memory that leave zeros where there is nothing to read.
template <int BYTES>
__device__ __forceinline__ void copy_or_zero(uint32_t to, const float* from, bool there) {
    if (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(from), "r"(there ? 16 : 0) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(from), "r"(there ? 4 : 0) : "memory");
}

// With SWIGLU the weight rows are 32 of the gate matrix, the same 32 of the up matrix, and so on.
template <int BN, int ROWS, bool SWIGLU, bool WHOLE>
__global__ void __launch_bounds__(F32_THREADS, 1) gemm_f32_kernel(const F32Args p) {
    using C = F32Cfg<BN, ROWS>;
    extern __shared__ uint8_t f32_smem[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)f32_smem + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + 2 * C::STAGE + C::RAW);  // full[2], empty[2], then full[2], empty[2] of w0 x0 and of the small products
    uint32_t* tmem_slot = (uint32_t*)(bars + 12);
    volatile int* give_up = (volatile int*)(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 16, first_full = full0 + 32, first_empty = full0 + 48, small_full = full0 + 64, small_empty = full0 + 80;
    const int features = SWIGLU ? p.rows / 2 : p.rows;
    const int n0 = blockIdx.x * features, m0 = blockIdx.y * p.width;
    const int tokens = min(p.width, p.M - m0), groups = (tokens + 15) >> 4;
    const int all = (p.K + F32_BK - 1) / F32_BK, segments = gridDim.z, per = (all + segments - 1) / segments;
    const int first = min((int)blockIdx.z * per, all), blocks = min(per, all - first);

    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(full0 + 8 * s, 32 * F32_CONVERTERS);
            mbar_init(empty0 + 8 * s, 1);
            mbar_init(first_full + 8 * s, 1);
            mbar_init(first_empty + 8 * s, F32_ADDERS);
            mbar_init(small_full + 8 * s, 1);
            mbar_init(small_empty + 8 * s, F32_ADDERS);
        }
        *give_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == F32_ADDERS + F32_CONVERTERS) tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // Registers: 640 threads of 96 at launch, 61,440 in all; 256 x 152 + 256 x 72 + 128 x 32 of them after the split.
    if (warp >= F32_ADDERS + F32_CONVERTERS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        if (warp == F32_ADDERS + F32_CONVERTERS && elect_one()) {
            // ---- MMA issuer ------------------------------------------------------------------------------------------
            const int x_part = groups * 16 * F32_BK * 2;
            const uint32_t idesc = instr_desc(F32_ROWS, 16 * groups), idesc2 = instr_desc(F32_ROWS, 32 * groups);
            bool ok = true;
            for (int b = 0; b < blocks && ok; ++b) {
                const int set = b % C::SETS;
                ok = mbar_wait(full0 + 8 * (b & 1), (b >> 1) & 1, give_up) &&
                     mbar_wait(first_empty + 8 * set, ((b / C::SETS) & 1) ^ 1, give_up);
                if (!ok) break;
                tc_fence_after();
                const uint32_t stage = smem_u32(smem) + (b & 1) * C::STAGE;
                const uint64_t w0 = smem_desc_sw128(stage), w1 = w0 + C::W_PART / 16, w2 = w1 + C::W_PART / 16;
                const uint64_t x0 = w2 + C::W_PART / 16, x1 = x0 + x_part / 16;
                const uint32_t small = tmem + C::SMALL + (b & 1) * 2 * BN;
#pragma unroll
                for (int k = 0; k < F32_BK / 16; ++k) umma_bf16(tmem + (set * 4 + k) * BN, w0 + 2 * k, x0 + 2 * k, idesc, 0u);
                umma_commit(first_full + 8 * set);
                ok = mbar_wait(small_empty + 8 * (b & 1), ((b >> 1) & 1) ^ 1, give_up);
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < F32_BK / 16; ++k) umma_bf16(small, w2 + 2 * k, x0 + 2 * k, idesc2, k > 0 ? 1u : 0u);
#pragma unroll
                for (int k = 0; k < F32_BK / 16; ++k) umma_bf16(small, w0 + 2 * k, x1 + 2 * k, idesc2, 1u);
#pragma unroll
                for (int k = 0; k < F32_BK / 16; ++k) umma_bf16(small, w1 + 2 * k, x0 + 2 * k, idesc2, 1u);
                umma_commit(empty0 + 8 * (b & 1));  // the stage has been read
                umma_commit(small_full + 8 * (b & 1));
            }
        }
        __syncwarp();
        if (segments > 1) {  // (the two that the others meet at below)
            f32_cluster_barrier();
            f32_cluster_barrier();
        }
    } else if (warp >= F32_ADDERS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        // ---- operands: eight numbers of a row a piece, eight pieces a row; a thread converts what it has copied itself.  Its
        // pieces lie 32 rows apart; two of them (a batch) are copied, awaited and converted together, so that their latencies
        // overlap (with one piece after the other a piece took a warp 400 cycles). ------------------------------------------------
        const int ct = tid - 32 * F32_ADDERS;
        constexpr int NT = 32 * F32_CONVERTERS, APART = NT / 8, BATCHES = (C::PIECES + 1) / 2;
        static_assert(APART == 32 && (!SWIGLU || C::W_PIECES % 2 == 0), "pieces of the gated weights: gate, up, gate, up");
        float* raw = (float*)(smem + 2 * C::STAGE) + ct * 8;  // piece i of block b: (b % AHEAD * PIECES + i) * NT pieces further
        const int r0 = ct >> 3;
        const float* const w_row = p.W + (size_t)(n0 + r0) * p.K;
        const float* const w2_row = SWIGLU ? p.W2 + (size_t)(n0 + r0) * p.K : nullptr;
        const float* const x_row = p.A + (size_t)(m0 + r0) * p.lda;
        auto has = [&](int i) {  // whether the tile has piece i's row (zeros among them)
            return i < C::W_PIECES ? r0 + i * APART < p.rows : r0 + (i - C::W_PIECES) * APART < 16 * groups;
        };
        const bool w_full = n0 + features <= p.N && p.rows == ROWS, x_full = tokens == BN;  // every piece has its row
        auto fetch = [&](int b, int i) {
            if (b >= blocks) return;
            const bool of_w = i < C::W_PIECES;
            const int k = (first + b) * F32_BK + (ct & 7) * 8;
            const int r = of_w ? (SWIGLU ? i / 2 * APART : i * APART) : (i - C::W_PIECES) * APART;
            const float* from = (of_w ? (SWIGLU && (i & 1) ? w2_row : w_row) + (size_t)r * p.K : x_row + (size_t)r * p.lda) + k;
            const uint32_t to = smem_u32(raw + (b % C::AHEAD * C::PIECES + i) * 8 * NT);
            if (WHOLE && (of_w ? w_full : x_full && (i + 1 - C::W_PIECES) * APART <= BN) && (first + b + 1) * F32_BK <= p.K) {
                copy_or_zero<16>(to, from, true);
                copy_or_zero<16>(to + 16, from + 4, true);
            } else if (has(i)) {
                const bool there = of_w ? n0 + r0 + r < p.N : r0 + r < tokens;
                const int live = there ? p.K - k : 0;  // numbers from here on (where there are none, nothing is read)
                if (WHOLE) {
                    copy_or_zero<16>(to, live > 0 ? from : p.W, live > 0);
                    copy_or_zero<16>(to + 16, live > 4 ? from + 4 : p.W, live > 4);
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) copy_or_zero<4>(to + 4 * j, live > j ? from + j : p.W, live > j);
                }
            }
        };
        auto fetch_batch = [&](int b, int at) {
#pragma unroll
            for (int i = 2 * at; i < 2 * at + 2; ++i)
                if (i < C::PIECES) fetch(b, i);
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        for (int b = 0; b < C::AHEAD; ++b)
#pragma unroll
            for (int at = 0; at < BATCHES; ++at) fetch_batch(b, at);
        bool ok = true;
        for (int b = 0; b < blocks && ok; ++b) {
            ok = mbar_wait(empty0 + 8 * (b & 1), ((b >> 1) & 1) ^ 1, give_up);
            if (!ok) break;
            uint8_t* const stage = smem + (b & 1) * C::STAGE + (((ct & 7) ^ (r0 & 7)) << 4) + r0 * 128;  // (rows 32 apart swizzle alike)
            const int x_part = groups * 16 * F32_BK * 2;
#pragma unroll
            for (int at = 0; at < BATCHES; ++at) {
                asm volatile("cp.async.wait_group %0;" ::"n"(C::AHEAD * BATCHES - 1) : "memory");
                float4 x[2][2];
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (2 * at + h < C::PIECES) {
                        const float* from = raw + (b % C::AHEAD * C::PIECES + 2 * at + h) * 8 * NT;
                        x[h][0] = *reinterpret_cast<const float4*>(from);
                        x[h][1] = *reinterpret_cast<const float4*>(from + 4);
                    }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int i = 2 * at + h;
                    if (i >= C::PIECES || !has(i)) continue;
                    const float y[8] = {x[h][0].x, x[h][0].y, x[h][0].z, x[h][0].w, x[h][1].x, x[h][1].y, x[h][1].z, x[h][1].w};
                    uint32_t q[3][4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float u = y[2 * j], v = y[2 * j + 1], u1 = u - first8(u), v1 = v - first8(v);
                        const uint32_t rounded = rounded2(u1, v1);
                        q[0][j] = upper2(u, v);
                        q[1][j] = rounded;
                        q[2][j] = upper2(u1 - __uint_as_float(rounded << 16), v1 - first8(__uint_as_float(rounded)));
                    }
                    const bool of_w = i < C::W_PIECES;
                    uint8_t* to = stage + (of_w ? i * APART * 128 : 3 * C::W_PART + (i - C::W_PIECES) * APART * 128);
                    const int part = of_w ? C::W_PART : x_part;
#pragma unroll
                    for (int j = 0; j < 3; ++j) *reinterpret_cast<uint4*>(to + j * part) = make_uint4(q[j][0], q[j][1], q[j][2], q[j][3]);
                }
                fetch_batch(b + C::AHEAD, at);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(full0 + 8 * (b & 1)) : "memory");
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        if (segments > 1) {
            f32_cluster_barrier();
            f32_cluster_barrier();
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 152;");
        float sum[C::MINE][16] = {}, lost[C::MINE][16] = {};  // [group][token]: this thread's feature, half of the groups of 16 tokens
        const int quarter = warp & 3, half = (groups + 1) >> 1, group0 = (warp >> 2) * half, mine_groups = min(half, groups - group0);
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16) + 16 * group0;
        bool ok = true;
        auto add_up = [&](int b) {
            // One accumulator's columns of all groups are loaded before the first is used: a load from tensor memory takes
            // about 200 cycles, and a group after the other paid them each time (80 tokens: 2,400 cycles per 64 k).
            uint32_t t[C::MINE][16], r[C::MINE][16];
            const bool reads = quarter * 32 < p.rows;
            auto load = [&](uint32_t (&to)[C::MINE][16], uint32_t column) {
#pragma unroll
                for (int g = 0; g < C::MINE; ++g)
                    if (g < mine_groups && reads) tmem_ld16_begin(lanes + column + 16 * g, to[g]);
            };
            auto landed = [&](uint32_t (&at)[C::MINE][16]) {
#pragma unroll
                for (int g = 0; g < C::MINE; ++g) tmem_landed(at[g]);
            };
            auto add = [&]() {
#pragma unroll
                for (int g = 0; g < C::MINE; ++g)
                    if (g < mine_groups)
#pragma unroll
                        for (int j = 0; j < 16; ++j) t[g][j] = __float_as_uint(__fadd_rn(__uint_as_float(t[g][j]), __uint_as_float(r[g][j])));
            };
            const int set = b % C::SETS;
            const uint32_t main0 = set * 4 * BN, small = C::SMALL + (b & 1) * 2 * BN;
            ok = __all_sync(0xffffffffu, mbar_wait(first_full + 8 * set, (b / C::SETS) & 1, give_up));
            if (!ok) return;
            tc_fence_after();
            load(t, main0);
            load(r, main0 + BN);
            landed(t);
            landed(r);
            add();
            load(r, main0 + 2 * BN);
            landed(r);
            add();
            load(r, main0 + 3 * BN);
            landed(r);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(first_empty + 8 * set) : "memory");
            add();
            ok = __all_sync(0xffffffffu, mbar_wait(small_full + 8 * (b & 1), (b >> 1) & 1, give_up));
            if (!ok) return;
            tc_fence_after();
            load(r, small);
            landed(r);
            add();
            load(r, small + 16 * groups);
            landed(r);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(small_empty + 8 * (b & 1)) : "memory");
            add();
#pragma unroll
            for (int g = 0; g < C::MINE; ++g)
                if (g < mine_groups)
#pragma unroll
                    for (int j = 0; j < 16; ++j) f32_add(sum[g][j], lost[g][j], __uint_as_float(t[g][j]));
        };
        for (int b = 0; b < blocks && ok; ++b) add_up(b);
        // ---- results: this thread's feature (tensor-memory lane `row`), tokens 16 (group0 + g) + j ---------------------------------------
        asm volatile("bar.sync 1, %0;" ::"n"(32 * F32_ADDERS) : "memory");  // nobody reads the operands any more
        const int row = quarter * 32 + lane;
        const bool mine = row < p.rows;
        auto each = [&](auto f) {  // f(token of the tile, sum, lost)
#pragma unroll
            for (int g = 0; g < C::MINE; ++g)
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int t = 16 * (group0 + g) + j;
                    if (g < half && t < tokens) f(t, sum[g][j], lost[g][j]);
                }
        };
        if (segments == 1) {
            float* ups = (float*)smem;  // [token][64 features]
            if (SWIGLU) {
                if (mine && (quarter & 1)) each([&](int t, float s, float) { ups[t * 64 + (quarter >> 1) * 32 + lane] = s; });
                asm volatile("bar.sync 1, %0;" ::"n"(32 * F32_ADDERS) : "memory");
            }
            const int n = n0 + (SWIGLU ? (quarter >> 1) * 32 + lane : row);
            if (mine && !(SWIGLU && (quarter & 1)) && n < p.N)
                each([&](int t, float s, float) { f32_store<SWIGLU>(p, m0 + t, n, s, SWIGLU ? ups[t * 64 + (quarter >> 1) * 32 + lane] : 0.f); });
        } else {
            float2* part = (float2*)smem;  // [token][weight row]: (sum, lost)
            if (mine) each([&](int t, float s, float l) { part[t * F32_ROWS + row] = make_float2(s, l); });
            f32_cluster_barrier();
            for (int e = (int)blockIdx.z * 32 * F32_ADDERS + tid; e < tokens * features; e += segments * 32 * F32_ADDERS) {
                const int t = e / features, f = e % features, n = n0 + f;
                if (n >= p.N) continue;
                float total[2] = {0.f, 0.f};
#pragma unroll
                for (int u = 0; u < (SWIGLU ? 2 : 1); ++u) {
                    const int r = SWIGLU ? (f >> 5) * 64 + u * 32 + (f & 31) : f;
                    float2 s[F32_MAX_SEGMENTS];
#pragma unroll
                    for (int i = 0; i < F32_MAX_SEGMENTS; ++i)
                        if (i < segments) s[i] = load_of_rank(&part[t * F32_ROWS + r], i);
                    float left = s[0].y;
                    total[u] = s[0].x;
#pragma unroll
                    for (int i = 1; i < F32_MAX_SEGMENTS; ++i)
                        if (i < segments) {
                            f32_add(total[u], left, s[i].x);
                            left += s[i].y;
                        }
                }
                f32_store<SWIGLU>(p, m0 + t, n, total[0], total[1]);
            }
            f32_cluster_barrier();  // nobody leaves while its partial sums are read
        }
    }
    tc_fence_before();
    __syncthreads();
    if (*give_up && tid == 0) cw_report(p.status, CW_ST_WAIT_TIMEOUT, blockIdx.x, -3);
    if (warp == F32_ADDERS + F32_CONVERTERS) tmem_dealloc(tmem, C::TMEM_COLS);
}

// ---- host side ---------------------------------------------------------------------------------------------------
template <int BN, int ROWS, bool SWIGLU, bool WHOLE>
static int launch_f32(const F32Args& p, int segments, cudaStream_t stream) {
    const int features = SWIGLU ? p.rows / 2 : p.rows;
    const cudaError_t e = cudaFuncSetAttribute(gemm_f32_kernel<BN, ROWS, SWIGLU, WHOLE>, cudaFuncAttributeMaxDynamicSharedMemorySize, F32Cfg<BN, ROWS>::SMEM);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.N + features - 1) / features, (p.M + p.width - 1) / p.width, segments);
    if (cfg.gridDim.y > 65535) return CW_ERR_BAD_SIZE;
    cfg.blockDim = F32_THREADS;
    cfg.dynamicSmemBytes = F32Cfg<BN, ROWS>::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {1, 1, (unsigned)segments};
    cfg.attrs = attr;
    cfg.numAttrs = segments > 1 ? 1 : 0;
    const cudaError_t err = cudaLaunchKernelEx(&cfg, gemm_f32_kernel<BN, ROWS, SWIGLU, WHOLE>, p);
    return err != cudaSuccess ? (int)err : CW_LAUNCH_CHECK();
}

template <int BN, int ROWS, bool SWIGLU>
static int launch_f32_any(const F32Args& p, int segments, cudaStream_t stream) {
    return p.whole ? launch_f32<BN, ROWS, SWIGLU, true>(p, segments, stream) : launch_f32<BN, ROWS, SWIGLU, false>(p, segments, stream);
}

// The tile with the least time by cycles per 64 k that fit what was measured: 11 for a row of either operand, 15 for a token, 600
// besides; a round of CTAs costs 5,000 more.  32 weight rows per CTA (64 with SwiGLU) pay where there are few tiles: 1 row by
// 2,048 x 1,536 takes 25 us so and 33 with 128.  The sums do not depend on the choice.
int gemm_f32_run(F32Args p, cudaStream_t stream) {
    int device = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return (int)e;
    const bool swiglu = p.W2 != nullptr;
    int segments = (p.K + F32_SEGMENT - 1) / F32_SEGMENT;
    if (segments > F32_MAX_SEGMENTS) segments = F32_MAX_SEGMENTS;
    const long long places = clusters_at_once(segments, 1, sms), blocks = ((p.K + F32_BK - 1) / F32_BK + segments - 1) / segments;
    double least = -1;
    const int few = swiglu ? 64 : 32;
    for (int rows = F32_ROWS; rows >= few; rows = rows > few ? few : 0)
        for (int width = rows == F32_ROWS ? F32_MAX_TOKENS : 32; width >= 16; width -= 16) {
            if (width > 16 && width - 16 >= p.M) continue;
            const int features = swiglu ? rows / 2 : rows;
            const long long tiles = (long long)((p.N + features - 1) / features) * ((p.M + width - 1) / width);
            const double block = 600 + 11.0 * (rows + width) + 15.0 * width;
            const double cost = (double)((tiles + places - 1) / places) * ((double)blocks * block + 5000);
            if (least < 0 || cost < least) least = cost, p.width = width, p.rows = rows;
        }
    if (p.rows < F32_ROWS)  // (with tiles of up to 32 tokens)
        return swiglu ? launch_f32_any<32, 64, true>(p, segments, stream) : launch_f32_any<32, 32, false>(p, segments, stream);
    if (p.width <= 32) return swiglu ? launch_f32_any<32, 128, true>(p, segments, stream) : launch_f32_any<32, 128, false>(p, segments, stream);
    return swiglu ? launch_f32_any<F32_MAX_TOKENS, 128, true>(p, segments, stream) : launch_f32_any<F32_MAX_TOKENS, 128, false>(p, segments, stream);
}

CW_TRACE_TU(gemm_f32)
