// Float32 products on the 5th-generation tensor cores, as exact as on the CUDA cores.
//
// A float32 number is the sum of three bfloat16 numbers: w = w0 + w1 + w2, x = x0 + x1 + x2, the first of 6 bits, the second of 8,
// both rounded, the third what is left, 8 bits at most.  The second comes times 2^8, the third times 2^16, so that none of it falls
// below bfloat16's range: the parts of every finite number are the number.  The tensor cores form w0 x0 and the seven products
// w1 x0, w0 x1 | w1 x1, w2 x0, w0 x2 | w1 x2, w2 x1 exactly and add them up in float32, cutting off what falls below the last bit;
// w2 x2, at most 2^-30 of w0 x0, is left out.  So that little falls off, w0 x0 (12 bits, a sum of which mostly fits whole) has an
// accumulator of its own for every 16 k, the small products three by their factor, 2^8, 2^16 and 2^24, for 64 k; per 64 k the four
// are read out of tensor memory, added in pairs, and the pairs are added into a running sum that carries its rounding errors
// along (Kahan); the small ones join what it carries.  Outputs that are not finite are formed again by fmaf (f32_plain).
// Root mean square of the error over the sum of the products' magnitudes, in 2^-24 (B200, 200 x 4,000 outputs six times, K 64,
// 1,536 and 8,960), this kernel and the chains of 16 fmaf with the same running sum that it replaced:
//   normal operands          0.093 0.025 0.010   chains 0.261 0.055 0.024
//   sizes spread over e      0.250 0.091 0.041          0.475 0.139 0.064
//   sizes spread over e^3    0.754 0.638 0.543          0.931 0.672 0.563
//   one sign                 0.494 0.336 0.417          0.732 0.349 0.444
//   between 0 and 1          0.478 0.391 0.529          0.720 0.402 0.562
// Tried: first parts of 8 bits, one sign 0.45 at K of 1,536; all four of w0 x0 and the small ones carried along one by one, 10 % less
// of an error and 296 us instead of 242 for [gate, up] of 200 rows.
//
// Every output's sum has the same order whatever M, N or the tile it falls in, so a row's result does not depend on the rest of
// the batch: 64 k at a time, a long K cut into segments of about F32_SEGMENT by K alone, each segment on a CTA of a cluster;
// the CTAs leave sums and what they lost in shared memory, share the outputs among them and add the segments up in order.
//
// A CTA: up to 128 weight rows (the MMA's M) by up to 64 tokens (its N).  Eight warps copy the operands' next 64 k into
// shared memory, cut them in three and store them there as the MMAs read them (K-major, 128-byte swizzle), two stages;
// a thread of another issues the MMAs.  The parts of the token rows follow one another, so that one MMA of two or three times the width
// forms w1 [x0 | x1 | x2], w2 [x0 | x1] or w0 [x1 | x2]: 16 MMAs per 64 k, none of which takes less than about 64 cycles however narrow.
// Eight other warps read out and add up what has been formed.  What bounds it: few rows, the 16 MMAs in a row (about 1,600 cycles per
// 64 k); many, the latencies of copying, cutting and adding with two warps of each a scheduler (issue slots 53 % busy, shared-memory
// pipe 36 %, tensor pipe 18 %; [gate, up] of 200 rows takes 214 us without the cutting and the carried errors).
// Measured (B200, us, chains of fmaf -> this): 200 rows, [gate, up] 2 x 8,960 by 1,536 373 -> 242, 1,536 by 8,960 219 -> 150, 2,048 by
// 1,536 64 -> 39; 64 rows 170 -> 70, 108 -> 47, 33 -> 29; 8 rows 39 -> 37, 37 -> 33, 27 -> 27; 1 row 37 -> 37, 36 -> 33, 27 -> 25.
// Tried: the same eight warps for both jobs, one after the other: every step's latency in a row.
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

// Two floats in one 64-bit register: an instruction for both (the issue slots bound this kernel).
typedef unsigned long long float_pair;
__device__ __forceinline__ float_pair pair_of(uint32_t x, uint32_t y) {
    float_pair v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(x), "r"(y));
    return v;
}
__device__ __forceinline__ void apart(float_pair v, uint32_t& x, uint32_t& y) { asm("mov.b64 {%0, %1}, %2;" : "=r"(x), "=r"(y) : "l"(v)); }
__device__ __forceinline__ float_pair pair_add(float_pair a, float_pair b) {
    float_pair v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ float_pair pair_sub(float_pair a, float_pair b) {
    float_pair v;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ float_pair pair_mul(float_pair a, float_pair b) {
    float_pair v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ float_pair pair_fma(float_pair a, float_pair b, float_pair c) {
    float_pair v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
    return v;
}
__device__ __forceinline__ float_pair both(float x) { return pair_of(__float_as_uint(x), __float_as_uint(x)); }
__device__ __forceinline__ void pair_add(float_pair& sum, float_pair& lost, float_pair x) {  // f32_add
    const float_pair y = pair_sub(x, lost);
    const float_pair t = pair_add(sum, y);
    lost = pair_sub(pair_sub(t, sum), y);
    sum = t;
}

// The first 6 of a float's 24 bits, rounded (half a step away from zero).
__device__ __forceinline__ uint32_t first6(uint32_t x) { return (x + 0x20000u) & 0xfffc0000u; }
// Of two floats, the upper halves side by side.
__device__ __forceinline__ uint32_t upper2(uint32_t x, uint32_t y) { return __byte_perm(x, y, 0x7632); }

// The three parts of two numbers, as bfloat16 side by side; the second comes times 2^8, the third times 2^16.  The parts of numbers
// from 2^126 on may be infinite: see f32_plain().
__device__ __forceinline__ void three_parts(uint32_t x, uint32_t y, uint32_t& q0, uint32_t& q1, uint32_t& q2) {
    const uint32_t x0 = first6(x), y0 = first6(y);
    q0 = upper2(x0, y0);
    const float_pair rest = pair_mul(pair_sub(pair_of(x, y), pair_of(x0, y0)), both(256.f));
    uint32_t u, v;
    apart(rest, u, v);
    const __nv_bfloat162 rounded = __floats2bfloat162_rn(__uint_as_float(u), __uint_as_float(v));
    q1 = *reinterpret_cast<const uint32_t*>(&rounded);
    apart(pair_mul(pair_sub(rest, pair_of(q1 << 16, q1 & 0xffff0000u)), both(256.f)), u, v);
    q2 = upper2(u, v);  // (whole: 8 bits at most are left)
}

// The product of two rows by fmaf, 16 k at a time: for the outputs that are not finite.  Parts of an infinite operand are no numbers, and
// those of the largest ones are infinite, where the product may be infinite, or finite.
__device__ __noinline__ float f32_plain(const float* a, const float* w, int K) {
    float sum = 0.f, lost = 0.f;
    for (int k0 = 0; k0 < K; k0 += 16) {
        float chain = 0.f;
        for (int k = k0; k < min(K, k0 + 16); ++k) chain = fmaf(a[k], w[k], chain);
        f32_add(sum, lost, chain);
    }
    return sum;
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
    if (!isfinite(v)) v = f32_plain(p.A + (size_t)m * p.lda, p.W + (size_t)n * p.K, p.K);
    if (SWIGLU && !isfinite(up)) up = f32_plain(p.A + (size_t)m * p.lda, p.W2 + (size_t)n * p.K, p.K);
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
    // Tensor memory: four accumulators of w0 x0 and three of the small products, twice where there is room, so that the next 64 k's
    // are formed while these are read out.
    static constexpr int SETS = BN <= 32 ? 2 : 1, SMALL = SETS * 4 * BN, TMEM_COLS = 512;
    // Pieces of eight numbers of 64 k that a converting thread brings, and how many times 64 k it has on their way: as many as there
    // is room for (few rows per CTA are bound by the latency of these copies).
    static constexpr int W_PIECES = ROWS * 8 / (32 * F32_CONVERTERS), PIECES = W_PIECES + (BN * 8 + 32 * F32_CONVERTERS - 1) / (32 * F32_CONVERTERS);
    static constexpr int ROOM = (226 * 1024 - 1280 - 2 * STAGE) / (PIECES * 1024 * F32_CONVERTERS);
    static constexpr int AHEAD = ROOM < 6 ? ROOM : 6;
    static constexpr int RAW = AHEAD * PIECES * 32 * F32_CONVERTERS * 32;
    static constexpr int SMEM = 2 * STAGE + RAW + 1024 + 256;
    static_assert(SETS * 7 * BN <= TMEM_COLS && BN % 32 == 0, "accumulators");
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

    // Registers: 640 threads of 96 at launch, 61,440 in all; 256 x 152 + 256 x 72 + 128 x 32 of them after the split (tiles of up to 32
    // tokens 144 and 80, with which their loops keep everything in registers).
    constexpr int ADDER_REGS = BN <= 32 ? 144 : 152, CONVERTER_REGS = BN <= 32 ? 80 : 72;
    static_assert(32 * (F32_ADDERS * ADDER_REGS + F32_CONVERTERS * CONVERTER_REGS) + (F32_THREADS - 32 * (F32_ADDERS + F32_CONVERTERS)) * 32 <= F32_THREADS * 96,
                  "the split draws on the registers of the launch");
    if (warp >= F32_ADDERS + F32_CONVERTERS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        if (warp == F32_ADDERS + F32_CONVERTERS && elect_one()) {
            // ---- MMA issuer ------------------------------------------------------------------------------------------
            const int x_part = groups * 16 * F32_BK * 2;
            const uint32_t wide = 16 * groups, idesc = instr_desc(F32_ROWS, wide), idesc2 = instr_desc(F32_ROWS, 2 * wide), idesc3 = instr_desc(F32_ROWS, 3 * wide);
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
                const uint32_t small = tmem + C::SMALL + set * 3 * BN;
#pragma unroll
                for (int k = 0; k < F32_BK / 16; ++k) umma_bf16(tmem + (set * 4 + k) * BN, w0 + 2 * k, x0 + 2 * k, idesc, 0u);
                umma_commit(first_full + 8 * set);
                ok = mbar_wait(small_empty + 8 * set, ((b / C::SETS) & 1) ^ 1, give_up);
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < F32_BK / 16; ++k) umma_bf16(small, w1 + 2 * k, x0 + 2 * k, idesc3, k > 0 ? 1u : 0u);
#pragma unroll
                for (int k = 0; k < F32_BK / 16; ++k) umma_bf16(small + wide, w2 + 2 * k, x0 + 2 * k, idesc2, 1u);
#pragma unroll
                for (int k = 0; k < F32_BK / 16; ++k) umma_bf16(small, w0 + 2 * k, x1 + 2 * k, idesc2, 1u);
                umma_commit(empty0 + 8 * (b & 1));  // the stage has been read
                umma_commit(small_full + 8 * set);
            }
        }
        __syncwarp();
        if (segments > 1) {  // (the two that the others meet at below)
            f32_cluster_barrier();
            f32_cluster_barrier();
        }
    } else if (warp >= F32_ADDERS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(CONVERTER_REGS));
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
                uint4 x[2][2];
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (2 * at + h < C::PIECES) {
                        const float* from = raw + (b % C::AHEAD * C::PIECES + 2 * at + h) * 8 * NT;
                        x[h][0] = *reinterpret_cast<const uint4*>(from);
                        x[h][1] = *reinterpret_cast<const uint4*>(from + 4);
                    }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int i = 2 * at + h;
                    if (i >= C::PIECES || !has(i)) continue;
                    const uint32_t y[8] = {x[h][0].x, x[h][0].y, x[h][0].z, x[h][0].w, x[h][1].x, x[h][1].y, x[h][1].z, x[h][1].w};
                    uint32_t q[3][4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) three_parts(y[2 * j], y[2 * j + 1], q[0][j], q[1][j], q[2][j]);
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
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(ADDER_REGS));
        float_pair sum[C::MINE][8] = {}, lost[C::MINE][8] = {};  // [group][tokens]: this thread's feature, half of the groups of 16 tokens
        const int quarter = warp & 3, half = (groups + 1) >> 1, group0 = (warp >> 2) * half, mine_groups = min(half, groups - group0);
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16) + 16 * group0;
        bool ok = true;
        auto add_up = [&](int b) {
            // One accumulator's columns of all groups are loaded before the first is used, and while the last ones are added: a load
            // from tensor memory takes about 200 cycles.
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
            auto each_pair = [&](auto f) {
#pragma unroll
                for (int g = 0; g < C::MINE; ++g)
                    if (g < mine_groups)
#pragma unroll
                        for (int j = 0; j < 8; ++j) f(g, j);
            };
            auto add = [&](uint32_t (&x)[C::MINE][16]) {
                each_pair([&](int g, int j) { pair_add(sum[g][j], lost[g][j], pair_of(x[g][2 * j], x[g][2 * j + 1])); });
            };
            auto plus = [&](uint32_t (&x)[C::MINE][16], uint32_t (&y)[C::MINE][16]) {
                each_pair([&](int g, int j) {
                    apart(pair_add(pair_of(x[g][2 * j], x[g][2 * j + 1]), pair_of(y[g][2 * j], y[g][2 * j + 1])), x[g][2 * j], x[g][2 * j + 1]);
                });
            };
            auto later = [&](uint32_t (&x)[C::MINE][16], float less) {  // the small products join what the sum has lost
                each_pair([&](int g, int j) { lost[g][j] = pair_fma(pair_of(x[g][2 * j], x[g][2 * j + 1]), both(less), lost[g][j]); });
            };
            auto read_out = [&](uint32_t barrier) {  // this warp has read the accumulators
                tc_fence_before();
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(barrier) : "memory");
            };
            const int set = b % C::SETS;
            const uint32_t parity = (b / C::SETS) & 1, main0 = set * 4 * BN, small = C::SMALL + set * 3 * BN, wide = 16 * groups;
            ok = __all_sync(0xffffffffu, mbar_wait(first_full + 8 * set, parity, give_up));
            if (!ok) return;
            tc_fence_after();
            // (which two are added first says nothing about the error, but every bit of a step follows from it)
            load(t, main0);
            load(r, main0 + 2 * BN);
            landed(t);
            landed(r);
            plus(t, r);
            load(r, main0 + BN);
            add(t);
            load(t, main0 + 3 * BN);
            landed(t);
            landed(r);
            read_out(first_empty + 8 * set);
            plus(t, r);
            add(t);
            ok = __all_sync(0xffffffffu, mbar_wait(small_full + 8 * set, parity, give_up));
            if (!ok) return;
            tc_fence_after();
            load(t, small);
            load(r, small + wide);
            landed(t);
            landed(r);
            later(t, -0x1p-8f);
            load(t, small + 2 * wide);
            later(r, -0x1p-16f);
            landed(t);
            read_out(small_empty + 8 * set);
            later(t, -0x1p-24f);
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
                    uint32_t s[2], l[2];
                    apart(sum[g][j / 2], s[0], s[1]);
                    apart(lost[g][j / 2], l[0], l[1]);
                    if (g < half && t < tokens) f(t, __uint_as_float(s[j & 1]), __uint_as_float(l[j & 1]));
                }
        };
        if (segments == 1) {
            float* ups = (float*)smem;  // [token][64 features]
            if (SWIGLU) {
                if (mine && (quarter & 1)) each([&](int t, float s, float l) { ups[t * 64 + (quarter >> 1) * 32 + lane] = s - l; });
                asm volatile("bar.sync 1, %0;" ::"n"(32 * F32_ADDERS) : "memory");
            }
            const int n = n0 + (SWIGLU ? (quarter >> 1) * 32 + lane : row);
            if (mine && !(SWIGLU && (quarter & 1)) && n < p.N)
                each([&](int t, float s, float l) { f32_store<SWIGLU>(p, m0 + t, n, s - l, SWIGLU ? ups[t * 64 + (quarter >> 1) * 32 + lane] : 0.f); });
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
                        if (i < segments) {  // (the segments are alike in size: what either addend loses goes into `left`)
                            const float sum = __fadd_rn(total[u], s[i].x), of_total = __fsub_rn(sum, s[i].x), of_next = __fsub_rn(sum, of_total);
                            left = __fadd_rn(left, __fsub_rn(s[i].y, __fadd_rn(__fsub_rn(total[u], of_total), __fsub_rn(s[i].x, of_next))));
                            total[u] = sum;
                        }
                    total[u] -= left;
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
// besides; a round of CTAs costs 5,000 more (six products at 1 to 600 rows: within 5 % of the best tile, once 10 %).  32 or 64 weight
// rows per CTA pay where there are few tiles: 1 row by 2,048 x 1,536 takes 27 us with 32 and 35 with 128, 1 row by 1,536 x 8,960, five
// segments, 34 us with 64, whose 24 clusters all find a place at once, 41 with 128.  The sums do not depend on the choice.
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
    for (int rows = F32_ROWS; rows >= (swiglu ? 64 : 32); rows /= 2)
        for (int width = rows == F32_ROWS ? F32_MAX_TOKENS : 32; width >= 16; width -= 16) {
            if (width > 16 && width - 16 >= p.M) continue;
            const int features = swiglu ? rows / 2 : rows;
            const long long tiles = (long long)((p.N + features - 1) / features) * ((p.M + width - 1) / width);
            const double block = 600 + 11.0 * (rows + width) + 15.0 * width;
            const double cost = (double)((tiles + places - 1) / places) * ((double)blocks * block + 5000);
            if (least < 0 || cost < least) least = cost, p.width = width, p.rows = rows;
        }
    if (p.rows == 32) return launch_f32_any<32, 32, false>(p, segments, stream);  // (with tiles of up to 32 tokens, like the next two)
    if (p.rows == 64) return swiglu ? launch_f32_any<32, 64, true>(p, segments, stream) : launch_f32_any<32, 64, false>(p, segments, stream);
    if (p.width <= 32) return swiglu ? launch_f32_any<32, 128, true>(p, segments, stream) : launch_f32_any<32, 128, false>(p, segments, stream);
    return swiglu ? launch_f32_any<F32_MAX_TOKENS, 128, true>(p, segments, stream) : launch_f32_any<F32_MAX_TOKENS, 128, false>(p, segments, stream);
}

CW_TRACE_TU(gemm_f32)
