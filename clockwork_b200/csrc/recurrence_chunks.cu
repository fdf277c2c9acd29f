// Recurrences with one decay per head and token, a chunk of CK tokens of a portion at a time.  Per head, with S [Dk, Dv]:
//
//   S <- a S + k u^T,  y = q_scale S^T q (+ skip v)     u = b v            (state-space, constant decays, a matrix memory)
//                                                       u = b (v - a S^T k)  (the gated delta rule)
//
// What the scans of recurrence.cu and recurrence_gated.cu do token by token is, for the tokens of a chunk and the state S that it
// begins with,
//   delta:  u_t = b_t v_t - b_t A_t S^T k_t - sum over s < t of G_ts u_s          G_ts = b_t c_ts (k_t . k_s)
//   y_t = q_scale (A_t S^T q_t + sum over s <= t of c_ts (q_t . k_s) u_s)
//   S  <- A_last S + sum of W_t k_t u_t
// with c_ts the product of the decays s + 1 .. t, A_t that of all up to t and W_t that of all behind t.  What stands beside S and u
// belongs to a head and not to a value column: chunk_gram_kernel makes it for all chunks side by side.  The scan is then bound
// by what its four warps, one a scheduler, issue: reads of q and k from shared memory (a 16-byte read takes the pipe four cycles,
// whatever the lanes share; the pipe 44 % busy) and multiply-adds, two or three per token, channel and column (37 %; issue slots 54 %): a thread owns two value columns and eight key channels, so that a
// read serves eight multiply-adds, and the sums over the channels meet once per chunk.  With one column and 16 channels a thread
// it ran 148 us instead of the 113 below.  The token-by-token scans read q and k once per column (the pipe 70 % busy in the delta
// rule), which besides waits for four shuffles per token.
// The sums' order depends on where a portion's chunks begin, so a request's bits depend on how its tokens were cut into steps:
// float32 runs, which promise that they do not, and steps of single tokens keep to the token-by-token scans.
// Measured (B200): delta rule, 1,024 tokens, 16 heads of 128 x 128: 202 -> 113 us (and 16 for what belongs to the heads); state space, portions of 900, 333 and 65 tokens,
// 64 heads of 128 x 64 that share q and k: 337 -> 161 us (and 19).
#include "request_tiles.cuh"

#define CK 16        // tokens of a chunk, and value columns of a block
#define CK_SMEM CW_SCAN_ALONE  // the most that a launch asks for
#define CK_WORDS 36  // per token s and head: G_ts of every t [16]; per token t: q_scale c_ts (q_t . k_s) of every s [16]; four factors

struct ChunkArgs {
    const float *q, *k, *v;  // rows of ldq, ldk, ldv floats: head h reads group h / heads_per_group of q and k
    int ldq, ldk, ldv;
    const float *a, *b;      // decays [N, lda] (lda 0: one row for all tokens) and input factors [N, ldb] (null: one), a column per head
    int lda, ldb;
    const float* skip;       // [H] or null
    float q_scale;
    int ones;                // the last value column is not in v: its input is one for every token
    float* state;            // S of head h: [Dv][Dk] at state_off + h Dv Dk of the request's slot
    long long state_stride, state_off;
    const long long* slots;
    const int *tok_seq, *q_start;
    int S, H, Dk, Dv, heads_per_group;
    int from;                // requests of fewer tokens are left alone (the token-by-token scans take them)
    float* out;              // [N, H Dv]
    float* gram;             // [N, H, CK_WORDS]
    // rows of `carry` [N, ldc] (C columns) whose last R of every portion go to the request's state at carry_off (null: none)
    const float* carry;
    int ldc, C, R;
    long long carry_off;
};

#define CK_HEADS 8  // heads of a group that a block of the kernel below makes the factors for
// A block per chunk of a request and up to CK_HEADS heads that share q and k; a thread per pair of tokens.
__global__ void __launch_bounds__(CK * CK) chunk_gram_kernel(const ChunkArgs p, int delta) {
    extern __shared__ __align__(16) float gram_smem[];  // k [CK][Dk + 4], q the same
    __shared__ int tile_row, tile_rows;
    __shared__ float a_s[CK_HEADS][CK], b_s[CK_HEADS][CK];
    const int splits = (p.heads_per_group + CK_HEADS - 1) / CK_HEADS, group = blockIdx.y / splits;
    const int h0 = group * p.heads_per_group + blockIdx.y % splits * CK_HEADS, heads = min(CK_HEADS, (group + 1) * p.heads_per_group - h0);
    const int tid = threadIdx.x, Dk = p.Dk, ld = Dk + 4;
    pdl_enter();
    if (tid < 32) {
        const RowTile tile = find_row_tile(blockIdx.x, false, p.q_start, p.tok_seq, p.S, 1, CK, p.from);
        if (tid == 0) tile_row = tile.row0, tile_rows = tile.seq < 0 ? 0 : tile.rows;
    }
    __syncthreads();
    const int row0 = tile_row, n = tile_rows;
    if (n == 0) return;
    float *ks = gram_smem, *qs = ks + CK * ld;
    const size_t column = (size_t)group * Dk;
    for (int e = tid; e < n * (Dk >> 2); e += CK * CK) {
        const int t = e / (Dk >> 2), i = (e - t * (Dk >> 2)) << 2;
        *(float4*)(ks + t * ld + i) = *(const float4*)(p.k + (size_t)(row0 + t) * p.ldk + column + i);
        *(float4*)(qs + t * ld + i) = *(const float4*)(p.q + (size_t)(row0 + t) * p.ldq + column + i);
    }
    if (tid < heads * CK) {
        const int x = tid / CK, t = tid % CK;
        if (t < n) {
            a_s[x][t] = p.a[(size_t)(row0 + t) * p.lda + h0 + x];
            b_s[x][t] = p.b != nullptr ? p.b[(size_t)(row0 + t) * p.ldb + h0 + x] : 1.f;
        }
    }
    __syncthreads();
    const int t = tid / CK, s = tid % CK;
    const bool pair = s <= t && t < n;
    float kk[2] = {0.f, 0.f}, qk[2] = {0.f, 0.f};
    if (pair) {
        for (int i = 0; i < Dk; i += 4) {
            const float4 x = *(const float4*)(ks + s * ld + i), z = *(const float4*)(qs + t * ld + i);
            qk[0] = fmaf(x.x, z.x, qk[0]);
            qk[1] = fmaf(x.y, z.y, qk[1]);
            qk[0] = fmaf(x.z, z.z, qk[0]);
            qk[1] = fmaf(x.w, z.w, qk[1]);
            if (delta) {
                const float4 y = *(const float4*)(ks + t * ld + i);
                kk[0] = fmaf(x.x, y.x, kk[0]);
                kk[1] = fmaf(x.y, y.y, kk[1]);
                kk[0] = fmaf(x.z, y.z, kk[0]);
                kk[1] = fmaf(x.w, y.w, kk[1]);
            }
        }
    }
    const float kq = qk[0] + qk[1], k2 = kk[0] + kk[1];
    const size_t step = (size_t)p.H * CK_WORDS;
    for (int x = 0; x < heads; ++x) {
        float c = 1.f;
        if (pair)
            for (int r = s + 1; r <= t; ++r) c *= a_s[x][r];
        float* rows = p.gram + ((size_t)row0 * p.H + h0 + x) * CK_WORDS;
        if (delta && s < n) rows[s * step + t] = pair && s < t ? b_s[x][t] * c * k2 : 0.f;
        if (t >= n) continue;
        rows[t * step + CK + s] = pair ? p.q_scale * c * kq : 0.f;
        if (s == 0) {
            float upto = 1.f, behind = 1.f;
            for (int r = 0; r <= t; ++r) upto *= a_s[x][r];
            for (int r = t + 1; r < n; ++r) behind *= a_s[x][r];
            *(float4*)(rows + t * step + 2 * CK) = make_float4(upto, behind, delta ? b_s[x][t] * upto : p.q_scale * upto, b_s[x][t]);
        }
    }
}

__device__ __forceinline__ void ck_cp16(float* smem, const float* gmem) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(gmem) : "memory");
}
__device__ __forceinline__ void ck_cp4(float* smem, const float* gmem) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(gmem) : "memory");
}

// Heads of Dk channels, blocks of Dk threads: columns 2 (tid % 8) and the next, channels 8 (tid / 8) ..
template <int Dk, bool DELTA>
__global__ void __launch_bounds__(Dk) chunk_scan_kernel(const ChunkArgs p) {
    constexpr int NW = Dk / 32, TP = 8 * CK / Dk;                 // TP: tokens (of its two columns) that a thread sums up and writes
    constexpr int SUMS = DELTA ? 2 : 1;                            // S^T q, S^T k
    constexpr int BUF = 2 * CK * Dk + CK * CK + CK * CK_WORDS;    // q, k, v, gram
    extern __shared__ __align__(16) float cs_smem[];
    float* sums = cs_smem + 2 * BUF;         // [NW][SUMS][token][column]
    float* us = sums + NW * SUMS * CK * CK;  // [token][column]: what a token writes, before what the chunk's earlier ones take off
    float* ws = us + CK * CK;                // [token] W
    const int seq = blockIdx.z, h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_enter();
    const int start = p.q_start[seq], end = p.q_start[seq + 1];
    if (end <= start || end - start < p.from) return;
    const int Dv = p.Dv, c = (tid & 7) * 2, grp = tid >> 3, j0 = blockIdx.x * CK, j = j0 + c;
    const bool live[2] = {j < Dv, j + 1 < Dv};
    const int ldo = p.H * Dv;
    float* out = p.out + (size_t)h * Dv + j;
    if (p.tok_seq[start] < 0) {  // padding rows of a fixed-shape step: no request, no state
        for (int t = start + grp; t < end; t += Dk / 8)
            for (int x = 0; x < 2; ++x)
                if (live[x]) out[(size_t)t * ldo + x] = 0.f;
        return;
    }
    float* row_state = p.state + p.slots[seq] * p.state_stride;
    float* S_mem = row_state + p.state_off + ((size_t)h * Dv + j) * Dk + grp * 8;
    float S[2][8];
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int r = 0; r < 8; ++r) S[x][r] = live[x] ? S_mem[x * Dk + r] : 0.f;
    const float skip = p.skip != nullptr ? p.skip[h] : 0.f;
    const size_t group = (size_t)(h / p.heads_per_group) * Dk;
    const int Dvin = p.ones ? Dv - 1 : Dv;  // value columns that v holds
    const float *qp = p.q + group, *kp = p.k + group, *vp = p.v + (size_t)h * Dvin + j0, *gp = p.gram + (size_t)h * CK_WORDS;
    auto fetch = [&](int t0, float* buf) {  // tokens t0 .. t0 + CK - 1; zeros behind the portion's end
        float *qs = buf, *ks = buf + CK * Dk, *vs = buf + 2 * CK * Dk, *gs = vs + CK * CK;
        const int n = min(CK, end - t0);
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const int e = tid + it * Dk, t = e / (Dk / 4), i = (e % (Dk / 4)) * 4;
            if (t < n) {
                ck_cp16(qs + t * Dk + i, qp + (size_t)(t0 + t) * p.ldq + i);
                ck_cp16(ks + t * Dk + i, kp + (size_t)(t0 + t) * p.ldk + i);
            } else {
                *(float4*)(qs + t * Dk + i) = *(float4*)(ks + t * Dk + i) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
#pragma unroll
        for (int it = 0; it < CK * CK / Dk; ++it) {
            const int e = tid + it * Dk, t = e >> 4, x = e & 15;
            if (t < n && j0 + x < Dvin)
                ck_cp4(vs + e, vp + (size_t)(t0 + t) * p.ldv + x);
            else
                vs[e] = t < n && p.ones && j0 + x == Dv - 1 ? 1.f : 0.f;
        }
        for (int e = tid; e < CK * (CK_WORDS / 4); e += Dk) {
            const int t = e / (CK_WORDS / 4), i = (e % (CK_WORDS / 4)) * 4;
            if (t < n)
                ck_cp16(gs + t * CK_WORDS + i, gp + (size_t)(t0 + t) * p.H * CK_WORDS + i);
            else
                *(float4*)(gs + t * CK_WORDS + i) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(start, cs_smem);
    if (p.carry != nullptr) {  // the blocks of the request share its channels out
        const int n = end - start, block = blockIdx.y * gridDim.x + blockIdx.x, blocks = gridDim.y * gridDim.x;
        float* kept = row_state + p.carry_off;
        for (int x = block * Dk + tid; x < p.C; x += blocks * Dk)
            for (int d = p.R; d >= 1; --d)  // ascending writes; what is read lies ahead of what was written
                kept[(size_t)(p.R - d) * p.C + x] =
                    d <= n ? p.carry[(size_t)(end - d) * p.ldc + x] : kept[(size_t)(p.R - (d - n)) * p.C + x];
    }
    int which = 0;
    for (int t0 = start; t0 < end; t0 += CK, which ^= 1) {
        const int n = min(CK, end - t0);
        const float *qs = cs_smem + which * BUF, *ks = qs + CK * Dk, *vs = ks + CK * Dk, *gs = vs + CK * CK;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // this chunk has landed; everyone has left the other buffer
        if (t0 + CK < end) fetch(t0 + CK, cs_smem + (which ^ 1) * BUF);
        float part[SUMS * 2][CK];  // the thread's channels of S^T q_t and S^T k_t, two columns each
#pragma unroll
        for (int t = 0; t < CK; ++t) {
#pragma unroll
            for (int x = 0; x < SUMS; ++x) {
                const float* from = (x == 0 ? qs : ks) + t * Dk + grp * 8;
                const float4 lo = *(const float4*)from, hi = *(const float4*)(from + 4);
#pragma unroll
                for (int col = 0; col < 2; ++col) {
                    float e0 = S[col][0] * lo.x, e1 = S[col][1] * lo.y;
                    e0 = fmaf(S[col][2], lo.z, e0);
                    e1 = fmaf(S[col][3], lo.w, e1);
                    e0 = fmaf(S[col][4], hi.x, e0);
                    e1 = fmaf(S[col][5], hi.y, e1);
                    e0 = fmaf(S[col][6], hi.z, e0);
                    e1 = fmaf(S[col][7], hi.w, e1);
                    part[2 * x + col][t] = e0 + e1;
                }
            }
        }
        // the four groups of lanes of a warp that hold the same columns: each is left with four of the tokens
        const bool up16 = lane & 16, up8 = lane & 8;
#pragma unroll
        for (int x = 0; x < 2 * SUMS; ++x) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float got = __shfl_xor_sync(0xffffffffu, up16 ? part[x][i] : part[x][i + 8], 16);
                part[x][i] = (up16 ? part[x][i + 8] : part[x][i]) + got;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float got = __shfl_xor_sync(0xffffffffu, up8 ? part[x][i] : part[x][i + 4], 8);
                part[x][i] = (up8 ? part[x][i + 4] : part[x][i]) + got;
            }
        }
#pragma unroll
        for (int x = 0; x < SUMS; ++x)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                *(float2*)(sums + ((warp * SUMS + x) * CK + (up16 ? 8 : 0) + (up8 ? 4 : 0) + i) * CK + c) = make_float2(part[2 * x][i], part[2 * x + 1][i]);
        __syncthreads();
        float y[TP][2];
#pragma unroll
        for (int i = 0; i < TP; ++i) {  // this thread's tokens: grp, grp + Dk / 8, ..
            const int t = grp + i * (Dk / 8);
            float2 e = make_float2(0.f, 0.f), d = e;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                const float2 v = *(const float2*)(sums + (w * SUMS * CK + t) * CK + c);
                e.x += v.x;
                e.y += v.y;
                if (DELTA) {
                    const float2 v2 = *(const float2*)(sums + ((w * SUMS + 1) * CK + t) * CK + c);
                    d.x += v2.x;
                    d.y += v2.y;
                }
            }
            const float4 f = *(const float4*)(gs + t * CK_WORDS + 2 * CK);  // A, W, b A or q_scale A, b
            const float2 v = *(const float2*)(vs + t * CK + c);
            *(float2*)(us + t * CK + c) = DELTA ? make_float2(fmaf(-f.z, d.x, f.w * v.x), fmaf(-f.z, d.y, f.w * v.y)) : make_float2(f.w * v.x, f.w * v.y);
            y[i][0] = DELTA ? f.x * e.x : fmaf(f.z, e.x, skip * v.x);
            y[i][1] = DELTA ? f.x * e.y : fmaf(f.z, e.y, skip * v.y);
            if (c == 0) ws[t] = f.y;
        }
        __syncthreads();
        float u[2][CK];
#pragma unroll
        for (int t = 0; t < CK; ++t) {
            const float2 v = *(const float2*)(us + t * CK + c);
            u[0][t] = v.x;
            u[1][t] = v.y;
        }
        if (DELTA) {
#pragma unroll
            for (int s = 0; s + 1 < CK; ++s)
#pragma unroll
                for (int t4 = (s + 1) & ~3; t4 < CK; t4 += 4) {
                    const float4 g = *(const float4*)(gs + s * CK_WORDS + t4);
                    const float gt[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (t4 + i > s) {
                            u[0][t4 + i] = fmaf(-gt[i], u[0][s], u[0][t4 + i]);
                            u[1][t4 + i] = fmaf(-gt[i], u[1][s], u[1][t4 + i]);
                        }
                }
        }
#pragma unroll
        for (int i = 0; i < TP; ++i) {
            const int t = grp + i * (Dk / 8);
            const float* row = gs + t * CK_WORDS + CK;
            float y1[2] = {0.f, 0.f};
#pragma unroll
            for (int s = 0; s < CK; s += 4) {
                const float4 w = *(const float4*)(row + s);
#pragma unroll
                for (int col = 0; col < 2; ++col) {  // (later tokens are left out, not multiplied by zero: theirs may be no numbers)
                    if (s <= t) y[i][col] = fmaf(w.x, u[col][s], y[i][col]);
                    if (s + 1 <= t) y1[col] = fmaf(w.y, u[col][s + 1], y1[col]);
                    if (s + 2 <= t) y[i][col] = fmaf(w.z, u[col][s + 2], y[i][col]);
                    if (s + 3 <= t) y1[col] = fmaf(w.w, u[col][s + 3], y1[col]);
                }
            }
#pragma unroll
            for (int col = 0; col < 2; ++col)
                if (live[col] && t < n) out[(size_t)(t0 + t) * ldo + col] = y[i][col] + y1[col];
        }
        const float last = gs[(n - 1) * CK_WORDS + 2 * CK];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            S[0][r] *= last;
            S[1][r] *= last;
        }
#pragma unroll
        for (int t4 = 0; t4 < CK; t4 += 4) {
            const float4 w = *(const float4*)(ws + t4);
            const float wt[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float* from = ks + (t4 + i) * Dk + grp * 8;
                const float4 lo = *(const float4*)from, hi = *(const float4*)(from + 4);
#pragma unroll
                for (int col = 0; col < 2; ++col) {
                    const float wu = wt[i] * u[col][t4 + i];
                    S[col][0] = fmaf(lo.x, wu, S[col][0]);
                    S[col][1] = fmaf(lo.y, wu, S[col][1]);
                    S[col][2] = fmaf(lo.z, wu, S[col][2]);
                    S[col][3] = fmaf(lo.w, wu, S[col][3]);
                    S[col][4] = fmaf(hi.x, wu, S[col][4]);
                    S[col][5] = fmaf(hi.y, wu, S[col][5]);
                    S[col][6] = fmaf(hi.z, wu, S[col][6]);
                    S[col][7] = fmaf(hi.w, wu, S[col][7]);
                }
            }
        }
    }
#pragma unroll
    for (int x = 0; x < 2; ++x)
        if (live[x]) {
#pragma unroll
            for (int r = 0; r < 8; ++r) S_mem[x * Dk + r] = S[x][r];
        }
}

template <int Dk, bool DELTA>
static int launch_chunks(const ChunkArgs& p, long long rows, cudaStream_t stream) {
    const dim3 grid((p.Dv + CK - 1) / CK, p.H, p.S);
    const size_t need = sizeof(float) * (size_t)(2 * (2 * CK * Dk + CK * CK + CK * CK_WORDS) + (Dk / 32 * (DELTA ? 2 : 1) + 1) * CK * CK + CK);
    static_assert(CK_SMEM >= sizeof(float) * (2 * (2 * CK * Dk + CK * CK + CK * CK_WORDS) + (Dk / 32 * 2 + 1) * CK * CK + CK), "what a block needs");
    const size_t smem = cw_scan_smem(need, rows, (long long)grid.x * grid.y);
    const cudaError_t e = cudaFuncSetAttribute(chunk_scan_kernel<Dk, DELTA>, cudaFuncAttributeMaxDynamicSharedMemorySize, CK_SMEM);
    if (e != cudaSuccess) return (int)e;
    return cw_launch(chunk_scan_kernel<Dk, DELTA>, grid, dim3(Dk), smem, stream, 1, p);
}

// rows: the rows of the step.  from: requests of fewer tokens are left alone.  delta: the second form above (no skip, q_scale 1, no column of ones).  Heads of 32, 64 or 128
// channels, rows of q and k whole 16-byte pieces at 16-byte addresses (CW_ERR_UNSUPPORTED otherwise).  gram: rows * H * 36
// floats of scratch.
extern "C" int cw_chunk_scan(int delta, const float* q, int ldq, const float* k, int ldk, const float* v, int ldv, const float* a, int lda,
                             const float* b, int ldb, const float* skip, float q_scale, int ones, float* state, long long state_stride,
                             long long state_off, const long long* slots, const int* tok_seq, const int* q_start, int S, int H, int Dk,
                             int Dv, int heads_per_group, int from, float* out, float* gram, const float* carry, int ldc, int C, int R,
                             long long carry_off, int rows, cudaStream_t stream) {
    if (S == 0 || rows == 0) return CW_OK;
    if (S < 0 || rows < 0 || H <= 0 || Dk <= 0 || Dv <= (ones ? 1 : 0) || heads_per_group <= 0 || H % heads_per_group) return CW_ERR_BAD_SIZE;
    if (carry != nullptr && (C <= 0 || R < 0 || ldc < C)) return CW_ERR_BAD_SIZE;
    if (delta && (skip != nullptr || q_scale != 1.f || ones)) return CW_ERR_UNSUPPORTED;
    if ((Dk != 32 && Dk != 64 && Dk != 128) || ldq % 4 || ldk % 4 || (((uintptr_t)q | (uintptr_t)k | (uintptr_t)gram) & 15) || H > 65535 || S > 65535)
        return CW_ERR_UNSUPPORTED;
    const ChunkArgs p = {q, k, v, ldq, ldk, ldv, a, b, lda, ldb, skip, q_scale, ones, state, state_stride, state_off, slots, tok_seq, q_start,
                         S, H, Dk, Dv, heads_per_group, from, out, gram, R > 0 ? carry : nullptr, ldc, C, R, carry_off};
    const int chunks = (rows + CK - 1) / CK + (rows < S ? rows : S);
    const int err = cw_launch(chunk_gram_kernel, dim3(chunks, H / heads_per_group * ((heads_per_group + CK_HEADS - 1) / CK_HEADS)), dim3(CK * CK), sizeof(float) * 2 * CK * (Dk + 4), stream, 1, p, delta);
    if (err != CW_OK) return err;
#define CK_GO(D) return delta ? launch_chunks<D, true>(p, rows, stream) : launch_chunks<D, false>(p, rows, stream)
    switch (Dk) {
        case 32: CK_GO(32);
        case 64: CK_GO(64);
        default: CK_GO(128);
    }
#undef CK_GO
}

CW_TRACE_TU(recurrence_chunks)
