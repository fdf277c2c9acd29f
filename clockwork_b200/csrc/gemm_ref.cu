// Plain tiled matrix product on the CUDA cores with float32 accumulation:
//   C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]),   W in nn.Linear layout (clockwork/engine/model.py:58-60, 74-77)
// It is the matrix product of the true-float32 path (fmaf only, no tensor cores, no TF32) and
// the fallback of the bfloat16 path for sizes the tensor-core kernel refuses.
// Every output element is summed in the same fixed order whatever M, N or the tile it falls in, so
// a row's result does not depend on the rest of the batch: fmaf chains over 16 consecutive k, in
// ascending order, whose results are added up with a compensated (Kahan) running sum.  One plain
// chain over a long inner dimension would lose more than the 1e-5 that the float32 path is held
// to: at K = 8960 its rounding error alone is of that order; summed this way the result stays
// within a few units in the last place of the exact dot product at any K.
//
// Epilogues: 0 store as T; 1 add into a float32 matrix (the residual stream); 2 store float32
// (logits); 4 store max(v, 0)^2 as T.  The SwiGLU variant computes silu(A Wg^T) * (A Wu^T) (clockwork/engine/model.py:62-63).
//
// Two kernels with the same sums in the same order up to F32_SEGMENT, so the same bits there: gemm_f32_kernel for float32 operands
// whose rows are whole 16-byte pieces, and gemm_ref_kernel for everything else (bfloat16 operands, odd inner sizes or strides).
#include "attention_mma.cuh"

#define BM 64
#define BN 64
#define BK 16

// sum += x with the rounding error of earlier additions carried along in `lost` (Kahan's summation;
// the order of the operations matters and the compiler keeps it: no fast-math flags are used)
__device__ __forceinline__ void kahan_add(float& sum, float& lost, float x) {
    const float y = __fsub_rn(x, lost);
    const float t = __fadd_rn(sum, y);
    lost = __fsub_rn(__fsub_rn(t, sum), y);
    sum = t;
}

template <typename T, bool SWIGLU>
__global__ void __launch_bounds__(256)
gemm_ref_kernel(const T* __restrict__ A, const T* __restrict__ W, const T* __restrict__ W2,
                const float* __restrict__ bias, void* __restrict__ Cout, int M, int N, int K,
                int lda, int ldc, int epilogue) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    __shared__ float W2s[SWIGLU ? BK : 1][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float sum[4][4] = {}, lost[4][4] = {};    // running sums and what their roundings have lost so far
    float sum2[4][4] = {}, lost2[4][4] = {};
    for (int k0 = 0; k0 < K; k0 += BK) {
        float acc[4][4] = {};
        float acc2[4][4] = {};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = tid + i * 256;      // 0..1023
            const int r = e >> 4, c = e & 15; // row in tile, k in tile
            const int k = k0 + c;
            float a = 0.f, w = 0.f, w2 = 0.f;
            if (k < K) {
                if (m0 + r < M) a = to_f(A[(size_t)(m0 + r) * lda + k]);
                if (n0 + r < N) {
                    w = to_f(W[(size_t)(n0 + r) * K + k]);
                    if (SWIGLU) w2 = to_f(W2[(size_t)(n0 + r) * K + k]);
                }
            }
            As[c][r] = a;
            Ws[c][r] = w;
            if (SWIGLU) W2s[c][r] = w2;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[4], w[4], w2[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = Ws[k][tx * 4 + j];
            if (SWIGLU) {
#pragma unroll
                for (int j = 0; j < 4; ++j) w2[j] = W2s[k][tx * 4 + j];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
                    if (SWIGLU) acc2[i][j] = fmaf(a[i], w2[j], acc2[i][j]);
                }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                kahan_add(sum[i][j], lost[i][j], acc[i][j]);
                if (SWIGLU) kahan_add(sum2[i][j], lost2[i][j], acc2[i][j]);
            }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            float v = sum[i][j];
            if (bias) v += bias[n];
            const size_t idx = (size_t)m * ldc + n;
            if (SWIGLU) {
                const float g = v, u = sum2[i][j];
                ((T*)Cout)[idx] = from_f<T>(g / (1.0f + expf(-g)) * u);
            } else if (epilogue == 0) {
                ((T*)Cout)[idx] = from_f<T>(v);
            } else if (epilogue == 4) {  // the square of what is positive
                v = fmaxf(v, 0.f);
                ((T*)Cout)[idx] = from_f<T>(v * v);
            } else if (epilogue == 1) {
                ((float*)Cout)[idx] += v;
            } else {
                ((float*)Cout)[idx] = v;
            }
        }
    }
}

// float32 operands with rows of whole 16-byte pieces.  Bound by the multiply-adds and the instructions around them: 71 TFLOP/s
// is what independent fmaf chains reach on this part, four fifths of that with the compensated sum behind every 16 of them (issue
// slots 70 % busy, the multiply-add and the shared-memory pipe 54 % each).
// Operands stay in the order they have in memory ([row][k], rows of 16 k padded to 20 floats so that neither the copies nor the
// 16-byte reads meet in a bank) and come by cp.async, three steps of 16 k ahead; a thread keeps RM x RN outputs whose rows and
// columns are RY and RX apart and reads four k of each of its rows and columns at a time (RM + RN reads for 4 RM RN
// multiply-adds).  A long inner dimension is cut into segments of about F32_SEGMENT, each with a running sum of its own on a CTA
// of a cluster of its own; the CTAs leave sums and what they lost in shared memory, share the outputs among them and add
// the segments up in order, compensated like the rest.  How K is cut depends on K alone, so a row's bits still do not depend on
// the batch.  The kernel it replaced for these operands took a step at a time through registers and single-word reads.
// Measured (B200, 200 rows): [gate, up] 2 x 8,960 by 1,536: 1,343 -> 374 us; 1,536 by 8,960: 1,005 -> 218 us (341 uncut).
#define F32_K 16
#define F32_LD 20
#define F32_STAGES 4
#define F32_SEGMENT 1536
#define F32_MAX_SEGMENTS 8

__device__ __forceinline__ void copy16_or_zero(uint32_t to, const float* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ float2 load_of_rank(const void* mine, int rank) {  // the same place in another CTA of the cluster
    uint32_t there;
    float2 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(smem_addr(mine)), "r"(rank));
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(there) : "memory");
    return v;
}

struct F32Args {
    const float *A, *W, *W2, *bias;
    float* C;
    int M, N, K, lda, ldc, epilogue;
};

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

template <int TM, int TN, int RM, int RN, bool SWIGLU>
__global__ void __launch_bounds__((TM / RM) * (TN / RN)) gemm_f32_kernel(const F32Args p) {
    constexpr int RY = TM / RM, RX = TN / RN, NT = RY * RX;
    constexpr int COLS = SWIGLU ? TN / 2 : TN;  // output columns of a block (with SWIGLU its W rows are COLS of each matrix)
    constexpr int PIECES = (TM + TN) * (F32_K / 4), EACH = (PIECES + NT - 1) / NT;
    static_assert(NT % 4 == 0 && (!SWIGLU || RN % 2 == 0), "a thread's copies keep their place in the step; gate and up side by side");
    static_assert(TM * TN * 2 <= F32_STAGES * (TM + TN) * F32_LD, "the partial sums fit where the operands were");
    __shared__ __align__(16) float tile[F32_STAGES][TM + TN][F32_LD];
    const int tid = threadIdx.x, tx = tid % RX, ty = tid / RX;
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * COLS;
    const int all = (p.K + F32_K - 1) / F32_K, segments = gridDim.z, per = (all + segments - 1) / segments;
    const int first = min((int)blockIdx.z * per, all), steps = min(per, all - first);

    const float* from[EACH];  // where this thread's pieces of the next step are; null: rows outside (zeros)
    const int piece = (tid & 3) * 4;
#pragma unroll
    for (int i = 0; i < EACH; ++i) {
        const int r = (tid + i * NT) >> 2;
        from[i] = nullptr;
        if (r < TM) {
            if (m0 + r < p.M) from[i] = p.A + (size_t)(m0 + r) * p.lda;
        } else if (r < TM + TN) {
            const int n = n0 + (r - TM) % COLS;
            if (n < p.N) from[i] = (SWIGLU && r - TM >= COLS ? p.W2 : p.W) + (size_t)n * p.K;
        }
        if (from[i]) from[i] += first * F32_K + piece;
    }
    const uint32_t to0 = smem_addr(&tile[0][tid >> 2][piece]);
    int k_next = first * F32_K + piece;  // of the step that is fetched next
    auto fetch = [&](int step) {
        if (step < steps) {
            const uint32_t to = to0 + (step % F32_STAGES) * (int)sizeof(tile[0]);
            const bool inside = k_next < p.K;
#pragma unroll
            for (int i = 0; i < EACH; ++i) {
                if (PIECES % NT != 0 && i == EACH - 1 && tid + i * NT >= PIECES) break;
                const bool valid = inside && from[i];
                copy16_or_zero(to + i * (NT / 4) * F32_LD * 4, valid ? from[i] : p.A, valid);
                from[i] = from[i] ? from[i] + F32_K : nullptr;
            }
            k_next += F32_K;
        }
        cp_async_commit();  // (empty groups behind the last step keep the count of groups in flight)
    };

    float sum[RM][RN] = {}, lost[RM][RN] = {};
#pragma unroll
    for (int s = 0; s < F32_STAGES - 1; ++s) fetch(s);
    for (int step = 0; step < steps; ++step) {
        cp_async_wait<F32_STAGES - 2>();
        __syncthreads();  // step's tile is there for all, and all have left the stage that is written next
        fetch(step + F32_STAGES - 1);
        const float(*at)[F32_LD] = tile[step % F32_STAGES];
        float acc[RM][RN] = {};
#pragma unroll
        for (int q = 0; q < F32_K / 4; ++q) {
            float4 a[RM], w[RN];
#pragma unroll
            for (int i = 0; i < RM; ++i) a[i] = *reinterpret_cast<const float4*>(&at[ty + RY * i][4 * q]);
#pragma unroll
            for (int j = 0; j < RN; ++j) w[j] = *reinterpret_cast<const float4*>(&at[TM + tx + RX * j][4 * q]);
#pragma unroll
            for (int i = 0; i < RM; ++i)
#pragma unroll
                for (int j = 0; j < RN; ++j) {
                    acc[i][j] = fmaf(a[i].x, w[j].x, acc[i][j]);
                    acc[i][j] = fmaf(a[i].y, w[j].y, acc[i][j]);
                    acc[i][j] = fmaf(a[i].z, w[j].z, acc[i][j]);
                    acc[i][j] = fmaf(a[i].w, w[j].w, acc[i][j]);
                }
        }
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < RN; ++j) kahan_add(sum[i][j], lost[i][j], acc[i][j]);
    }
    if (segments == 1) {
#pragma unroll
        for (int i = 0; i < RM; ++i) {
            const int m = m0 + ty + RY * i;
            if (m >= p.M) continue;
#pragma unroll
            for (int j = 0; j < (SWIGLU ? RN / 2 : RN); ++j) {
                const int n = n0 + tx + RX * j;
                if (n < p.N) f32_store<SWIGLU>(p, m, n, sum[i][j], SWIGLU ? sum[i][j + RN / 2] : 0.f);
            }
        }
        return;
    }
    cp_async_wait<0>();
    __syncthreads();  // the last step's tile has been read
    float2* part = reinterpret_cast<float2*>(&tile[0][0][0]);  // [TM][TN]: (sum, lost)
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) part[(ty + RY * i) * TN + tx + RX * j] = make_float2(sum[i][j], lost[i][j]);
    cluster_barrier();
    for (int e = blockIdx.z * NT + tid; e < TM * COLS; e += segments * NT) {
        const int r = e / COLS, c = e % COLS, m = m0 + r, n = n0 + c;
        if (m >= p.M || n >= p.N) continue;
        float total[2] = {0.f, 0.f};
#pragma unroll
        for (int half = 0; half < (SWIGLU ? 2 : 1); ++half) {
            float2 v[F32_MAX_SEGMENTS];
#pragma unroll
            for (int s = 0; s < F32_MAX_SEGMENTS; ++s)
                if (s < segments) v[s] = load_of_rank(&part[r * TN + half * COLS + c], s);
            float left = v[0].y;
            total[half] = v[0].x;
#pragma unroll
            for (int s = 1; s < F32_MAX_SEGMENTS; ++s)
                if (s < segments) {
                    kahan_add(total[half], left, v[s].x);
                    left += v[s].y;
                }
        }
        f32_store<SWIGLU>(p, m, n, total[0], total[1]);
    }
    cluster_barrier();  // nobody leaves while its partial sums are read
}

template <int TM, int TN, int RM, int RN, bool SWIGLU>
static int launch_f32(const F32Args& p, cudaStream_t stream) {
    constexpr int COLS = SWIGLU ? TN / 2 : TN;
    cudaLaunchConfig_t cfg = {};
    int segments = (p.K + F32_SEGMENT - 1) / F32_SEGMENT;
    if (segments > F32_MAX_SEGMENTS) segments = F32_MAX_SEGMENTS;
    cfg.gridDim = dim3((p.N + COLS - 1) / COLS, (p.M + TM - 1) / TM, segments);
    cfg.blockDim = (TM / RM) * (TN / RN);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {1, 1, (unsigned)segments};
    cfg.attrs = attr;
    cfg.numAttrs = segments > 1 ? 1 : 0;
    const cudaError_t err = cudaLaunchKernelEx(&cfg, gemm_f32_kernel<TM, TN, RM, RN, SWIGLU>, p);
    return err != cudaSuccess ? (int)err : CW_LAUNCH_CHECK();
}

// Tiles of 8 RM x 64 outputs, RM x 4 a thread, with the RM from 4 to 8 that leaves the least work for rows that do not exist and
// for idle SMs (per output the smaller RM cost more: RM + 4 reads for 16 RM multiply-adds); 200 rows: 40 x 64, 374 us for
// [gate, up], 425 us with 64 x 64.  With fewer than two tiles per SM what counts is how many loads are in flight:
// 16 x 32, 2 x 4 a thread (200 x 2,048 by 1,536: 64 us against 72 with 64 x 64); up to 8 rows: 8 x 64, 2 x 4 ([gate, up] of 4 rows: 38 us
// against 53).  The sums do not depend on the choice.
template <bool SWIGLU>
static int run_f32(const F32Args& p, cudaStream_t stream) {
    if (p.M <= 8) return launch_f32<8, 64, 2, 4, SWIGLU>(p, stream);
    const long long columns = (p.N + (SWIGLU ? 31 : 63)) / (SWIGLU ? 32 : 64);
    const long long segments = (p.K + F32_SEGMENT - 1) / F32_SEGMENT;
    const long long across = columns * (segments < F32_MAX_SEGMENTS ? segments : F32_MAX_SEGMENTS);
    if (p.M <= 16 || across * ((p.M + 63) / 64) < 2 * 148) return launch_f32<16, 32, 2, 4, SWIGLU>(p, stream);
    int best = 8;
    double least = 0;
    for (int rm = 8; rm >= 4; --rm) {
        const long long tiles = across * ((p.M + 8 * rm - 1) / (8 * rm));
        const double cost = (double)((tiles + 147) / 148) * (rm + 1.0);
        if (rm == 8 || cost < least) best = rm, least = cost;
    }
    switch (best) {
        case 4: return launch_f32<32, 64, 4, 4, SWIGLU>(p, stream);
        case 5: return launch_f32<40, 64, 5, 4, SWIGLU>(p, stream);
        case 6: return launch_f32<48, 64, 6, 4, SWIGLU>(p, stream);
        case 7: return launch_f32<56, 64, 7, 4, SWIGLU>(p, stream);
        default: return launch_f32<64, 64, 8, 4, SWIGLU>(p, stream);
    }
}

// (with 16-row tiles the grid ends at 65,535 * 16 rows)
static bool whole_pieces(const void* p, int stride) { return (uintptr_t)p % 16 == 0 && stride % 4 == 0; }

extern "C" int cw_gemm_ref(const void* A, const void* W, const float* bias, void* C, int M, int N,
                           int K, int lda, int ldc, int epilogue, int dtype,
                           cudaStream_t stream) {
    if (M == 0 || N == 0) return CW_OK;
    if (M < 0 || N < 0 || K <= 0 || lda < K || ldc < N) return CW_ERR_BAD_SIZE;
    if (epilogue < 0 || (epilogue > 2 && epilogue != 4)) return CW_ERR_UNSUPPORTED;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return CW_ERR_BAD_SIZE;
    if (dtype == 0 && whole_pieces(A, lda) && whole_pieces(W, K) && M <= 65535 * 16)
        return run_f32<false>({(const float*)A, (const float*)W, nullptr, bias, (float*)C, M, N, K, lda, ldc, epilogue}, stream);
    if (dtype == 0)
        gemm_ref_kernel<float, false><<<grid, 256, 0, stream>>>(
            (const float*)A, (const float*)W, nullptr, bias, C, M, N, K, lda, ldc, epilogue);
    else if (dtype == 1)
        gemm_ref_kernel<bf16, false><<<grid, 256, 0, stream>>>(
            (const bf16*)A, (const bf16*)W, nullptr, bias, C, M, N, K, lda, ldc, epilogue);
    else
        return CW_ERR_BAD_DTYPE;
    return CW_LAUNCH_CHECK();
}

extern "C" int cw_gemm_ref_swiglu(const void* A, const void* Wgate, const void* Wup, void* C,
                                  int M, int N, int K, int dtype, cudaStream_t stream) {
    if (M == 0 || N == 0) return CW_OK;
    if (M < 0 || N < 0 || K <= 0) return CW_ERR_BAD_SIZE;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return CW_ERR_BAD_SIZE;
    if (dtype == 0 && whole_pieces(A, K) && whole_pieces(Wgate, K) && whole_pieces(Wup, K) && M <= 65535 * 16)
        return run_f32<true>({(const float*)A, (const float*)Wgate, (const float*)Wup, nullptr, (float*)C, M, N, K, K, N, 0}, stream);
    if (dtype == 0)
        gemm_ref_kernel<float, true><<<grid, 256, 0, stream>>>(
            (const float*)A, (const float*)Wgate, (const float*)Wup, nullptr, C, M, N, K, K, N, 0);
    else if (dtype == 1)
        gemm_ref_kernel<bf16, true><<<grid, 256, 0, stream>>>(
            (const bf16*)A, (const bf16*)Wgate, (const bf16*)Wup, nullptr, C, M, N, K, K, N, 0);
    else
        return CW_ERR_BAD_DTYPE;
    return CW_LAUNCH_CHECK();
}

CW_TRACE_TU(gemm_ref)
