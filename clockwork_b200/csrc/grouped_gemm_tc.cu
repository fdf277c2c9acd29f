// Products in groups (grouped_gemm.cu) on the 5th-generation tensor cores.
//
// As in gemm_tc.cu the weights ride the MMA's M dimension: a tile is 128 output features of one group by up to BN of its rows,
// D[feature, row] in tensor memory.  One CTA per SM walks the tiles of all groups; how many there are follows from the
// offsets, which only the device knows, so every CTA forms the groups' running tile counts at its start.  Weight tiles come by
// TMA through one map of all groups' matrices stacked.  Rows that lie next to one another come by TMA in boxes of 32 (rows of
// the next group among them, whose results nobody reads); rows that lie scattered (an index says where) by TMA gathers of four
// rows each, a lane of the producer warp per gather.  An SM gets a gathered row in about 20 cycles, which is enough for the few
// rows of single tokens and not for a prompt's (gate and up of the sizes below: 385 us): those are copied into the
// order of their groups first (cw_gather_rows), and only the narrow tiles gather.  A group's rows are cut in tiles of equal width, a multiple of 16, and tiles that share a weight tile are
// neighbours in the walk, so that it is read from HBM once.  Two accumulators in tensor memory: the epilogue of a tile (eight
// warps, straight from tensor memory to global memory: a warp's 32 features of a row are one line in float32, and in
// bfloat16 two lanes swap halves of two rows so that a lane stores two features) runs beside the next tile's MMAs.
//
// What bounds it: a prompt's routed layer has each expert's weights for a hundred or two of rows, which is what HBM and the
// tensor cores take about equally long for, and waits of one for the other (HBM at 53 % of its peak for gate and up, 60 % for down, the tensor
// pipe at 43 and 40 %); single tokens are bound by the weights alone, and BN = 32 leaves room for more
// weight tiles in flight.  The mma.sync kernel it replaced for these sizes stages both operands by cp.async, three steps of 32.
// Measured (B200, 2,048 tokens, 64 experts of 1,408 of which 6, width 2,048): gate and up 672 -> 169 us, down 366 -> 99 us; 8 tokens:
// 128 -> 67 us and 72 -> 34 us; per-head products of 2,048 tokens (16 x 128 to 512, gated 16 x 512 to 128): 36 -> 23 us and 61 -> 44 us.
//
// Every wait on an mbarrier is bounded, as in gemm_tc.cu.
#include "grouped_gemm.cuh"
#include "tc_common.cuh"

#define GT_BM 128
#define GT_BK 64
#define GT_EPI_WARPS 8
#define GT_THREADS (64 + 32 * GT_EPI_WARPS)
#define GT_MAX_GROUPS 1024
#define GT_SMALL_ROWS 32
#define GT_BOX 32  // rows of a box where they lie next to one another

template <int BN, bool TWO>
struct GtCfg {
    static constexpr int W_BYTES = GT_BM * GT_BK * 2 * (TWO ? 2 : 1);
    static constexpr int STAGE_BYTES = W_BYTES + BN * GT_BK * 2;
    static constexpr int STAGES = (200 * 1024) / STAGE_BYTES > 8 ? 8 : (200 * 1024) / STAGE_BYTES;
    static constexpr int ACC_COLS = BN * (TWO ? 2 : 1);
    static constexpr int TMEM_COLS = 2 * ACC_COLS;
    static_assert(TMEM_COLS >= 32 && TMEM_COLS <= 512 && (TMEM_COLS & (TMEM_COLS - 1)) == 0, "two accumulators in tensor memory");
    static int smem(int G) { return 1024 + STAGES * STAGE_BYTES + 256 + 2 * (G + 1) * 4; }
};

struct GtTile {
    int g, f0, row, width, rows;  // group, first feature, first row, MMA columns (a multiple of 16), rows that exist
};

// Tile `t` of the walk: groups in order; within a group the row tiles of a feature tile are neighbours.
__device__ __forceinline__ GtTile gt_tile(const GroupedArgs& p, const int* cum, const int* first, int ftiles, int t) {
    const int u = t / ftiles;
    int lo = 0, hi = p.G;  // the last group whose first row tile is at or before u (groups without rows have no tiles)
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (cum[mid] <= u) lo = mid;
        else hi = mid;
    }
    GtTile x;
    x.g = lo;
    const int row_tiles = cum[lo + 1] - cum[lo], local = t - cum[lo] * ftiles;
    const int n = p.offsets != nullptr ? first[lo + 1] - first[lo] : p.M;
    x.f0 = local / row_tiles * GT_BM;
    x.width = ((n + row_tiles - 1) / row_tiles + 15) & ~15;
    const int at = local % row_tiles * x.width;
    x.row = first[lo] + at;
    x.rows = min(x.width, n - at);  // (never none: a tile fewer would not hold the rows at the full width)
    return x;
}

__device__ __forceinline__ void gather_rows(uint32_t dst, const CUtensorMap* map, int x, const int (&y)[4], uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y[0]), "r"(y[1]), "r"(y[2]), "r"(y[3])
        : "memory");
}

template <int BN, int EPI>
__global__ void __launch_bounds__(GT_THREADS, 1)
grouped_gemm_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_w2,
                       const __grid_constant__ CUtensorMap map_x, const GroupedArgs p) {
    constexpr bool TWO = EPI == GG_EPI_SILU_MUL;
    using C = GtCfg<BN, TWO>;
    extern __shared__ uint8_t gt_smem[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)gt_smem + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + C::STAGES * C::STAGE_BYTES);  // full[S], empty[S], acc_full[2], acc_empty[2]
    uint32_t* tmem_slot = (uint32_t*)(bars + 2 * C::STAGES + 4);
    volatile int* give_up = (volatile int*)(tmem_slot + 1);
    int* cum = (int*)(bars + 32);    // [G + 1] row tiles of the groups before
    int* first = cum + p.G + 1;      // [G + 1] where a group's rows begin
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + C::STAGES);
    const uint32_t accf0 = smem_u32(bars + 2 * C::STAGES), acce0 = accf0 + 16;

    if (tid == 64) {
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(accf0 + 8 * b, 1);
            mbar_init(acce0 + 8 * b, GT_EPI_WARPS);
        }
        *give_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
    pdl_wait();
    if (warp == 0) {
        int run = 0;
        for (int g0 = 0; g0 < p.G; g0 += 32) {
            const int g = g0 + lane;
            int tiles = 0;
            if (g < p.G) {
                const int begin = p.offsets != nullptr ? p.offsets[g] : 0, end = p.offsets != nullptr ? p.offsets[g + 1] : p.M;
                tiles = (end - begin + BN - 1) / BN;
                first[g] = begin;
                if (g == p.G - 1) first[p.G] = end;
            }
            int upto = tiles;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            if (g < p.G) cum[g] = run + upto - tiles;
            run += __shfl_sync(0xffffffffu, upto, 31);
        }
        if (lane == 0) cum[p.G] = run;
    }
    tc_fence_before();
    __syncthreads();
    pdl_release();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int ftiles = (p.Nout + GT_BM - 1) / GT_BM, tiles = cum[p.G] * ftiles, num_kb = (p.K + GT_BK - 1) / GT_BK;

    if (warp == 0) {
        // ---- producer warp: lane 0 the weight tiles, every lane the gathers of its rows ---------------------------
        constexpr bool GATHERS = BN == GT_SMALL_ROWS;
        int next_y[4];
        auto find_rows = [&](const GtTile& x) {  // (rows past the tile's end: its last one again)
            if (!GATHERS) return;
#pragma unroll
            for (int i = 0; i < 4; ++i) next_y[i] = p.a_index != nullptr ? p.a_index[x.row + min(lane * 4 + i, x.rows - 1)] / p.a_div : 0;
        };
        int i = 0;
        bool ok = true;
        GtTile x = {};
        if ((int)blockIdx.x < tiles) {
            x = gt_tile(p, cum, first, ftiles, blockIdx.x);
            find_rows(x);
        }
        for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
            int y[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) y[k] = GATHERS ? next_y[k] : 0;
            const GtTile now = x;
            if (t + (int)gridDim.x < tiles) {  // the next tile's rows are looked up while this one's copies are issued
                x = gt_tile(p, cum, first, ftiles, t + gridDim.x);
                find_rows(x);
            }
            const int x0 = now.g * p.a_group_off, w0 = now.g * p.Nout + now.f0;
            const bool gather = GATHERS && p.a_index != nullptr;
            const int fetched = gather ? now.width : (now.width + GT_BOX - 1) / GT_BOX * GT_BOX;  // (BN is whole boxes)
            const uint32_t tx = C::W_BYTES + fetched * GT_BK * 2;
            for (int kb = 0; kb < num_kb; ++kb, ++i) {
                const int s = i % C::STAGES;
                ok = mbar_wait(empty0 + 8 * s, ((i / C::STAGES) & 1) ^ 1, give_up);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                const uint32_t w_dst = smem_u32(smem + s * C::STAGE_BYTES), bar = full0 + 8 * s;
                if (lane == 0) {
                    mbar_expect_tx(bar, tx);
                    tma_load_2d(w_dst, &map_w, kb * GT_BK, w0, bar);
                    if (TWO) tma_load_2d(w_dst + C::W_BYTES / 2, &map_w2, kb * GT_BK, w0, bar);
                }
                __syncwarp();
                if (!gather) {
                    if (lane * GT_BOX < fetched)
                        tma_load_2d(w_dst + C::W_BYTES + lane * GT_BOX * GT_BK * 2, &map_x, x0 + kb * GT_BK, now.row + lane * GT_BOX, bar);
                    continue;
                }
                if (lane * 4 < now.width) gather_rows(w_dst + C::W_BYTES + lane * 4 * GT_BK * 2, &map_x, x0 + kb * GT_BK, y, bar);
            }
        }
        if (*give_up && lane == 0) {
            for (int k = max(0, i - C::STAGES); k < i; ++k) {  // the copies in flight, bounded
                const long long t0 = clock64();
                while (!mbar_try_wait(full0 + 8 * (k % C::STAGES), (k / C::STAGES) & 1) && clock64() - t0 < WAIT_CYCLES) {
                }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            // ---- MMA issuer: the walk's tile `it` accumulates into buffer it & 1 ---------------------------------
            const uint64_t desc0 = smem_desc_sw128(smem_u32(smem));
            uint64_t adesc = desc0;  // (16-byte units: a stage further is STAGE_BYTES / 16)
            int it = 0, s = 0;
            uint32_t parity = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++it) {
                const uint32_t idesc = instr_desc(GT_BM, gt_tile(p, cum, first, ftiles, t).width);
                const int buf = it & 1;
                ok = mbar_wait(acce0 + 8 * buf, ((it >> 1) & 1) ^ 1, give_up);
                if (!ok) break;
                tc_fence_after();
                const uint32_t acc = tmem_base + buf * C::ACC_COLS;
                for (int kb = 0; kb < num_kb; ++kb) {
                    ok = mbar_wait(full0 + 8 * s, parity, give_up);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t a2desc = adesc + C::W_BYTES / 2 / 16, bdesc = adesc + C::W_BYTES / 16;
#pragma unroll
                    for (int k = 0; k < GT_BK / 16; ++k) {
                        const uint32_t accumulate = (kb > 0 || k > 0) ? 1u : 0u;
                        umma_bf16(acc, adesc + 2 * k, bdesc + 2 * k, idesc, accumulate);
                        if (TWO) umma_bf16(acc + BN, a2desc + 2 * k, bdesc + 2 * k, idesc, accumulate);
                    }
                    umma_commit(empty0 + 8 * s);
                    adesc += C::STAGE_BYTES / 16;
                    if (++s == C::STAGES) {
                        s = 0;
                        parity ^= 1;
                        adesc = desc0;
                    }
                }
                if (ok) umma_commit(accf0 + 8 * buf);
            }
        }
    } else {
        // ---- epilogue: warp w reads tensor-memory lanes 32 (w % 4) .. +31, every other 16 columns --------------------
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        int it = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++it) {
            const GtTile x = gt_tile(p, cum, first, ftiles, t);
            const int buf = it & 1;
            ok = mbar_wait(accf0 + 8 * buf, (it >> 1) & 1, give_up);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + buf * C::ACC_COLS + ((uint32_t)(quarter * 32) << 16);
            const int f = x.f0 + quarter * 32 + lane;
            const size_t column = (size_t)x.g * p.c_group_off + f;
            for (int c = half * 16; c < x.rows; c += 32) {
                float v[16], u[16];
                tmem_ld16(taddr + c, v);
                if (TWO) tmem_ld16(taddr + BN + c, u);
                // lane i holds where row c + i goes (and its gate)
                const int r = c + (lane & 15);
                int my_dst = -1;
                if (r < x.rows) my_dst = p.c_index != nullptr ? p.c_index[x.row + r] : x.row + r;
                float my_open = 1.f;
                if (EPI == GG_EPI_GROUP_GATE && my_dst >= 0)
                    my_open = 1.f / (1.f + expf(-((const float*)p.gate)[(size_t)my_dst * p.ldg + x.g]));
                if (EPI == GG_EPI_STORE_F32) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const int dst = __shfl_sync(0xffffffffu, my_dst, j);
                        if (dst >= 0 && f < p.Nout) ((float*)p.C)[(size_t)dst * p.ldc + column] = v[j];
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (TWO) v[j] = gg_glu(v[j], u[j], p.glu_limit);
                        if (EPI == GG_EPI_RELU2) v[j] = fmaxf(v[j], 0.f) * fmaxf(v[j], 0.f);
                    }
#pragma unroll
                    for (int j = 0; j < 16; j += 2) {  // even lanes: features f, f + 1 of row j; odd lanes: f - 1, f of row j + 1
                        const bool odd = lane & 1;
                        const float got = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
                        float a = odd ? got : v[j], b = odd ? v[j + 1] : got;
                        const int dst = __shfl_sync(0xffffffffu, my_dst, j + (lane & 1));
                        if (EPI == GG_EPI_GROUP_GATE) {
                            const float open = __shfl_sync(0xffffffffu, my_open, j + (lane & 1));
                            a *= open;
                            b *= open;
                        }
                        if (dst >= 0 && f < p.Nout) {  // (Nout is even: both features exist or none)
                            const size_t pair = column & ~(size_t)1;
                            if (EPI == GG_EPI_SIGMOID_GATE) {
                                const __nv_bfloat162 gate = *reinterpret_cast<const __nv_bfloat162*>((const bf16*)p.gate + (size_t)dst * p.ldg + pair);
                                a = a / (1.f + expf(-__low2float(gate)));
                                b = b / (1.f + expf(-__high2float(gate)));
                            }
                            *reinterpret_cast<__nv_bfloat162*>((bf16*)p.C + (size_t)dst * p.ldc + pair) = __floats2bfloat162_rn(a, b);
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acce0 + 8 * buf) : "memory");
        }
    }
    __syncwarp();
    if (*give_up && tid == 0) cw_report(p.status, CW_ST_WAIT_TIMEOUT, blockIdx.x, -2);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, C::TMEM_COLS);
}

// ---- rows into the order of their groups ---------------------------------------------------------------------------
// out[r] = a[index[r] / div] for the offsets[G] rows that belong to a group; a block per row, 16 bytes a thread.
__global__ void __launch_bounds__(256) gather_rows_kernel(const uint4* __restrict__ a, uint4* __restrict__ out, const int* __restrict__ index,
                                                          const int* __restrict__ rows, int div, int pieces) {
    pdl_enter();
    if ((int)blockIdx.x >= *rows) return;
    const uint4* from = a + (size_t)(index[blockIdx.x] / div) * pieces;
    for (int c = threadIdx.x; c < pieces; c += 256) out[(size_t)blockIdx.x * pieces + c] = from[c];
}

// a [.., row_bytes] rows, out [M, row_bytes]; row_bytes and both bases whole 16-byte pieces.  `rows` (on the device): how many of
// the M places of `index` hold one.
extern "C" int cw_gather_rows(const void* a, void* out, const int* index, const int* rows, int M, int div, long long row_bytes,
                              cudaStream_t stream) {
    if (M == 0) return CW_OK;
    if (M < 0 || div <= 0 || row_bytes <= 0) return CW_ERR_BAD_SIZE;
    if (row_bytes % 16 || row_bytes / 16 > 0x7fffffffLL || ((uintptr_t)a | (uintptr_t)out) % 16) return CW_ERR_UNSUPPORTED;
    return cw_launch(gather_rows_kernel, dim3(M), dim3(256), 0, stream, 1, (const uint4*)a, (uint4*)out, index, rows, div, (int)(row_bytes / 16));
}

// ---- host side ---------------------------------------------------------------------------------------------------
// A [rows, columns] bfloat16 matrix with rows of `ld` elements, read in boxes of `box_rows` x 64.
static int gt_map(CUtensorMap* map, const void* ptr, long long rows, long long columns, long long ld, int box_rows) {
    const cuuint64_t dims[2] = {(cuuint64_t)columns, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {GT_BK, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elem,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : -1;
}

// Rows per group, as far as the host knows (a router spreads them): few of them take the narrow tiles.
static bool gt_few(const GroupedArgs& p) { return (p.offsets != nullptr ? (p.M + p.G - 1) / p.G : p.M) <= GT_SMALL_ROWS; }

// TMA wants 16-byte rows and bases and all groups' matrices stacked; a group's columns of A must end where a step of 64 does (a
// step past them would read the next group's); the epilogue stores two features at a time.
bool grouped_tc_takes(const GroupedArgs& p, int epilogue) {
    if (p.G > GT_MAX_GROUPS || p.K % 8 || p.lda % 8 || p.a_group_off % 8 || ((uintptr_t)p.A | (uintptr_t)p.B | (uintptr_t)p.B2) % 16) return false;
    if (p.b_stride != (long long)p.Nout * p.K || (long long)p.G * p.Nout > 0x7fffffffLL) return false;
    if (p.a_group_off != 0 && p.K % GT_BK) return false;
    if (p.a_index != nullptr && !gt_few(p)) return false;
    if (p.Nout % 2 || p.ldc % 2 || p.c_group_off % 2 || (uintptr_t)p.C % 8) return false;
    if (epilogue == GG_EPI_SIGMOID_GATE && (p.ldg % 2 || (uintptr_t)p.gate % 4)) return false;
    return true;
}

template <int BN, int EPI>
static int gt_launch(const GroupedArgs& p, const CUtensorMap& w, const CUtensorMap& w2, const CUtensorMap& x, int grid, cudaStream_t stream) {
    using C = GtCfg<BN, EPI == GG_EPI_SILU_MUL>;
    const int smem = C::smem(p.G);
    const cudaError_t e = cudaFuncSetAttribute(grouped_gemm_tc_kernel<BN, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::smem(GT_MAX_GROUPS));
    if (e != cudaSuccess) return (int)e;
    return cw_launch(grouped_gemm_tc_kernel<BN, EPI>, dim3(grid), dim3(GT_THREADS), (size_t)smem, stream, 1, w, w2, x, p);
}

int grouped_tc_run(const GroupedArgs& p, int epilogue, cudaStream_t stream) {
    if (load_encode() != 0) return CW_ERR_UNSUPPORTED;
    int device = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return (int)e;
    const long long rows = p.a_index != nullptr ? (p.M + p.a_div - 1) / p.a_div : p.M;
    CUtensorMap w, w2, x;
    if (gt_map(&w, p.B, (long long)p.G * p.Nout, p.K, p.K, GT_BM) != 0 ||
        gt_map(&w2, p.B2 != nullptr ? p.B2 : p.B, (long long)p.G * p.Nout, p.K, p.K, GT_BM) != 0 ||
        gt_map(&x, p.A, rows, p.a_group_off != 0 ? (long long)(p.G - 1) * p.a_group_off + p.K : p.K, p.lda,
               p.a_index != nullptr ? 1 : GT_BOX) != 0)
        return CW_ERR_UNSUPPORTED;
    const bool few = gt_few(p);
    const int bn = few ? GT_SMALL_ROWS : epilogue == GG_EPI_SILU_MUL ? 128 : 256;
    const long long ftiles = (p.Nout + GT_BM - 1) / GT_BM;
    const long long row_tiles = p.offsets != nullptr ? (long long)(p.M + bn - 1) / bn + (p.M < p.G ? p.M : p.G) : (long long)p.G * ((p.M + bn - 1) / bn);
    if (row_tiles * ftiles > 0x3fffffffLL) return CW_ERR_UNSUPPORTED;
    const int grid = (int)(row_tiles * ftiles < sms ? row_tiles * ftiles : sms);
#define GT_GO(E, WIDE) return few ? gt_launch<GT_SMALL_ROWS, E>(p, w, w2, x, grid, stream) : gt_launch<WIDE, E>(p, w, w2, x, grid, stream)
    switch (epilogue) {
        case GG_EPI_STORE: GT_GO(GG_EPI_STORE, 256);
        case GG_EPI_STORE_F32: GT_GO(GG_EPI_STORE_F32, 256);
        case GG_EPI_SILU_MUL: GT_GO(GG_EPI_SILU_MUL, 128);
        case GG_EPI_SIGMOID_GATE: GT_GO(GG_EPI_SIGMOID_GATE, 256);
        case GG_EPI_RELU2: GT_GO(GG_EPI_RELU2, 256);
        case GG_EPI_GROUP_GATE: GT_GO(GG_EPI_GROUP_GATE, 256);
    }
#undef GT_GO
    return CW_ERR_UNSUPPORTED;
}

CW_TRACE_TU(grouped_gemm_tc)
