// Greedy and stochastic sampling over float32 logits, a cluster of thread blocks per row.
//
// Reference: clockwork/engine/model_runner.py:134-164.  Greedy is the first maximal index
// (:136-137).  Otherwise logits are divided by the temperature (:149); top-k keeps logits not
// below the k-th largest (:150-152); top-p sorts descending, accumulates softmax mass and drops
// a token when the mass *before* it already exceeds top_p, so the token that crosses the
// threshold stays (:153-163); the token is then drawn from the softmax of what is left.
// The reference draws with torch.multinomial from a per-request generator; here the caller
// supplies one uniform number u in [0,1) per row and the token is the first index whose
// cumulative probability (in index order) exceeds u.  Equal logits are kept or dropped together: under
// top-p a token stays iff the mass of the logits strictly above it does not exceed top_p (the reference's
// sort may cut between equal logits, in an order it does not define; every token it could keep stays here).
//
// Nothing is sorted: the k-th largest value and the top-p cut-off are found by searches over an order-preserving
// integer image of the logits: bit by bit in sample_kernel (32 counting passes each, a block per row, kept to compare
// against), by histograms in sample_rows_kernel.
#include "common.cuh"

#define ST 1024

__device__ __forceinline__ unsigned ordered_key(float f) {
    unsigned b = __float_as_uint(f);
    b = (b == 0x80000000u) ? 0u : b;  // -0.0 and +0.0 compare equal as floats: one image for both
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// The same with what is no number below everything else, whatever its sign: it is not the largest, and has no mass.
__device__ __forceinline__ unsigned logit_key(float f) { return f == f ? ordered_key(f) : 0u; }

// A sampled token leaves through here.  With a request-state table given (request_state.cu) the token
// also becomes the request's `last token`, and its position and draw counter advance by one: the next
// step can then be launched before the host has read this one's tokens.
__device__ __forceinline__ void emit_token(int row, int token, int* __restrict__ out, const int* __restrict__ row_slot,
                                           int* __restrict__ state, int num_slots) {
    out[row] = token;
    if (state != nullptr) {
        const int slot = row_slot[row];
        if (slot >= 0 && slot < num_slots) {
            state[CW_RS_LAST_TOKEN * num_slots + slot] = token;
            state[CW_RS_POSITION * num_slots + slot] += 1;
            state[CW_RS_DRAWS * num_slots + slot] += 1;
        }
    }
}

__device__ __forceinline__ float block_sum_1024(float v, float* scratch) { return block_sum(v, scratch); }

__global__ void __launch_bounds__(ST)
sample_kernel(const float* __restrict__ logits, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ top_p,
              const float* __restrict__ uniform, int* __restrict__ out, int V, size_t row_stride,
              const int* __restrict__ row_slot, int* __restrict__ state, int num_slots) {
    __shared__ float scratch[33];
    __shared__ float warp_tot[32];
    __shared__ int first_thread, last_thread;
    pdl_launch_dependents();
    pdl_wait();
    const int r = blockIdx.x, tid = threadIdx.x;
    const float* row = logits + (size_t)r * row_stride;
    const float temp = temperature[r];
    if (!(temp > 0.f)) {  // greedy row inside a mixed batch
        float best = -INFINITY;
        int idx = 0x7fffffff;
        for (int i = tid; i < V; i += ST) {
            const float v = row[i];
            if (v > best || (v == best && i < idx)) { best = v; idx = i; }
        }
        const float gmax = block_max(best, scratch);
        int cand = (best == gmax) ? idx : 0x7fffffff;
        if (tid == 0) first_thread = 0x7fffffff;
        __syncthreads();
        atomicMin(&first_thread, cand);
        __syncthreads();
        if (tid == 0) emit_token(r, first_thread == 0x7fffffff ? 0 : first_thread, out, row_slot, state, num_slots);
        return;
    }
    // pass 1: maximum of the scaled logits
    float mx = -INFINITY;
    for (int i = tid; i < V; i += ST) mx = fmaxf(mx, row[i] / temp);
    mx = block_max(mx, scratch);

    unsigned keep_key = 0u;  // a token is kept iff ordered_key(l) >= keep_key
    const int k = top_k[r];
    if (k > 0 && k < V) {
        unsigned thr = 0u;
        for (int bit = 31; bit >= 0; --bit) {
            const unsigned cand = thr | (1u << bit);
            float cnt = 0.f;
            for (int i = tid; i < V; i += ST) cnt += (ordered_key(row[i] / temp) >= cand) ? 1.f : 0.f;
            cnt = block_sum(cnt, scratch);
            if (cnt >= (float)k) thr = cand;
        }
        keep_key = thr;
    }
    const float p_lim = top_p[r];
    if (p_lim < 1.0f) {
        float zk = 0.f;
        for (int i = tid; i < V; i += ST) {
            const float l = row[i] / temp;
            if (ordered_key(l) >= keep_key) zk += expf(l - mx);
        }
        zk = block_sum(zk, scratch);
        // largest K0 whose strictly-greater mass still exceeds top_p; kept keys are > K0
        unsigned k0 = 0u;
        for (int bit = 31; bit >= 0; --bit) {
            const unsigned cand = k0 | (1u << bit);
            float g = 0.f;
            for (int i = tid; i < V; i += ST) {
                const float l = row[i] / temp;
                const unsigned key = ordered_key(l);
                if (key >= keep_key && key > cand) g += expf(l - mx);
            }
            g = block_sum(g, scratch);
            if (g > p_lim * zk) k0 = cand;
        }
        if (k0 != 0xffffffffu && k0 + 1u > keep_key) keep_key = k0 + 1u;
    }
    // final pass: inverse CDF in index order; thread t owns a contiguous range
    const int per = (V + ST - 1) / ST;
    const int lo = min(V, tid * per), hi = min(V, lo + per);
    float mine = 0.f;
    for (int i = lo; i < hi; ++i) {
        const float l = row[i] / temp;
        if (ordered_key(l) >= keep_key) mine += expf(l - mx);
    }
    // block-wide exclusive scan of `mine` in thread order
    const int lane = tid & 31, warp = tid >> 5;
    float incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
    }
    if (lane == 31) warp_tot[warp] = incl;
    if (tid == 0) { first_thread = 0x7fffffff; last_thread = -1; }
    __syncthreads();
    float warp_off = 0.f, total = 0.f;
    for (int w = 0; w < 32; ++w) {
        if (w < warp) warp_off += warp_tot[w];
        total += warp_tot[w];
    }
    const float excl = warp_off + incl - mine;
    const float target = uniform[r] * total;
    if (mine > 0.f) {
        atomicMax(&last_thread, tid);
        if (excl + mine > target) atomicMin(&first_thread, tid);
    }
    __syncthreads();
    // when rounding leaves the target beyond the last kept token, the last owner takes it
    const int owner = first_thread != 0x7fffffff ? first_thread : last_thread;
    if (owner < 0) {
        if (tid == 0) emit_token(r, 0, out, row_slot, state, num_slots);
        return;
    }
    if (tid == owner) {
        float run = excl;
        int pick = -1, last_kept = lo;
        for (int i = lo; i < hi; ++i) {
            const float l = row[i] / temp;
            if (ordered_key(l) >= keep_key) {
                run += expf(l - mx);
                last_kept = i;
                if (run > target) { pick = i; break; }
            }
        }
        emit_token(r, pick >= 0 ? pick : last_kept, out, row_slot, state, num_slots);
    }
}

extern "C" int cw_sample_state(const float* logits, const float* temperature, const int* top_k, const float* top_p,
                               const float* uniform, int* out, int R, int V, long long row_stride, const int* row_slot,
                               int* state, int num_slots, cudaStream_t stream) {
    if (R == 0) return CW_OK;
    if (R < 0 || V <= 0 || row_stride < V || (state != nullptr && (row_slot == nullptr || num_slots <= 0))) return CW_ERR_BAD_SIZE;
    return cw_launch(sample_kernel, dim3(R), dim3(ST), 0, stream, 1, logits, temperature, top_k, top_p, uniform, out, V,
                     (size_t)row_stride, row_slot, state, num_slots);
}

extern "C" int cw_sample(const float* logits, const float* temperature, const int* top_k,
                         const float* top_p, const float* uniform, int* out, int R, int V,
                         long long row_stride, cudaStream_t stream) {
    return cw_sample_state(logits, temperature, top_k, top_p, uniform, out, R, V, row_stride, nullptr, nullptr, 0, stream);
}

// ---------------------------------------------------------------------------------------------
// The same rule with a cluster of SR_CTAS thread blocks per row.
//
// sample_kernel above walks a row 65 times with one block: a vocabulary of 150,000 costs it a
// millisecond and more.  Here every block of a cluster reads its part of the row once, keeps the
// order-preserving keys in shared memory, and both searches run there: histograms over bins that fall
// in the order of the keys, added up over the cluster through distributed shared memory, each search
// going on inside the bin that it found until one key is left:
//   top-k: counts per bin; the bin in which the count from the top reaches k is refined;
//   top-p: mass per bin (of the keys top-k kept); the highest bin at which the mass from the top
//          exceeds top_p * Z is refined; the key found is the lowest one kept.
// The first bins are 1/73 wide in units of the logits (scaled by the temperature) and count down from
// the row's maximum: leading bits of a key would put most of a vocabulary into a handful of bins, whose
// atomics then wait for one another.  The last of them takes all that is too far below to have any mass;
// what falls there is summed in registers.  Later levels cut the range of the bin's keys in 2,048.
// What can still be kept is moved together, in index order.  Under a top-k of at most SR_THREADS, first of all within each
// block: the k-th largest of its threads' maxima bounds the row's k-th largest from below.  Then what lies in the first bin
// found or above it: in one block's memory if it fits there (the other blocks are then done, and no barrier of the cluster
// is left: top-k of 50 keeps some sixty logits), else within each block.
// Masses are integers, exp(l - max) * 2^40 truncated: sums of integers do not depend on the order in
// which blocks and threads add them up, so a row's token is the same on every run whatever the
// scheduling (floating-point atomics would not give that), and the final walk along the row in index
// order compares exact cumulative sums with u * total.
// What bounds it: the instructions of the first passes (37 keys a thread; issue slots 48 % busy over the launch), then the latency of
// the barriers, the first of its stalls.
// Measured (B200, 64 rows of 151,936 with top-k 50 and top-p 0.9): 62 us; a chain of eight kernels that
// re-read the row from L2 and kept its histograms in global memory took 224; one row: 21 and 68.
// Rows of more than SR_CTAS * SR_STAGED logits are read again from global memory on each pass.
// ---------------------------------------------------------------------------------------------
#define SR_CTAS 8
#define SR_THREADS 512
#define SR_WARPS (SR_THREADS / 32)
#define SR_BINS 2048
#define SR_SLICE (SR_BINS / SR_CTAS)  // the bins that a block adds up for the cluster
#define SR_RANGE 28.0f                // exp(-28) * 2^40 < 1: no mass beyond
#define SR_STAGED 49152               // keys that a block holds in shared memory
#define SR_LOADS 16                   // logits of a thread in flight
#define SR_LIST 1024                  // and of those that are left, its own and the cluster's
#define SP_MASS_ONE 1099511627776.0f  // 2^40

typedef unsigned long long u64;

__device__ __forceinline__ float key_to_float(unsigned key) {
    const unsigned b = (key & 0x80000000u) ? (key & 0x7fffffffu) : ~key;
    return __uint_as_float(b);
}
// (none where the exponential is no number, which the conversion would turn into 2^63)
__device__ __forceinline__ u64 mass_of(float l, float mx) { return (u64)(fmaxf(expf(l - mx), 0.f) * SP_MASS_ONE); }

struct SampleParams {
    const float* logits; size_t row_stride; int V;
    const float* temperature; const int* top_k; const float* top_p; const float* uniform;
    int* out; const int* row_slot; int* state; int num_slots;
    int chunk, staged;  // logits of a block's part; whether its keys stay in shared memory
};

__device__ __forceinline__ void sr_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The word of block `rank` that lies where `mine` does here.
__device__ __forceinline__ unsigned sr_remote(const void* mine, unsigned rank) {
    unsigned at;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((unsigned)__cvta_generic_to_shared(mine)), "r"(rank));
    return at;
}
__device__ __forceinline__ u64 sr_read(const u64* mine, unsigned rank) {
    u64 v;
    asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(sr_remote(mine, rank)) : "memory");
    return v;
}
__device__ __forceinline__ unsigned sr_read(const unsigned* mine, unsigned rank) {
    unsigned v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(sr_remote(mine, rank)) : "memory");
    return v;
}

struct SampleShared {
    unsigned low[SR_BINS], high[SR_BINS];  // a bin's sum here, in two words (shared memory adds 32 bits at a time)
    u64 slice[SR_SLICE];                   // the cluster's sums of this block's slice of the bins
    u64 box[6];                            // for the other blocks: best, slice's sum, lowest and highest key, kept mass, keys left
    u64 gathered[SR_CTAS];
    u64 warp[SR_WARPS];
    u64 above;
    int bin, first;
    unsigned list[2][SR_LIST], index[2][SR_LIST];  // the keys that are left and where they lie in the row: here, in the cluster
};

enum { SR_SUM, SR_MAX, SR_MIN };
template <int OP>
__device__ __forceinline__ u64 sr_combine(u64 a, u64 b) {
    return OP == SR_SUM ? a + b : (OP == SR_MAX ? (a > b ? a : b) : (a < b ? a : b));
}
template <int OP>
__device__ u64 sr_block(u64 v, SampleShared& s) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = sr_combine<OP>(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s.warp[threadIdx.x >> 5] = v;
    __syncthreads();
    u64 all = s.warp[0];
#pragma unroll
    for (int w = 1; w < SR_WARPS; ++w) all = sr_combine<OP>(all, s.warp[w]);
    return all;
}
// Every block's word `b` of its box, in s.gathered; the blocks' boxes are written (a cluster barrier lies between).
__device__ __forceinline__ void sr_gather(SampleShared& s, int b) {
    __syncthreads();
    if (threadIdx.x < SR_CTAS) s.gathered[threadIdx.x] = sr_read(&s.box[b], threadIdx.x);
    __syncthreads();
}
// A value per thread combined over the cluster, through word `b` of the boxes (alone: over this block).
template <int OP>
__device__ u64 sr_cluster(u64 v, SampleShared& s, int b, bool alone) {
    v = sr_block<OP>(v, s);
    if (alone) return v;
    if (threadIdx.x == 0) s.box[b] = v;
    sr_cluster_sync();
    sr_gather(s, b);
    u64 all = s.gathered[0];
#pragma unroll
    for (int c = 1; c < SR_CTAS; ++c) all = sr_combine<OP>(all, s.gathered[c]);
    return all;
}
__device__ __forceinline__ void sr_add(SampleShared& s, int bin, u64 v, bool mass) {
    if (!mass) {  // (a count: no carry to look for)
        atomicAdd(&s.low[bin], (unsigned)v);
        return;
    }
    const unsigned lo = (unsigned)v, old = atomicAdd(&s.low[bin], lo);
    const unsigned hi = (unsigned)(v >> 32) + (old + lo < old ? 1u : 0u);
    if (hi != 0) atomicAdd(&s.high[bin], hi);
}

// The sums of the warps before this thread's and of its own up to it; *all: of the block.
__device__ __forceinline__ u64 sr_scan(u64 v, SampleShared& s, u64* all) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 n = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += n;
    }
    __syncthreads();
    if (lane == 31) s.warp[warp] = v;
    __syncthreads();
    u64 sum = 0;
    for (int w = 0; w < SR_WARPS; ++w) {
        if (w < warp) v += s.warp[w];
        sum += s.warp[w];
    }
    *all = sum;
    return v;
}

// One level of a search: the blocks' histograms are complete; the first bin at which the running sum from bin 0
// satisfies the rule: counts, sum >= want (the want-th largest key lies in it); masses, sum > want.  `fraction` >= 0:
// want is that fraction of the whole sum.  What lies before the bin is taken off `want`; the histogram is cleared.
// Every thread of the cluster gets the same answer.  `alone`: the histogram is this block's only.
__device__ int sr_level(SampleShared& s, unsigned rank, bool alone, double& want, double fraction, bool strictly) {
    constexpr int PER = SR_BINS / SR_THREADS;
    const int tid = threadIdx.x;
    auto enough = [&](u64 sum) { return strictly ? (double)sum > want : (double)sum >= want; };
    u64 v[PER] = {}, before = 0;  // this thread's bins of those among which the answer is
    int first_bin = tid * PER, bins = PER;
    if (alone) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            v[i] = (u64)s.low[tid * PER + i] + ((u64)s.high[tid * PER + i] << 32);
            s.low[tid * PER + i] = s.high[tid * PER + i] = 0u;
        }
    } else {
        sr_cluster_sync();
        u64 mine = 0;
        if (tid < SR_SLICE) {
#pragma unroll
            for (int c = 0; c < SR_CTAS; ++c) {
                const int b = (int)rank * SR_SLICE + tid;
                mine += (u64)sr_read(&s.low[b], c) + ((u64)sr_read(&s.high[b], c) << 32);
            }
            s.slice[tid] = mine;
        }
        const u64 sum = sr_block<SR_SUM>(mine, s);
        if (tid == 0) s.box[1] = sum;
        sr_cluster_sync();
        for (int i = tid; i < SR_BINS; i += SR_THREADS) s.low[i] = s.high[i] = 0u;
        sr_gather(s, 1);
        if (fraction >= 0.) {
            u64 all = 0;
            for (int c = 0; c < SR_CTAS; ++c) all += s.gathered[c];
            want = fraction * (double)all;
        }
        int slice = 0;
        for (; slice < SR_CTAS - 1 && !enough(before + s.gathered[slice]); ++slice) before += s.gathered[slice];
        if (tid < SR_SLICE) v[0] = sr_read(&s.slice[tid], slice);
        first_bin = slice * SR_SLICE + tid;
        bins = 1;
    }
    u64 mine = 0, all;
    for (int i = 0; i < PER; ++i) mine += v[i];
    if (tid == 0) s.first = SR_THREADS;
    const u64 incl = before + sr_scan(mine, s, &all);
    if (alone && fraction >= 0.) want = fraction * (double)all;
    const int last = alone ? SR_THREADS - 1 : SR_SLICE - 1;
    if (tid <= last && enough(incl)) atomicMin(&s.first, tid);
    __syncthreads();
    if (tid == min(s.first, last)) {  // (no bin qualifies, by rounding: the lowest, with everything before it)
        u64 run = incl - mine;
        int i = 0;
        for (; i < bins - 1 && !enough(run + v[i]); ++i) run += v[i];
        s.bin = first_bin + i;
        s.above = run;
    }
    __syncthreads();
    want -= (double)s.above;
    return s.bin;
}

__global__ void __launch_bounds__(SR_THREADS, 2)
sample_rows_kernel(const SampleParams p) {
    extern __shared__ unsigned sr_keys[];
    __shared__ SampleShared s;
    pdl_launch_dependents();
    pdl_wait();
    const int r = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const unsigned rank = blockIdx.z;
    const float temp = p.temperature[r];
    const bool sampled = temp > 0.f;
    const int from = min(p.V, (int)rank * p.chunk), n = min(p.V, from + p.chunk) - from;
    const float* row = p.logits + (size_t)r * p.row_stride + from;
    const int k = p.top_k[r];
    const float lim = p.top_p[r];
    const bool by_k = sampled && k > 0 && k < p.V, by_p = sampled && lim < 1.0f;
    auto read = [&](int i) { return logit_key(sampled ? row[i] / temp : row[i]); };
    int count = n;       // the keys that are left here ..
    int packed = 0;      // .. in the row itself, or s.list[packed - 1]
    bool alone = false;  // and nowhere else
    auto key_at = [&](int i) { return packed != 0 ? s.list[packed - 1][i] : (p.staged ? sr_keys[i] : read(i)); };
    auto index_of = [&](int i) { return packed != 0 ? s.index[packed - 1][i] : (unsigned)(from + i); };

    u64 best = 0;  // the largest key, its first index behind it
    auto load = [&](auto scaled) {
        for (int i0 = tid; i0 < n; i0 += SR_LOADS * SR_THREADS) {  // (loads first: a store to shared memory between them would hold the next ones up)
            float l[SR_LOADS];
#pragma unroll
            for (int j = 0; j < SR_LOADS; ++j) l[j] = i0 + j * SR_THREADS < n ? __ldg(row + i0 + j * SR_THREADS) : 0.f;
#pragma unroll
            for (int j = 0; j < SR_LOADS; ++j) {
                const int i = i0 + j * SR_THREADS;
                if (i >= n) break;
                const unsigned key = logit_key(scaled() ? l[j] / temp : l[j]);
                if (scaled() && p.staged) sr_keys[i] = key;
                const u64 cand = ((u64)key << 32) | (u64)(~(unsigned)(from + i));
                best = cand > best ? cand : best;
            }
        }
    };
    if (sampled)
        load([] { return true; });
    else
        load([] { return false; });
    for (int i = tid; i < SR_BINS; i += SR_THREADS) s.low[i] = s.high[i] = 0u;
    const u64 my_best = best;
    best = sr_cluster<SR_MAX>(best, s, 0, false);
    const int best_index = (int)(~(unsigned)(best & 0xffffffffu));
    if (!sampled || (by_p && lim < 0.f)) {  // (a limit below nothing keeps nothing)
        if (rank == 0 && tid == 0) emit_token(r, best_index, p.out, p.row_slot, p.state, p.num_slots);
        sr_cluster_sync();  // (the others may still read this block's word)
        return;
    }
    const float mx = key_to_float((unsigned)(best >> 32));
    auto first_bin = [&](unsigned key) {  // falls with the key; what is no number, the lowest key, goes last
        const float below = mx - key_to_float(key);
        return below < SR_RANGE ? (int)(below * ((SR_BINS - 1) / SR_RANGE)) : SR_BINS - 1;
    };
    // Moves what lies in first bin `bin` or above together, `joint`: in the first block's memory if it fits there, else within
    // each block, and leaves it where it is if it does not fit there either.  false: the first block goes on.
    auto pack = [&](unsigned floor, int bin, bool joint) -> bool {
        const int per = ((count + SR_THREADS - 1) / SR_THREADS) | 1, lo = min(count, tid * per), hi = min(count, lo + per);  // (odd: no bank twice)
        auto left = [&](unsigned key) { return key >= floor && first_bin(key) <= bin; };
        u64 found = 0, here;  // which of the thread's first 64 keys stay
        int mine = 0;
#pragma unroll 4
        for (int i = lo; i < hi; ++i)
            if (left(key_at(i))) {
                if (i - lo < 64) found |= 1ULL << (i - lo);
                ++mine;
            }
        u64 at = sr_scan((u64)mine, s, &here) - (u64)mine;
        bool together = false;
        u64 all = 0, before = 0;
        if (joint) {
            if (tid == 0) s.box[5] = here;
            sr_cluster_sync();
            sr_gather(s, 5);
            for (int c = 0; c < SR_CTAS; ++c) {
                if (c < (int)rank) before += s.gathered[c];
                all += s.gathered[c];
            }
            together = all <= SR_LIST;
        }
        if (!together && (packed != 0 || here > SR_LIST)) return true;
        if (together) at += before;
        const int to = together ? 1 : 0;
        if (mine != 0) {
            const unsigned list = sr_remote(s.list[to], together ? 0 : rank), index = sr_remote(s.index[to], together ? 0 : rank);
            auto put = [&](int i) {
                asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(list + 4 * (unsigned)at), "r"(key_at(i)) : "memory");
                asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(index + 4 * (unsigned)at), "r"(index_of(i)) : "memory");
                ++at;
            };
            for (; found != 0; found &= found - 1) put(lo + __ffsll((long long)found) - 1);
            for (int i = lo + 64; i < hi; ++i)
                if (left(key_at(i))) put(i);
        }
        if (together)
            sr_cluster_sync();
        else
            __syncthreads();
        packed = to + 1;
        alone = together;
        count = (int)(together ? all : here);
        return !together || rank == 0;
    };
    // The key at which the sum over keys >= `floor`, from the top, of 1 or of their masses satisfies the rule.  false: another
    // block goes on.
    auto search = [&](bool masses, unsigned floor, double want, unsigned& found) -> bool {
        u64 far = 0;
#pragma unroll 4
        for (int i = tid; i < count; i += SR_THREADS) {
            const unsigned key = key_at(i);
            if (key < floor) continue;
            const int bin = first_bin(key);
            const u64 v = masses ? mass_of(key_to_float(key), mx) : 1;
            if (bin == SR_BINS - 1)
                far += v;
            else if (v != 0)
                sr_add(s, bin, v, masses);
        }
        far = sr_block<SR_SUM>(far, s);
        if (tid == 0 && far != 0) sr_add(s, SR_BINS - 1, far, masses);
        const int bin = sr_level(s, rank, alone, want, masses ? (double)lim : -1., masses);
        if (!alone && !pack(floor, bin, true)) return false;
        u64 lowest = 0xffffffffu, highest = 0;
        for (int i = tid; i < count; i += SR_THREADS) {
            const unsigned key = key_at(i);
            if (key >= floor && first_bin(key) == bin) {
                lowest = sr_combine<SR_MIN>(lowest, key);
                highest = sr_combine<SR_MAX>(highest, key);
            }
        }
        unsigned lo = (unsigned)sr_cluster<SR_MIN>(lowest, s, 2, alone), hi = (unsigned)sr_cluster<SR_MAX>(highest, s, 3, alone);
        found = 0u;
        if (lo > hi) return true;  // (no key at all: only where no bin qualified)
        while (lo < hi) {
            const int bits = 32 - __clz(hi - lo), shift = bits > 11 ? bits - 11 : 0;
            for (int i = tid; i < count; i += SR_THREADS) {
                const unsigned key = key_at(i);
                if (key < lo || key > hi) continue;
                const u64 v = masses ? mass_of(key_to_float(key), mx) : 1;
                if (v != 0) sr_add(s, (hi - key) >> shift, v, masses);
            }
            const unsigned b = min((unsigned)sr_level(s, rank, alone, want, -1., masses), (hi - lo) >> shift);
            hi -= b << shift;
            const unsigned width = (1u << shift) - 1u;
            lo = hi - lo > width ? hi - width : lo;
        }
        found = hi;
        return true;
    };
    unsigned keep = 0u;
    if (by_k && k <= SR_THREADS) {
        int bin = SR_BINS - 1;
        if (n >= k) {
            if (tid < n) sr_add(s, first_bin((unsigned)(my_best >> 32)), 1, false);
            double want = (double)k;
            bin = sr_level(s, rank, true, want, -1., false);
        }
        pack(0u, bin, false);
    }
    if (by_k && !search(false, 0u, (double)k, keep)) return;
    if (by_p) {
        unsigned found;
        if (!search(true, keep, 0., found)) return;
        keep = max(keep, found);
    }

    // the token: the first index, in index order, at which the kept mass so far exceeds u * total
    u64 mine = 0, all;
    const int per = ((count + SR_THREADS - 1) / SR_THREADS) | 1, my_lo = min(count, tid * per), my_hi = min(count, my_lo + per);
#pragma unroll 4
    for (int i = my_lo; i < my_hi; ++i) {
        const unsigned key = key_at(i);
        if (key >= keep) mine += mass_of(key_to_float(key), mx);
    }
    const u64 incl = sr_scan(mine, s, &all);
    u64 total = all, base = 0;
    int part = 0;
    if (tid == 0) s.first = SR_THREADS;
    if (!alone) total = sr_cluster<SR_SUM>(mine, s, 4, false);
    const double target = (double)p.uniform[r] * (double)total;
    if (!alone)
        for (; part < SR_CTAS && !((double)(base + s.gathered[part]) > target); ++part) base += s.gathered[part];
    __syncthreads();
    if ((int)rank == part && mine > 0 && (double)(base + incl) > target) atomicMin(&s.first, tid);
    __syncthreads();
    if (s.first < SR_THREADS) {
        if (tid == s.first) s.above = base + incl - mine;
        __syncthreads();
        if (tid < 32) {  // the keys of the thread that was first, a lane each
            const int lo = s.first * per, hi = min(count, lo + per);
            u64 run = s.above;
            for (int i = lo + lane; __any_sync(0xffffffffu, i < hi); i += 32) {
                const unsigned key = i < hi ? key_at(i) : 0u;
                const u64 mass = i < hi && key >= keep ? mass_of(key_to_float(key), mx) : 0;
                u64 sum = mass;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const u64 v = __shfl_up_sync(0xffffffffu, sum, o);
                    if (lane >= o) sum += v;
                }
                const unsigned over = __ballot_sync(0xffffffffu, mass > 0 && (double)(run + sum) > target);
                if (over != 0) {
                    if (lane == __ffs(over) - 1) emit_token(r, (int)index_of(i), p.out, p.row_slot, p.state, p.num_slots);
                    break;
                }
                run += __shfl_sync(0xffffffffu, sum, 31);
            }
        }
    } else if (tid == 0 && rank == 0 && (alone || part == SR_CTAS)) {
        emit_token(r, best_index, p.out, p.row_slot, p.state, p.num_slots);  // (no mass: cannot happen while the best key's is 2^40)
    }
    if (!alone) sr_cluster_sync();  // (the others may still read this block's words)
}

// Greedy rows: the first of the largest logits (numbers that are none do not take part), a cluster per row.
// Bound by the latency of the loads, of which every thread has SR_LOADS in flight: 8 rows of 151,936 6 us; with a block of
// 1,024 threads per row 14.
__global__ void __launch_bounds__(SR_THREADS)
argmax_kernel(const float* __restrict__ logits, int* __restrict__ out, int V, size_t row_stride,
              const int* __restrict__ row_slot, int* __restrict__ state, int num_slots) {
    __shared__ u64 mine;
    __shared__ u64 of_warp[SR_WARPS];
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, ctas = gridDim.z, chunk = (V - 1) / ctas + 1, from = min(V, (int)blockIdx.z * chunk), n = min(V, from + chunk) - from;
    const float* row = logits + (size_t)blockIdx.x * row_stride + from;
    float best = -INFINITY;
    int idx = 0x7fffffff;
    for (int i0 = tid; i0 < n; i0 += SR_LOADS * SR_THREADS) {
        float l[SR_LOADS];
#pragma unroll
        for (int j = 0; j < SR_LOADS; ++j) l[j] = i0 + j * SR_THREADS < n ? __ldg(row + i0 + j * SR_THREADS) : NAN;
#pragma unroll
        for (int j = 0; j < SR_LOADS; ++j)
            if (l[j] > best || (l[j] == best && idx == 0x7fffffff)) {  // (indices rise)
                best = l[j];
                idx = from + i0 + j * SR_THREADS;
            }
    }
    u64 all = ((u64)ordered_key(best) << 32) | (u64)(~(unsigned)idx);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) all = sr_combine<SR_MAX>(all, __shfl_xor_sync(0xffffffffu, all, o));
    if ((tid & 31) == 0) of_warp[tid >> 5] = all;
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < SR_WARPS; ++w) all = sr_combine<SR_MAX>(all, of_warp[w]);
        mine = all;
    }
    sr_cluster_sync();
    if (tid == 0 && blockIdx.z == 0) {
        for (int c = 1; c < ctas; ++c) all = sr_combine<SR_MAX>(all, sr_read(&mine, c));
        const int first = (int)(~(unsigned)(all & 0xffffffffu));
        emit_token(blockIdx.x, first == 0x7fffffff ? 0 : first, out, row_slot, state, num_slots);
    }
    sr_cluster_sync();  // (the first block reads the others' words)
}

// row_slot / state (both or neither): see emit_token.
extern "C" int cw_argmax_state(const float* logits, int* out, int R, int V, long long row_stride, const int* row_slot,
                               int* state, int num_slots, cudaStream_t stream) {
    if (R == 0) return CW_OK;
    if (R < 0 || V <= 0 || row_stride < V || (state != nullptr && (row_slot == nullptr || num_slots <= 0))) return CW_ERR_BAD_SIZE;
    int ctas = SR_CTAS;  // as many as the SMs hold at a time, four each (256 rows: 8 blocks a row 40 us, 34 with 2)
    while (ctas > 2 && (long long)R * ctas > 4 * 148) ctas >>= 1;
    // .. and no more than leave a thread a full round of loads (1,000 logits: a cluster's launch and barriers cost a step 2 us)
    while (ctas > 1 && V <= SR_THREADS * SR_LOADS * (ctas / 2)) ctas >>= 1;
    return cw_launch(argmax_kernel, dim3(R, 1, ctas), dim3(SR_THREADS), 0, stream, ctas, logits, out, V, (size_t)row_stride, row_slot,
                     state, num_slots);
}

extern "C" int cw_argmax(const float* logits, int* out, int R, int V, long long row_stride,
                         cudaStream_t stream) {
    return cw_argmax_state(logits, out, R, V, row_stride, nullptr, nullptr, 0, stream);
}

// As cw_sample_state, over SR_CTAS thread blocks per row.
extern "C" int cw_sample_rows(const float* logits, const float* temperature, const int* top_k, const float* top_p,
                              const float* uniform, int* out, int R, int V, long long row_stride, const int* row_slot,
                              int* state, int num_slots, cudaStream_t stream) {
    if (R == 0) return CW_OK;
    if (R < 0 || V <= 0 || row_stride < V || (state != nullptr && (row_slot == nullptr || num_slots <= 0))) return CW_ERR_BAD_SIZE;
    if (R > 65535) return CW_ERR_BAD_SIZE;
    const int chunk = (V - 1) / SR_CTAS + 1, staged = chunk <= SR_STAGED;
    const SampleParams p = {logits, (size_t)row_stride, V, temperature, top_k, top_p, uniform, out, row_slot, state, num_slots, chunk, staged};
    const size_t smem = staged ? (size_t)chunk * sizeof(unsigned) : 0;
    if (smem > (12u << 10)) {  // (with the tables, beyond the 48 KB that need no asking)
        const cudaError_t e = cudaFuncSetAttribute(sample_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SR_STAGED * (int)sizeof(unsigned));
        if (e != cudaSuccess) return (int)e;
    }
    return cw_launch(sample_rows_kernel, dim3(R, 1, SR_CTAS), dim3(SR_THREADS), smem, stream, SR_CTAS, p);
}

CW_TRACE_TU(sampling)
