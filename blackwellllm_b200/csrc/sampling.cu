// Token choice from float32 logits [R, V], a cluster of 8 blocks per row, or one block for short rows and for many.
//
//  * temperature <= 0: argmax, the lowest index winning a tie.
//  * temperature  > 0: softmax(logits / temperature) in float32; optional nucleus
//    (top_p < 1): keep the most probable tokens whose mass reaches top_p (all
//    tokens tied with the last one kept are kept too); then the inverse CDF over
//    the kept tokens IN INDEX ORDER at the uniform number u[r] given by the host.
//    The draw therefore depends on (logits row, u) only, not on the batch.
//
// Beside it: the repetition penalty on a row's logits before the choice, and the log
// probability of a given token (the reference's src/kernels/sampling.cu:85-118 and 213-247).
#include "common.cuh"
#include <cooperative_groups.h>

namespace {

namespace cg = cooperative_groups;
typedef unsigned long long u64;

constexpr int THREADS = 1024;
constexpr int WARPS = THREADS / 32;
constexpr int ROW_BLOCKS = 8;       // blocks of a row, a cluster
constexpr int BINS = 1024;          // one per thread: ten bits of a weight's float pattern at a time

__device__ __forceinline__ void argmax_pair(float& v, int& i, float ov, int oi) {
    if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}
__device__ __forceinline__ u64 warp_sum_u64(u64 v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ u64 warp_scan_u64(u64 v) {   // inclusive
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// A histogram of masses as two words per bin (shared memory adds 32-bit integers natively).
struct Hist { unsigned lo[BINS], hi[BINS]; };
__device__ __forceinline__ void hist_add(Hist& h, unsigned bin, u64 q) {
    const unsigned low = (unsigned)q;
    const unsigned old = atomicAdd(&h.lo[bin], low);
    const unsigned up = (unsigned)(q >> 32) + (old + low < old ? 1u : 0u);
    if (up) atomicAdd(&h.hi[bin], up);
}

// One row per cluster (of CLUSTER blocks).  The weights e = exp((x - max) / T) are made once and stay in registers (NV a thread; NV = 0: a row too
// long for that is read again for every pass) or, with more rows than clusters that fit at one block an SM, in shared memory (IN_SMEM:
// two blocks an SM at 32 registers a thread).  Masses are integers, e * 2^shift rounded (`scale` = 2^shift, shift at most 45 and
// such that a row's mass fits 62 bits): their sums are exact in any order, so the blocks of a row may add them as they come.
// The nucleus threshold, the largest weight whose mass together with all larger ones reaches the target, is found ten bits of the
// float pattern at a time (30 bits: e <= 1) from histograms that the blocks read from one another's shared memory: three passes
// over registers, in place of the 30 passes over the row that a bisection takes.
// What bounds it: latency (five cluster barriers, three histogram passes); a row of 128,256 is 0.5 MB.  Measured, temperature 0.6,
// top_p 0.9: a row of 128,256 in 26 us, 32 rows of 152,064 in 63 us (79 in registers; one block per row and the bisection: 728 and
// 1,162 us).
template <int NV, bool IN_SMEM = false, int CLUSTER = ROW_BLOCKS>
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(THREADS, IN_SMEM || (NV == 0 && CLUSTER == 1) ? 2 : 1)
sample_kernel(const float* __restrict__ logits, const float* __restrict__ temperature,
              const float* __restrict__ top_p, const float* __restrict__ u, int* __restrict__ out,
              int V, size_t ld, float scale) {
    BW_PDL_TRIGGER();
    BW_PDL_WAIT();
    extern __shared__ float kept_smem[];        // IN_SMEM: [WARPS][per_warp]
    __shared__ Hist hist[3];
    __shared__ float sv[WARPS], all_max[CLUSTER];
    __shared__ int si[WARPS], all_arg[CLUSTER];
    __shared__ u64 sums[WARPS], all_mass[CLUSTER], above;
    __shared__ unsigned bin_found;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), r = blockIdx.x / CLUSTER;
    cluster.barrier_arrive();       // (waited for before the first access to another block's memory: that block has then begun)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float* row = logits + (size_t)r * ld;
    const float T = temperature ? temperature[r] : 0.f;
    const bool greedy = !(T > 0.f);
    const float tp = (!greedy && top_p) ? top_p[r] : 1.f;

    // this warp's tokens: a contiguous stretch of the block's contiguous stretch of the row
    const int per_block = (V + CLUSTER - 1) / CLUSTER;
    const int per_warp = ((per_block + WARPS - 1) / WARPS + 31) & ~31;
    const int iters = per_warp >> 5;
    const long long block_end = (long long)(rank + 1) * per_block;
    const int end = (int)(block_end < V ? block_end : V);
    const long long start = (long long)rank * per_block + (long long)warp * per_warp + lane;
    const int first = (int)(start < V ? start : V), left = min(end - first, per_warp - lane);   // the token 32 i behind the first: where 32 i < left
    constexpr int KEEP = NV > 0 ? NV : 1;
    float e[KEEP];

    float mx = -INFINITY;
    int arg = 0x7fffffff;
    if constexpr (NV > 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) e[i] = 32 * i < left ? row[first + 32 * i] : -INFINITY;
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (32 * i < left) argmax_pair(mx, arg, e[i], first + 32 * i);
    } else {
#pragma unroll 4
        for (int i = 0; i < iters; ++i) {
            const float x = 32 * i < left ? row[first + 32 * i] : -INFINITY;
            if constexpr (IN_SMEM) kept_smem[warp * per_warp + 32 * i + lane] = x;
            if (32 * i < left) argmax_pair(mx, arg, x, first + 32 * i);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, mx, o);
        const int oi = __shfl_xor_sync(0xffffffffu, arg, o);
        argmax_pair(mx, arg, ov, oi);
    }
    if (lane == 0) { sv[warp] = mx; si[warp] = arg; }
    if (tp < 1.f)
        for (int i = tid; i < 3 * BINS; i += THREADS) { hist[i / BINS].lo[i % BINS] = 0; hist[i / BINS].hi[i % BINS] = 0; }
    cluster.barrier_wait();
    __syncthreads();
    if (warp == 0) {
        mx = sv[lane]; arg = si[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, mx, o);
            const int oi = __shfl_xor_sync(0xffffffffu, arg, o);
            argmax_pair(mx, arg, ov, oi);
        }
        if (lane < CLUSTER) {
            *cluster.map_shared_rank(&all_max[rank], lane) = mx;
            *cluster.map_shared_rank(&all_arg[rank], lane) = arg;
        }
    }
    cluster.sync();
    mx = all_max[0]; arg = all_arg[0];
#pragma unroll
    for (int c = 1; c < CLUSTER; ++c) argmax_pair(mx, arg, all_max[c], all_arg[c]);
    if (greedy) {
        if (rank == 0 && tid == 0) out[r] = arg == 0x7fffffff ? 0 : arg;
        return;
    }

    const float invT = 1.f / T;
    auto weight = [&](int i) {     // of this thread's i-th token; -1: there is none
        if constexpr (NV > 0) return e[i];
        else if constexpr (IN_SMEM) return kept_smem[warp * per_warp + 32 * i + lane];
        else return 32 * i < left ? expf((row[first + 32 * i] - mx) * invT) : -1.f;
    };
    auto mass = [&](float w) { return __float2ull_rn(w * scale); };
    const int passes = NV > 0 ? NV : iters;
    if constexpr (NV > 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) e[i] = 32 * i < left ? expf((e[i] - mx) * invT) : -1.f;
    }
    if constexpr (IN_SMEM) {       // (each thread its own)
        for (int i = 0; i < iters; ++i) {
            float& k = kept_smem[warp * per_warp + 32 * i + lane];
            k = 32 * i < left ? expf((k - mx) * invT) : -1.f;
        }
    }
    float tau = 0.f;
    if (tp < 1.f) {
        // bits 29..20, then 19..10, then 9..0 of the weights that share the bits found so far
        unsigned prefix = 0;
        u64 target = 0;
        bool nucleus = true;
#pragma unroll
        for (int round = 0; round < 3; ++round) {
            const int shift = 20 - 10 * round;
#pragma unroll
            for (int i = 0; i < passes; ++i) {
                const float w = weight(i);
                const unsigned bits = __float_as_uint(w);
                if (w > 0.f && (round == 0 || (bits >> (shift + 10)) == prefix)) hist_add(hist[round], (bits >> shift) & (BINS - 1), mass(w));
                // a weight that is no number leaves the mass undefined: every token is kept then
                if (round == 0 && w != w) hist[0].hi[BINS - 1] = 1u;
            }
            cluster.sync();
            // this thread's bin, counted from the largest weights; a weight is at most 1, so bins 1017.. of the first pass stay empty
            const unsigned bin = BINS - 1 - tid;
            u64 m = 0;
#pragma unroll
            for (int c = 0; c < CLUSTER; ++c) {
                const Hist* h = cluster.map_shared_rank(&hist[round], c);
                m += ((u64)h->hi[bin] << 32) + h->lo[bin];
            }
            if (round == 0 && __syncthreads_or(tid == 0 && m != 0)) { nucleus = false; break; }
            u64 sum = warp_scan_u64(m);
            if (lane == 31) sums[warp] = sum;
            __syncthreads();
            u64 before = 0, total = 0;
#pragma unroll 8
            for (int w = 0; w < WARPS; ++w) { const u64 s = sums[w]; total += s; if (w < warp) before += s; }
            sum += before;
            if (round == 0) {
                target = __double2ull_ru((double)tp * (double)total);
                if (target < 1) target = 1;        // (top_p <= 0 keeps the most probable token)
                if (target > total) target = total;
            }
            if (sum - m < target && target <= sum) { bin_found = bin; above = sum - m; }
            if (tid == 0 && total == 0) { bin_found = 0; above = 0; }
            __syncthreads();
            prefix = (prefix << 10) | bin_found;
            target -= above;
        }
        if (nucleus) tau = __uint_as_float(prefix);
    }

    // the kept mass of every warp, of every block; then the block and the warp that the draw falls into walk their tokens
    u64 kept = 0;
#pragma unroll
    for (int i = 0; i < passes; ++i) { const float w = weight(i); if (w >= tau) kept += mass(w); }
    kept = warp_sum_u64(kept);
    __syncthreads();
    if (lane == 0) sums[warp] = kept;
    __syncthreads();
    if (warp == 0) {
        const u64 s = warp_sum_u64(sums[lane]);
        if (lane < CLUSTER) *cluster.map_shared_rank(&all_mass[rank], lane) = s;
    }
    cluster.sync();      // (also: nobody leaves while another block may read its histograms)
    u64 total = 0, before = 0;
#pragma unroll
    for (int c = 0; c < CLUSTER; ++c) { if (c < rank) before += all_mass[c]; total += all_mass[c]; }
    if (total == 0) {    // no token has a weight (a row of infinities or of none): the last of the first tokens whose weight is a number
        if (rank == 0 && tid == 0) {
            int last = -1;
            for (int c = 0; c < min(V, (V + THREADS - 1) / THREADS); ++c)
                if (expf((row[c] - mx) * invT) >= tau) last = c;
            out[r] = last;
        }
        return;
    }
    const double at = (double)u[r] * (double)total;
    u64 goal = at > 0.0 ? __double2ull_rd(at) : 0;
    if (goal >= total) goal = total - 1;
    for (int w = 0; w < warp; ++w) before += sums[w];
    if (goal < before || goal >= before + kept) return;
#pragma unroll
    for (int i = 0; i < passes; ++i) {
        const float w = weight(i);
        const u64 upto = before + warp_scan_u64(w >= tau ? mass(w) : 0);
        const unsigned past = __ballot_sync(0xffffffffu, upto > goal);
        if (past) {
            if (lane == __ffs(past) - 1) out[r] = first + 32 * i;
            return;
        }
        before = __shfl_sync(0xffffffffu, upto, 31);
    }
}

// The greedy choice of one row per block: the row is read once and nothing else is done.
__global__ void __launch_bounds__(THREADS)
argmax_kernel(const float* __restrict__ logits, int* __restrict__ out, int V, size_t ld) {
    BW_PDL_TRIGGER();
    BW_PDL_WAIT();
    __shared__ float sv[WARPS];
    __shared__ int si[WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float* row = logits + (size_t)blockIdx.x * ld;
    float mx = -INFINITY;
    int arg = 0x7fffffff;
    for (int c = threadIdx.x; c < V; c += THREADS) argmax_pair(mx, arg, row[c], c);
    auto over_warp = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, mx, o);
            const int oi = __shfl_xor_sync(0xffffffffu, arg, o);
            argmax_pair(mx, arg, ov, oi);
        }
    };
    over_warp();
    if (lane == 0) { sv[warp] = mx; si[warp] = arg; }
    __syncthreads();
    if (warp) return;
    mx = sv[lane]; arg = si[lane];
    over_warp();
    if (lane == 0) out[blockIdx.x] = arg == 0x7fffffff ? 0 : arg;
}

// Repetition penalty in place, one block per row: every DISTINCT id of the row's history
// ids[begin[r] .. begin[r+1]) has its logit divided by penalty[r] when positive and multiplied
// by it when not, once however often the id occurs (only an id's first occurrence acts).
// penalty <= 1 and ids outside [0, V) do nothing.
__global__ void repetition_penalty_kernel(float* __restrict__ logits, const int* __restrict__ ids,
                                          const int* __restrict__ begin, const float* __restrict__ penalty,
                                          int V, size_t ld) {
    BW_PDL_TRIGGER();
    BW_PDL_WAIT();
    const int r = blockIdx.x;
    const float pen = penalty[r];
    if (!(pen > 1.f)) return;
    const int* mine = ids + begin[r];
    const int n = begin[r + 1] - begin[r];
    float* row = logits + (size_t)r * ld;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int id = mine[i];
        if (id < 0 || id >= V) continue;
        bool first = true;
        for (int j = 0; j < i && first; ++j) first = mine[j] != id;
        if (!first) continue;
        const float v = row[id];
        row[id] = v > 0.f ? v / pen : v * pen;
    }
}

// log softmax(row)[target[r]] per row, float32: (x_t - max) - log(sum exp(x - max)).
__global__ void __launch_bounds__(THREADS)
log_prob_kernel(const float* __restrict__ logits, const int* __restrict__ target, float* __restrict__ out,
                int V, size_t ld) {
    BW_PDL_TRIGGER();
    BW_PDL_WAIT();
    __shared__ float sf[32];
    const int r = blockIdx.x;
    const float* row = logits + (size_t)r * ld;
    float mx = -INFINITY;
    for (int c = threadIdx.x; c < V; c += blockDim.x) mx = fmaxf(mx, row[c]);
    mx = bw::block_max(mx, sf);
    float s = 0.f;
    for (int c = threadIdx.x; c < V; c += blockDim.x) s += expf(row[c] - mx);
    s = bw::block_sum(s, sf);
    if (threadIdx.x == 0) out[r] = (row[target[r]] - mx) - logf(s);
}

}  // namespace

BW_EXPORT int bw_repetition_penalty(float* logits, const int* ids, const int* begin, const float* penalty,
                                    int R, int V, long long ld, void* stream) {
    if (R <= 0) return 0;
    if (V <= 0 || ld < V || !ids || !begin || !penalty) return BW_ERR_BAD_ARG;
    bw::launch((repetition_penalty_kernel), dim3(R), dim3(256), 0, (cudaStream_t)stream, logits, ids, begin, penalty,
               V, (size_t)ld);
    BW_LAUNCH_CHECK();
    return 0;
}

// target[r] must lie in [0, V): the caller checks it on the host.
BW_EXPORT int bw_log_prob(const float* logits, const int* target, float* out, int R, int V, long long ld,
                          void* stream) {
    if (R <= 0) return 0;
    if (V <= 0 || ld < V || !target || !out) return BW_ERR_BAD_ARG;
    bw::launch((log_prob_kernel), dim3(R), dim3(THREADS), 0, (cudaStream_t)stream, logits, target, out, V, (size_t)ld);
    BW_LAUNCH_CHECK();
    return 0;
}

// temperature, top_p: per row (may be null: greedy / no nucleus); u: per row uniform in [0,1).
BW_EXPORT int bw_sample(const float* logits, const float* temperature, const float* top_p, const float* u,
                        int* out, int R, int V, long long ld, void* stream) {
    if (R <= 0) return 0;
    if (V <= 0 || ld < V) return BW_ERR_BAD_ARG;
    if (temperature && !u) return BW_ERR_BAD_ARG;
    int bits = 0;
    while ((1ll << bits) < V) ++bits;
    const float scale = (float)(1ull << (62 - bits < 45 ? 62 - bits : 45));
    const dim3 block(THREADS);
    // The greedy choice alone needs one pass, and clusters take turns of 17 rows or so: a block a row, but for a few long rows (us on
    // clusters and in blocks: 8 rows of 24,000 3.1 and 3.2, of 32,000 3.2 and 3.8, of 128,256 4.1 and 8.1; 18 of 32,000 5.4 and 3.8; 36
    // of 128,256 10.4 and 8.3; 256 of them 71 and 25; 18 of 200,000 14.6 and 11.2).
    if (!temperature && (V <= 24 * 1024 || R > (V > 100 * 1024 && V <= 160 * 1024 ? 32 : 16))) {
        bw::launch(argmax_kernel, dim3((unsigned)R), block, 0, (cudaStream_t)stream, logits, out, V, (size_t)ld);
        BW_LAUNCH_CHECK();
        return 0;
    }
    // Else one block a row where that is faster: a row that fits a block's registers (64 rows of 5,000: nucleus 14 us, 69 on clusters;
    // alone 13 and 20), or so many rows that their clusters take turns for longer than a block walks its row (temperature / nucleus, on
    // clusters and in blocks: 64 rows of 32,000 19 / 75 and 27 / 63, 128 of 64,000 47 / 158 and 55 / 137, 256 of 128,256 168 / 404 and
    // 156 / 365; of 256,000, which a cluster's registers do not hold, 479 / 1,180 and 323 / 717).
    if (V <= 8 * THREADS || R > (V > 160 * 1024 ? 100 : V / 512)) {
        const auto kernel = V <= 8 * THREADS ? sample_kernel<8, false, 1> : sample_kernel<0, false, 1>;
        bw::launch(kernel, dim3((unsigned)R), block, 0, (cudaStream_t)stream, logits, temperature, top_p, u, out, V, (size_t)ld, scale);
        BW_LAUNCH_CHECK();
        return 0;
    }
    // tokens of a thread: its warp's share of the block's share of the row, in rows of 32
    const int per_block = (V + ROW_BLOCKS - 1) / ROW_BLOCKS;
    const int iters = ((per_block + WARPS - 1) / WARPS + 31) / 32;
    const dim3 grid((unsigned)R * ROW_BLOCKS);
    // more rows than clusters at one block an SM: two blocks an SM, weights in shared memory (19 rows of 152,064 61 us, 32 63 us; in registers 79)
    const int at_once = bw::num_sms() / ROW_BLOCKS;
    const size_t kept = (size_t)iters * 32 * WARPS * sizeof(float);
    if (temperature && R > at_once && kept <= 80 * 1024) {      // (two blocks and their histograms in an SM's shared memory)
        static bool done[bw::MAX_DEVICES] = {};
        if (const cudaError_t e = bw::allow_dynamic_smem(sample_kernel<0, true>, 80 * 1024, done); e != cudaSuccess) return (int)e;
        bw::launch(sample_kernel<0, true>, grid, block, kept, (cudaStream_t)stream, logits, temperature, top_p, u, out, V, (size_t)ld, scale);
        BW_LAUNCH_CHECK();
        return 0;
    }
#define BW_SAMPLE(NV) bw::launch(sample_kernel<NV>, grid, block, 0, (cudaStream_t)stream, logits, temperature, top_p, u, out, V, (size_t)ld, scale)
    // registers for 8 tokens a thread (rows up to 65,536) or 20 (up to 163,840: 64 registers a thread allow no more); longer rows are
    // read again for every pass (a row of 200,000 in 54 us, 32 rows in 146)
    if (iters <= 8) BW_SAMPLE(8);
    else if (iters <= 20) BW_SAMPLE(20);
    else BW_SAMPLE(0);
#undef BW_SAMPLE
    BW_LAUNCH_CHECK();
    return 0;
}
