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
constexpr int VALUE_ROWS = 64;      // rows whose parameters travel with the launch

// The rows' parameters: arrays on the device (any null: greedy, or no nucleus), or values in the launch itself.
struct Rows {
    const float *temperature, *top_p, *u;
    int by_value;
    float v[3][VALUE_ROWS];
};

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

// What the warps before this one left in sums[], and all warps: the same in all lanes.
__device__ __forceinline__ void over_warps(const u64* sums, u64& before, u64& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u64 mine = sums[lane], upto = warp_scan_u64(mine);
    total = __shfl_sync(0xffffffffu, upto, 31);
    before = __shfl_sync(0xffffffffu, upto - mine, warp);
}

// A histogram of masses as two words per bin (shared memory adds 32-bit integers natively).
struct Hist { unsigned lo[BINS], hi[BINS]; };
__device__ __forceinline__ void hist_add(Hist& h, unsigned bin, u64 q) {
    const unsigned low = (unsigned)q;
    const unsigned old = atomicAdd(&h.lo[bin], low);
    const unsigned up = (unsigned)(q >> 32) + (old + low < old ? 1u : 0u);
    if (up) atomicAdd(&h.hi[bin], up);
}

// The cuts of the lists of largest weights, from the highest: 2^-6, 2^-8 .. 2^-16 of the largest; a row's lists have LISTED tokens at most.
constexpr int LEVELS = 6, LISTED = 4 * THREADS;
__device__ __forceinline__ float level_cut(int l) { return __uint_as_float((unsigned)(127 - 6 - 2 * l) << 23); }

// One row per cluster (of CLUSTER blocks).  The weights e = exp((x - max) / T) are made once and stay in registers (NV a thread; NV = 0: a row too
// long for that is read again for every pass) or, with more rows than clusters that fit at one block an SM, in shared memory (IN_SMEM:
// two blocks an SM at 32 registers a thread).  Masses are integers, e * 2^shift rounded (`scale` = 2^shift, shift at most 45 and
// such that a row's mass fits 62 bits): their sums are exact in any order, so the blocks of a row may add them as they come.
// The nucleus threshold, the largest weight whose mass together with all larger ones reaches the target, is found ten bits of the
// float pattern at a time (30 bits: e <= 1) from histograms that the blocks read from one another's shared memory: three passes
// over registers, in place of the 30 passes over the row that a bisection takes.
// Before that, the nucleus is looked for among the row's largest weights alone: every block lists its tokens down to the lowest of LEVELS
// cuts of which it has few enough, in index order, and the row's first block, with all lists and the row's mass, selects and draws
// among them by itself: up to 32 tokens in one warp, more (up to four a thread) from histograms of its own.  Where they do not reach the
// target mass (a flat row), or a weight is no number, the histograms over all blocks decide; both find the same token.
// What bounds it: latency (three cluster barriers without a nucleus, four with the list, eight with the histograms over all blocks; 20
// exponentials, masses and votes a thread); a row of 128,256 is 0.5 MB.  Measured, temperature 0.6, top_p 0.9, logits as a language model gives them: a row of 128,256 in 14 us, 32 rows
// of 152,064 in 32 us (25 and 61 with the histograms over all blocks alone; one block per row and a bisection: 728 and 1,162).
template <int NV, bool IN_SMEM = false, int CLUSTER = ROW_BLOCKS>
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(THREADS, IN_SMEM || (NV == 0 && CLUSTER == 1) ? 2 : 1)
sample_kernel(const float* __restrict__ logits, const __grid_constant__ Rows rows, int* __restrict__ out,
              int V, size_t ld, float scale) {
    BW_PDL_TRIGGER();
    BW_PDL_WAIT();
    extern __shared__ float kept_smem[];        // IN_SMEM: [WARPS][per_warp]
    __shared__ Hist hist[3];
    __shared__ float sv[WARPS], all_max[CLUSTER];
    __shared__ int si[WARPS], all_arg[CLUSTER];
    __shared__ u64 sums[WARPS], all_mass[CLUSTER], above;
    __shared__ unsigned bin_found, all_cut[CLUSTER];
    __shared__ int all_listed[CLUSTER], counts[LEVELS][WARPS], own_level, again;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), r = blockIdx.x / CLUSTER;
    cluster.barrier_arrive();       // (waited for before the first access to another block's memory: that block has then begun)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float* row = logits + (size_t)r * ld;
    const float T = rows.by_value ? rows.v[0][r] : rows.temperature ? rows.temperature[r] : 0.f;
    const bool greedy = !(T > 0.f);
    const float tp = greedy ? 1.f : rows.by_value ? rows.v[1][r] : rows.top_p ? rows.top_p[r] : 1.f;

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
    } else if constexpr (IN_SMEM) {
        // (each lane its own tokens, all asked for at once: through registers, four at a time, the 19 of 152,064 took 12 us)
        float* to = kept_smem + warp * per_warp + lane;
        for (int i = 0; i < iters; ++i)
            if (32 * i < left)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(to + 32 * i)), "l"(row + first + 32 * i) : "memory");
        asm volatile("cp.async.wait_all;" ::: "memory");
        for (int i = 0; 32 * i < left; ++i) argmax_pair(mx, arg, to[32 * i], first + 32 * i);
    } else {
#pragma unroll 4
        for (int i = 0; i < iters; ++i) {
            const float x = 32 * i < left ? row[first + 32 * i] : -INFINITY;
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
    auto make_weight = [&](int i) {     // from the logit that is kept
        if constexpr (NV > 0) e[i] = 32 * i < left ? expf((e[i] - mx) * invT) : -1.f;
        else if constexpr (IN_SMEM) {
            float& k = kept_smem[warp * per_warp + 32 * i + lane];
            k = 32 * i < left ? expf((k - mx) * invT) : -1.f;
        }
        return weight(i);
    };
    auto mass = [&](float w) { return __float2ull_rn(w * scale); };
    const int passes = NV > 0 ? NV : iters;
    const float uniform = rows.by_value ? rows.v[2][r] : rows.u[r];
    // this thread's bin of a histogram, counted from the largest weights, m its mass: where the target lies
    auto select = [&](unsigned bin, u64 m, auto&& set_target, u64& target, unsigned& prefix) {
        u64 sum = warp_scan_u64(m);
        if (lane == 31) sums[warp] = sum;
        __syncthreads();
        u64 before, total;
        over_warps(sums, before, total);
        sum += before;
        set_target(total);
        if (sum - m < target && target <= sum) { bin_found = bin; above = sum - m; }
        if (tid == 0 && total == 0) { bin_found = 0; above = 0; }
        __syncthreads();
        prefix = (prefix << 10) | bin_found;
        target -= above;
    };
    auto nucleus_target = [&](u64 total) {
        u64 t = __double2ull_ru((double)tp * (double)total);
        if (t < 1) t = 1;        // (top_p <= 0 keeps the most probable token)
        return t > total ? total : t;
    };
    auto drawn = [&](u64 total) {
        const double at = (double)uniform * (double)total;
        const u64 goal = at > 0.0 ? __double2ull_rd(at) : 0;
        return goal >= total ? total - 1 : goal;
    };

    if (!(tp < 1.f)) {
        if constexpr (NV > 0 || IN_SMEM) {
#pragma unroll
            for (int i = 0; i < passes; ++i) make_weight(i);
        }
    } else {
        // the weights, their mass, and how many tokens lie above each cut
        u64 q = 0;
        int many[LEVELS] = {};
        bool number = true;
#pragma unroll
        for (int i = 0; i < passes; ++i) {
            const float w = make_weight(i), x = w * scale;
            number &= w == w;
            // (most masses fit 32 bits, whose conversion is a fraction of the other's)
            if (x < 0x1p31f) q += __float2uint_rn(x);              // (none: -1, no mass)
            if (__any_sync(0xffffffffu, !(x < 0x1p31f))) { if (x >= 0x1p31f) q += mass(w); }
            if (__any_sync(0xffffffffu, w >= level_cut(LEVELS - 1))) {
#pragma unroll
                for (int l = 0; l < LEVELS; ++l) many[l] += __popc(__ballot_sync(0xffffffffu, w >= level_cut(l)));
            }
        }
        q = warp_sum_u64(q);
        number = __all_sync(0xffffffffu, number);
        if (lane == 0) {
            sums[warp] = q;
#pragma unroll
            for (int l = 0; l < LEVELS; ++l) counts[l][warp] = number ? many[l] : LISTED + 1;
        }
        __syncthreads();
        if (warp == 0) {
            const u64 block = warp_sum_u64(sums[lane]);
            int l = LEVELS - 1, listed = 0, mine = 0;
            for (; l >= 0; --l) {
                mine = counts[l][lane];
                listed = __reduce_add_sync(0xffffffffu, mine);
                if (listed <= (CLUSTER > 1 ? LISTED / CLUSTER : BINS)) break;
            }
            int upto = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, upto, o); if (lane >= o) upto += t; }
            si[lane] = upto - mine;             // where this warp's tokens begin in the block's list
            const unsigned cut = l < 0 ? 0xffffffffu : __float_as_uint(level_cut(l));
            if (lane < CLUSTER) {
                *cluster.map_shared_rank(&all_mass[rank], lane) = block;
                *cluster.map_shared_rank(&all_listed[rank], lane) = l < 0 ? 0 : listed;
                *cluster.map_shared_rank(&all_cut[rank], lane) = cut;
            }
            if (lane == 0) { bin_found = cut; own_level = l; }
        }
        __syncthreads();
        Hist& list = hist[2];                   // the block's list: weights, tokens
        if (own_level >= 0 && counts[own_level][warp] > 0) {
            const float own_cut = __uint_as_float(bin_found);
            int at = si[warp];
#pragma unroll
            for (int i = 0; i < passes; ++i) {
                const float w = weight(i);
                const bool in = w >= own_cut;
                const unsigned who = __ballot_sync(0xffffffffu, in);
                if (in) {
                    const int to = at + __popc(who & ((1u << lane) - 1));
                    list.lo[to] = __float_as_uint(w);
                    list.hi[to] = (unsigned)(first + 32 * i);
                }
                at += __popc(who);
            }
        }
        cluster.sync();
        if (rank == 0) {
            u64 total = 0;
            unsigned cut = 0;
            int n = 0;
#pragma unroll
            for (int c = 0; c < CLUSTER; ++c) { total += all_mass[c]; cut = max(cut, all_cut[c]); n += all_listed[c]; }
            // entry j of the blocks' lists end to end (tokens in index order); one below the row's cut counts as none
            auto entry = [&](int j, unsigned& bits, unsigned& token) {
                int c = 0;
                bits = token = 0;
                if (j >= n) return;
                while (j >= all_listed[c]) j -= all_listed[c++];
                const Hist* h = cluster.map_shared_rank(&hist[2], c);
                bits = h->lo[j]; token = h->hi[j];
                if (bits < cut) bits = 0;
            };
            u64 target = nucleus_target(total);
            bool found = false;
            if (cut == 0xffffffffu || total == 0 || n == 0) {
                // the histograms decide
            } else if (n <= 32) {
                if (warp == 0) {                // a lane an entry, all in one warp
                    unsigned bits, token;
                    entry(lane, bits, token);
                    const u64 m = bits ? mass(__uint_as_float(bits)) : 0;
                    u64 larger = 0, upto = 0;   // the mass of larger weights; of those and this weight's ties
                    for (int k = 0; k < n; ++k) {
                        const unsigned b = __shfl_sync(0xffffffffu, bits, k);
                        const u64 mk = __shfl_sync(0xffffffffu, m, k);
                        if (b > bits) larger += mk;
                        if (b >= bits) upto += mk;
                    }
                    const unsigned hit = __ballot_sync(0xffffffffu, m && larger < target && target <= upto);
                    found = hit != 0;
                    if (found) {
                        const unsigned least = __shfl_sync(0xffffffffu, bits, __ffs(hit) - 1);
                        const u64 kept = bits >= least ? m : 0, sum = warp_scan_u64(kept);
                        const u64 goal = drawn(__shfl_sync(0xffffffffu, sum, 31));
                        if (kept && goal < sum && goal >= sum - kept) out[r] = (int)token;
                    }
                }
            } else {
                constexpr int PER = LISTED / THREADS;
                const int per = (n + THREADS - 1) / THREADS;
                unsigned bits[PER], token[PER];
                u64 reached = 0;
#pragma unroll
                for (int k = 0; k < PER; ++k) {
                    bits[k] = token[k] = 0;
                    if (k < per) entry(tid * per + k, bits[k], token[k]);
                    if (bits[k]) reached += mass(__uint_as_float(bits[k]));
                }
                reached = warp_sum_u64(reached);
                __syncthreads();                // (the list has been read, sums too)
                if (lane == 0) sums[warp] = reached;
                hist[2].lo[tid] = hist[2].hi[tid] = 0;
                __syncthreads();
                u64 before;
                over_warps(sums, before, reached);
                found = reached >= target;
                if (found) {
                    unsigned prefix = 0;
#pragma unroll
                    for (int round = 0; round < 3; ++round) {
                        const int shift = 20 - 10 * round;
#pragma unroll
                        for (int k = 0; k < PER; ++k)
                            if (bits[k] && (round == 0 || (bits[k] >> (shift + 10)) == prefix))
                                hist_add(hist[round], (bits[k] >> shift) & (BINS - 1), mass(__uint_as_float(bits[k])));
                        __syncthreads();
                        const unsigned bin = BINS - 1 - tid;
                        select(bin, ((u64)hist[round].hi[bin] << 32) + hist[round].lo[bin], [](u64) {}, target, prefix);
                    }
                    u64 kept = 0;
#pragma unroll
                    for (int k = 0; k < PER; ++k) kept += bits[k] >= prefix && bits[k] ? mass(__uint_as_float(bits[k])) : 0;
                    u64 upto = warp_scan_u64(kept), all;
                    if (lane == 31) sums[warp] = upto;
                    __syncthreads();
                    over_warps(sums, before, all);
                    upto += before - kept;
                    const u64 goal = drawn(all);
#pragma unroll
                    for (int k = 0; k < PER; ++k) {
                        const u64 m = bits[k] >= prefix && bits[k] ? mass(__uint_as_float(bits[k])) : 0;
                        if (m && goal >= upto && goal < upto + m) out[r] = (int)token[k];
                        upto += m;
                    }
                }
            }
            if (warp == 0 && lane < CLUSTER) *cluster.map_shared_rank(&again, lane) = !found;
        }
        cluster.sync();
        if (!again) return;
        if (rank == 0)       // (the other blocks' first two are as they were)
            for (int i = tid; i < 2 * BINS; i += THREADS) hist[i / BINS].lo[i % BINS] = hist[i / BINS].hi[i % BINS] = 0;
        hist[2].lo[tid] = hist[2].hi[tid] = 0;
        __syncthreads();
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
            select(bin, m, [&](u64 total) { if (round == 0) target = nucleus_target(total); }, target, prefix);
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
    const u64 goal = drawn(total);
    u64 mine, block;
    over_warps(sums, mine, block);
    before += mine;
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

// Whether rows that are not all greedy take a block each, not a cluster: a row that fits a block's registers, or so many rows that their
// clusters take turns for longer than a block walks its row.  With a nucleus a block walks it several times, so the line depends on it.
// Temperature alone, us, on clusters and in blocks, logits from memory: 32 rows of 9,000 10.5 and 11.0, 48 of them 16.6 and 11.3; 128 of
// 32,000 39 and 42, 160 of them 48 and 43; 200 of 64,000 70 and 77, 256 of them 88 and 79; 512 of 100,000 214 and 228; 256 of 128,256
// 120 and 166; rows that a cluster's registers do not hold: 128 of 170,000 173 and 182, 160 of them 213 and 201, 160 of 256,000 297 and
// 314, 200 of them 376 and 323.  With a nucleus, likely tokens few: 32 of 9,000 15 and 16, 64 of them 25 and 17; 128 of 32,000 52 and 54, 256
// of them 96 and 73; 256 of 64,000 120 and 181, 1,024 of them 448 and 367; 256 of 128,256 162 and 361; 128 of 200,000 286 and 517, 256
// of them 559 and 594.
BW_EXPORT int bw_sample_row_in_a_block(int R, int V, int nucleus) {
    if (V <= 8 * THREADS) return 1;
    if (V > 160 * 1024) return R > (nucleus ? 200 : V / 1300);
    if (!nucleus) return V <= 80 * 1024 && R > V / 256;
    return R > V / 200;
}

static int sample(const float* logits, const Rows& rows, bool greedy, bool nucleus, int* out, int R, int V, long long ld, void* stream) {
    int bits = 0;
    while ((1ll << bits) < V) ++bits;
    const float scale = (float)(1ull << (62 - bits < 45 ? 62 - bits : 45));
    const dim3 block(THREADS);
    // The greedy choice alone needs one pass, and clusters take turns of 17 rows or so: a block a row, but for a few long rows (us on
    // clusters and in blocks: 8 rows of 24,000 3.1 and 3.2, of 32,000 3.2 and 3.8, of 128,256 4.1 and 8.1; 18 of 32,000 5.4 and 3.8; 36
    // of 128,256 10.4 and 8.3; 256 of them 71 and 25; 18 of 200,000 14.6 and 11.2).
    if (greedy && (V <= 24 * 1024 || R > (V > 100 * 1024 && V <= 160 * 1024 ? 32 : 16))) {
        bw::launch(argmax_kernel, dim3((unsigned)R), block, 0, (cudaStream_t)stream, logits, out, V, (size_t)ld);
        BW_LAUNCH_CHECK();
        return 0;
    }
    if (bw_sample_row_in_a_block(R, V, nucleus)) {
        const auto kernel = V <= 8 * THREADS ? sample_kernel<8, false, 1> : sample_kernel<0, false, 1>;
        bw::launch(kernel, dim3((unsigned)R), block, 0, (cudaStream_t)stream, logits, rows, out, V, (size_t)ld, scale);
        BW_LAUNCH_CHECK();
        return 0;
    }
    // tokens of a thread: its warp's share of the block's share of the row, in rows of 32
    const int per_block = (V + ROW_BLOCKS - 1) / ROW_BLOCKS;
    const int iters = ((per_block + WARPS - 1) / WARPS + 31) / 32;
    const dim3 grid((unsigned)R * ROW_BLOCKS);
    // more rows than clusters at one block an SM: two blocks an SM, weights in shared memory (nucleus, us, so and in registers: 32 rows of
    // 32,000 17 and 24, of 128,256 29 and 33, 64 of 152,064 62 and 66)
    const int at_once = bw::num_sms() / ROW_BLOCKS;
    const size_t kept = (size_t)iters * 32 * WARPS * sizeof(float);
    if (!greedy && R > at_once && kept <= 80 * 1024) {      // (two blocks and their histograms in an SM's shared memory)
        static bool done[bw::MAX_DEVICES] = {};
        if (const cudaError_t e = bw::allow_dynamic_smem(sample_kernel<0, true>, 80 * 1024, done); e != cudaSuccess) return (int)e;
        bw::launch(sample_kernel<0, true>, grid, block, kept, (cudaStream_t)stream, logits, rows, out, V, (size_t)ld, scale);
        BW_LAUNCH_CHECK();
        return 0;
    }
#define BW_SAMPLE(NV) bw::launch(sample_kernel<NV>, grid, block, 0, (cudaStream_t)stream, logits, rows, out, V, (size_t)ld, scale)
    // registers for 8 tokens a thread (rows up to 65,536) or 20 (up to 163,840: 64 registers a thread allow no more); longer rows are
    // read again for every pass (nucleus, a row of 200,000 in 24 us, 32 rows in 71)
    if (iters <= 8) BW_SAMPLE(8);
    else if (iters <= 20) BW_SAMPLE(20);
    else BW_SAMPLE(0);
#undef BW_SAMPLE
    BW_LAUNCH_CHECK();
    return 0;
}

// temperature, top_p: per row (may be null: greedy / no nucleus); u: per row uniform in [0,1).
BW_EXPORT int bw_sample(const float* logits, const float* temperature, const float* top_p, const float* u,
                        int* out, int R, int V, long long ld, void* stream) {
    if (R <= 0) return 0;
    if (V <= 0 || ld < V) return BW_ERR_BAD_ARG;
    if (temperature && !u) return BW_ERR_BAD_ARG;
    Rows rows{};
    rows.temperature = temperature; rows.top_p = top_p; rows.u = u;
    return sample(logits, rows, !temperature, top_p != nullptr, out, R, V, ld, stream);
}

// The same with the rows' parameters in the caller's memory: they travel with the launch, no copy and no buffer on the device.  All three
// arrays, at most VALUE_ROWS rows.
BW_EXPORT int bw_sample_values(const float* logits, const float* temperature, const float* top_p, const float* u, int* out, int R, int V,
                               long long ld, void* stream) {
    if (R <= 0) return 0;
    if (V <= 0 || ld < V || !temperature || !top_p || !u || R > VALUE_ROWS) return BW_ERR_BAD_ARG;
    Rows rows{};
    rows.by_value = 1;
    bool nucleus = false;
    for (int r = 0; r < R; ++r) {
        rows.v[0][r] = temperature[r]; rows.v[1][r] = top_p[r]; rows.v[2][r] = u[r];
        nucleus |= temperature[r] > 0.f && top_p[r] < 1.f;
    }
    return sample(logits, rows, false, nucleus, out, R, V, ld, stream);
}
