// out[M, N] (=|+=) x[M, K] . w[N, K]^T (+ bias), float32 in and out, on the tensor cores.
//
// Every operand is split into two TF32 numbers, hi = x rounded to 11 bits and lo = x - hi, which is exact and has at most 12 bits, of
// which the tensor cores read 11 (what they drop is at most 2^-23 |x|), and three products are summed, hi hi apart from hi lo + lo hi (lo
// lo is below 2^-22 of the product).  The tensor cores' own sums are kept short: an accumulator takes 64 channels and is then added into float32 registers, rounded to
// nearest, so no long chain runs through the tensor cores' accumulation.  Measured against 64 bits over the products of an 8B
// decoder (K 4096 and 14336): relative error 2.2e-7 to 2.6e-7, where one chain of float32 FMAs (gemm_simt.cu) has 1.2e-6 to 2.2e-6.
// What the split drops of an operand is at most 2^-23 of it, one unit of float32's last place: a product by itself (a row of x with one
// entry) is off by up to 2^-21 where an FMA rounds by 2^-24.  Below 1e-34 an operand's lo is no normal number and keeps multiples of
// 2^-136 only (relative error at 1e-35 6.6e-7, at 1e-36 6.6e-6).  Results that come out as no number are made again by FMAs: see chain().
//
// Weights are the 128-row operand (from tensor memory), tokens the other (from shared memory).  The tokens are split beforehand by a
// small kernel (they are read again by every block of features); the weights, which are read once, on the way: a warp a quarter
// of the rows, a lane a row, from the TMA tile into tensor memory.
// hi hi goes into two accumulators in turn; the small products have one of their own over a whole piece (their sums are 2^-11 of the
// others', and so is what the accumulation drops).
// Three rings: the weights' tiles, which are free again once they are split; the split weights in tensor memory; the tokens' tiles.
// With one ring for all three (a stage held from its load to its MMAs' end) four stages of loads were in flight, and every
// accumulator was drained while nothing ran: 64 tokens took 138 us, 128 tokens 188 us, 301 tokens 508 us at the sizes below.
// A token's result is the same whatever else is in the batch: the channels of all tiles of features, laid end to end, are cut into one
// range per SM, whatever the number of tokens; a range's part of a tile is summed as above, and a tile's parts are added in their
// order by a second kernel.  (So every SM also streams the same number of bytes, and no round of blocks ends half empty.)
// Roles (896 threads): warp 0 loads weights; warp 1 TMEM owner and MMAs; warp 2 loads tokens; warps 4..11 split the weights, two
// groups that take stages in turn; warps 12..27 add the accumulators up, 32 tokens each group of four, and write the result.  Every
// wait is bounded; a timeout sets the status word and all roles fall through to the exit.
// What bounds it: up to 16 tokens the weights' bytes; beyond, shared memory: a stage of 32 channels at 112 tokens moves 103 KB of it (the
// weights' tile in and out 32, the tokens' in 28, what its twelve MMAs read 43), 800 cycles at 128 bytes, of which the MMAs alone need 670.
// Measured, x 28672 x 4096, with the small kernels, on several B200s: 1 to 16 tokens 79 to 84 us (5.6 to 6.0 TB/s), 64 tokens 114, 128
// tokens 149 (202 TFLOP/s), 301 tokens 404 to 415.  gemm_simt.cu: 301 tokens 3.1 ms.
#include "tcgen05.cuh"

using bf16 = __nv_bfloat16;

namespace {

constexpr int BM = 128, BK = 32, MAX_BN = 128;
constexpr int A_BYTES = BM * BK * 4;
constexpr int SUM_STAGES = 2;      // stages of an accumulator before it is added up
constexpr int SPLIT_GROUPS = 2, SUM_GROUPS = 4;     // of four warps each, from warps 4 and 12 on
constexpr int THREADS = 32 * (4 + 4 * SPLIT_GROUPS + 4 * SUM_GROUPS);
constexpr int SMEM_BUDGET = 224 * 1024;
constexpr int MAX_W = 12, MAX_T = 4, MAX_X = 6;     // stages of the rings: weights' tiles, split weights, tokens' tiles

__device__ int g_status = 0;

// Tensor memory: the small products' accumulator, two of hi hi, then the split weights, 64 columns (hi, lo) a stage.
__host__ __device__ constexpr int acc_cols(int bn) { return (bn + 31) / 32 * 32; }
__host__ __device__ constexpr int t_stages(int bn) { return (512 - 3 * acc_cols(bn)) / 64 < MAX_T ? (512 - 3 * acc_cols(bn)) / 64 : MAX_T; }
static_assert(t_stages(MAX_BN) == 2, "two stages of split weights beside the accumulators");
// Shared memory: what the tokens' ring leaves goes to the weights.
__host__ __device__ constexpr int x_bytes(int bn) { return 2 * bn * BK * 4; }
__host__ __device__ constexpr int x_stages(int bn) { return bn > 64 ? 4 : MAX_X; }
__host__ __device__ constexpr int w_stages(int bn) {
    const int n = (SMEM_BUDGET - x_stages(bn) * x_bytes(bn)) / A_BYTES;
    return n < MAX_W ? n : MAX_W;
}
// A warp that waits for a phase by its parity must not be two phases ahead of it.  The split groups take stages in turn, and what holds
// a group back is its own slot among the split weights: behind it at most t_stages stages are unfinished.  So no slot may have two
// groups waiting for it, and a stage of the weights' ring may come round again only after the group that had it before is done.  A
// slot of the tokens' ring is always the same group's.
constexpr bool rings_hold() {
    for (int bn = 16; bn <= MAX_BN; bn += 16)
        if (t_stages(bn) < SPLIT_GROUPS || w_stages(bn) < t_stages(bn) + SPLIT_GROUPS || x_stages(bn) % SPLIT_GROUPS) return false;
    return true;
}
static_assert(rings_hold(), "a split group could pass a wait two phases early");
// More than 64 tokens: the warps that split the weights, which wait most of the time, also wait, in the MMA warp's place, for the stage's
// tokens and for the accumulator that a pair of stages begins: each wait between two stages' products leaves the tensor pipe without
// work (it has about two instructions queued): x 28672 x 4096, 93 tokens 140 us, 129 so; 128 tokens 163 and 152, K 14336, 301 tokens 234
// and 217.  Up to 64 tokens the weights' bytes bound, and the split is on their way (16 tokens 86 us, 89 so).  A wait for an accumulator of
// stage i, the first of a pair p, must find the wait of pair p - 2 over: that pair begins with stage i - 2, the group's own, or with an
// earlier one, done as the group knows from its wait for the slot of stage i, if there are three slots at most.
__host__ __device__ constexpr bool split_waits(int bn) { return bn > 64; }
static_assert(t_stages(80) <= 3 && t_stages(128) <= 3, "with four slots stage i - 3 may be another group's, unfinished");
__host__ __device__ constexpr int ring_bytes(int bn) { return w_stages(bn) * A_BYTES + x_stages(bn) * x_bytes(bn); }

// x rounded to TF32, halves away from zero (three integer instructions fewer than the conversion instruction takes; a NaN whose
// bits overflow here stays one in x - hi)
__device__ __forceinline__ float tf32_hi(float v) { return __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xffffe000u); }
// D[tmem] (+)= A[tmem] * B[smem]^T, TF32 inputs, float32 accumulators; one thread issues
__device__ __forceinline__ void umma_tf32_ts(uint32_t d, uint32_t a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                 "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n}"
                 ::"r"(d), "r"(a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// float32 accumulator, TF32 A and B (format 2), both K-major
__device__ __forceinline__ uint32_t idesc_tf32(int n) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

struct Out {
    float* out; const void* bias; float* part;   // part: [piece][M][BM], see Cut
    const float *x, *w;                           // the operands as they are, for chain()
    long long ldo, ldx;
    int bias_type, accumulate, M, N, K;
};

// The stages (32 channels of a tile of features) of all tiles, dealt out to `ctas` ranges.
struct Cut {
    int kb_total, tiles_n, ctas;
    __host__ __device__ long long total() const { return (long long)tiles_n * kb_total; }
    __host__ __device__ long long begin(int c) const { return c * total() / ctas; }
    __host__ __device__ int owner(long long kb) const { return (int)(((kb + 1) * ctas + total() - 1) / total()) - 1; }
    __host__ __device__ int first_part(int tile) const { return owner((long long)tile * kb_total); }
    __host__ __device__ int parts(int tile) const { return owner((long long)(tile + 1) * kb_total - 1) - first_part(tile) + 1; }
    // The piece that a range has of a tile it shares: a range shares its first tile and its last at most.  (So the scratch is two tiles
    // a range, 78 MB at 512 tokens, whatever the weight's size: of the 1,002 tiles of a head of 128,256 rows 146 are shared.)
    __host__ __device__ int piece(int range, int tile) const { return 2 * range + (begin(range) / kb_total != tile); }
    __host__ bool shared() const {
        for (int c = 1; c < ctas; ++c) if (begin(c) % kb_total) return true;
        return false;
    }
};
// One CTA's items: for every tile of tokens that is its own (a weight of fewer ranges than SMs has them dealt out, blockIdx.y), its
// range's piece of every tile of features.
struct Items {
    Cut cut;
    int tiles_m, mt;
    int lo, hi, at;
    int tile, kb0, n;        // the item: tile of features, first stage, stages (tile of tokens: mt)
    __device__ Items(const Cut& c, int tiles_m_) : cut(c), tiles_m(tiles_m_), mt(blockIdx.y) {
        lo = (int)cut.begin(blockIdx.x); hi = (int)cut.begin(blockIdx.x + 1); at = lo;
    }
    __device__ bool next() {
        if (at >= hi) { at = lo; mt += gridDim.y; }
        if (mt >= tiles_m || lo >= hi) return false;
        tile = at / cut.kb_total;
        kb0 = at - tile * cut.kb_total;
        n = min(cut.kb_total - kb0, hi - at);
        at += n;
        return true;
    }
};

__device__ __forceinline__ float bias_at(const Out& o, int n) {
    if (!o.bias) return 0.f;
    return o.bias_type == BW_F32 ? ((const float*)o.bias)[n] : __bfloat162float(((const bf16*)o.bias)[n]);
}

// One result by float32 FMAs, made by a whole warp (the same in all lanes).  An operand that is not finite, or so near float32's largest
// that hi is not, makes every result it enters a NaN (its lo is one, or the infinity that cancels hi's), and no other operand does unless
// a sum overflows.  So a result that is a NaN, and only that, is made again here, from the operands as they are: infinities stay
// infinities.  x 28672 x 4096, 301 tokens of which so many hold a NaN: none 0.49 ms, one 2.0, 16 3.6, all 28 (gemm_simt.cu 3.1).
__device__ __noinline__ float chain(const float* x, const float* w, int K) {
    float s = 0.f;
#pragma unroll 4
    for (int k = (threadIdx.x & 31) * 4; k < K; k += 128) {
        const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + k);
        s = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
    }
    return bw::warp_sum(s);
}
// chain() for every lane of a converged warp that wants it, for token m and feature n of that lane
__device__ __forceinline__ float chains(const Out& o, bool wanted, float otherwise, int m, int n) {
    for (unsigned lanes = __ballot_sync(0xffffffffu, wanted); lanes; lanes &= lanes - 1) {
        const int from = __ffs(lanes) - 1, mm = __shfl_sync(0xffffffffu, m, from), nn = __shfl_sync(0xffffffffu, n, from);
        const float v = chain(o.x + (size_t)mm * o.ldx, o.w + (size_t)nn * o.K, o.K);
        if ((threadIdx.x & 31) == from) otherwise = v;
    }
    return otherwise;
}

// hi and lo parts of x, [2][M][K]; K % 4 == 0.  A row of the grid a token: no division, and as many bytes on their way as there are
// (301 tokens of 4096 and 14336: 5.1 and 12.1 us with a division for each four channels, 4.4 and 10.2 so)
__global__ void __launch_bounds__(256)
split_kernel(const float* __restrict__ x, float* __restrict__ xs, int M, int K, long long ldx) {
    BW_PDL_TRIGGER();
    BW_PDL_WAIT();
    const int row = blockIdx.x;
    for (int c = (blockIdx.y * 256 + threadIdx.x) * 4; c < K; c += gridDim.y * 1024) {
        const float4 v = *reinterpret_cast<const float4*>(x + row * ldx + c);
        const float in[4] = {v.x, v.y, v.z, v.w};
        float hi[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            hi[j] = tf32_hi(in[j]);
            lo[j] = in[j] - hi[j];
        }
        *reinterpret_cast<float4*>(xs + (size_t)row * K + c) = make_float4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<float4*>(xs + ((size_t)M + row) * K + c) = make_float4(lo[0], lo[1], lo[2], lo[3]);
    }
}

template <bool SPLIT_WAITS>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, Out o, int bn, Cut cut,
                   int tiles_m) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t bars[2 * (MAX_W + MAX_T + MAX_X) + 5];
    __shared__ uint32_t tmem_slot[2];
    BW_PDL_TRIGGER();
    const int ws = w_stages(bn), ts = t_stages(bn), xs = x_stages(bn);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t wfull0 = bw::smem_u32(bars), wfree0 = wfull0 + 8 * MAX_W, ready0 = wfree0 + 8 * MAX_W, tfree0 = ready0 + 8 * MAX_T;
    const uint32_t xfull0 = tfree0 + 8 * MAX_T, xfree0 = xfull0 + 8 * MAX_X;
    const uint32_t sum_full0 = xfree0 + 8 * MAX_X, sum_free0 = sum_full0 + 16, small_free = sum_free0 + 16;
    uint8_t* smem_x = smem + ws * A_BYTES;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ws; ++s) { bw::mbar_init(wfull0 + 8 * s, 1); bw::mbar_init(wfree0 + 8 * s, 4); }
        for (int s = 0; s < ts; ++s) { bw::mbar_init(ready0 + 8 * s, 4); bw::mbar_init(tfree0 + 8 * s, 1); }
        for (int s = 0; s < xs; ++s) { bw::mbar_init(xfull0 + 8 * s, 1); bw::mbar_init(xfree0 + 8 * s, 1); }
        for (int a = 0; a < 2; ++a) { bw::mbar_init(sum_full0 + 8 * a, 1); bw::mbar_init(sum_free0 + 8 * a, 4 * SUM_GROUPS); }
        bw::mbar_init(small_free, 4 * SUM_GROUPS);
        bw::fence_barrier_init();
        bw::tma_prefetch_desc(&tm_w);
        bw::tma_prefetch_desc(&tm_x);
        tmem_slot[1] = (uint32_t)g_status;      // an earlier timeout: later launches do no work
    }
    if (warp == 1) bw::tmem_alloc(bw::smem_u32(tmem_slot), 512);
    bw::tc_fence_before();
    __syncthreads();
    bw::tc_fence_after();
    const uint32_t tmem = tmem_slot[0];
    const bool dead = tmem_slot[1] != 0;
    Items it(cut, tiles_m);

    if (dead) {
        // fall through to the exit
    } else if (warp == 0) {
        if (lane == 0) {       // the weights are nobody's output: no wait for the earlier kernels
            int s = 0, ph = 1;
            bool ok = true;
            while (ok && it.next()) {
                for (int i = 0; i < it.n; ++i) {
                    if (!bw::mbar_wait(wfree0 + 8 * s, ph, &g_status, 1)) { ok = false; break; }
                    bw::mbar_expect_tx(wfull0 + 8 * s, A_BYTES);
                    bw::tma_load_2d(bw::smem_u32(smem + s * A_BYTES), &tm_w, wfull0 + 8 * s, (it.kb0 + i) * BK, it.tile * BM);
                    if (++s == ws) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 2) {
        if (lane == 0) {
            const int bytes = x_bytes(bn);
            int s = 0, ph = 1;
            bool ok = true;
            BW_PDL_WAIT();
            while (ok && it.next()) {
                for (int i = 0; i < it.n; ++i) {
                    if (!bw::mbar_wait(xfree0 + 8 * s, ph, &g_status, 2)) { ok = false; break; }
                    const uint32_t dst = bw::smem_u32(smem_x + s * bytes);
                    bw::mbar_expect_tx(xfull0 + 8 * s, bytes);
                    bw::tma_load_2d(dst, &tm_x, xfull0 + 8 * s, (it.kb0 + i) * BK, it.mt * bn);
                    bw::tma_load_2d(dst + bytes / 2, &tm_x, xfull0 + 8 * s, (it.kb0 + i) * BK, o.M + it.mt * bn);
                    if (++s == xs) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // the whole warp walks the stages and one elected lane issues (see tcgen05.cuh, elect_one; in a branch of one lane an MMA took
        // 100 to 150 cycles to issue, whatever its size; so 9, or what the tensor pipe needs)
        const uint32_t small = __shfl_sync(0xffffffffu, tmem, 0), cols_a = small + 3 * acc_cols(bn);
        const uint32_t idesc = idesc_tf32(bn), smem0 = bw::smem_u32(smem_x), lo_units = (uint32_t)bn * BK * 4 / 16;
        int xst = 0, xph = 0, tst = 0, tph = 0, p = 0, items = 0;
        bool ok = true;
        while (ok && __shfl_sync(0xffffffffu, (int)it.next(), 0)) {
            const int n = __shfl_sync(0xffffffffu, it.n, 0);      // (each lane's own: 301 tokens 476 us, so 454 on the same GPU)
            ok = __all_sync(0xffffffffu, bw::mbar_wait(small_free, (items++ & 1) ^ 1, &g_status, 3));
            for (int i = 0; ok && i < n; ++i) {
                const int buf = p & 1;
                const bool fresh = i % SUM_STAGES == 0, last = i % SUM_STAGES == SUM_STAGES - 1 || i == n - 1;
                if constexpr (SPLIT_WAITS) {     // (the warps that say `ready` have waited for the tokens' tile and the accumulator)
                    ok = bw::mbar_wait(ready0 + 8 * tst, tph, &g_status, 5);
                } else {
                    ok = bw::mbar_wait(xfull0 + 8 * xst, xph, &g_status, 4) && bw::mbar_wait(ready0 + 8 * tst, tph, &g_status, 5);
                    if (fresh) ok = ok && bw::mbar_wait(sum_free0 + 8 * buf, ((p >> 1) & 1) ^ 1, &g_status, 6);
                }
                if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                bw::tc_fence_after();
                const uint32_t d = small + (1 + buf) * acc_cols(bn), hi = cols_a + tst * 64;
                const uint64_t b = bw::umma_smem_desc_sw128(smem0 + xst * x_bytes(bn));
                if (bw::elect_one()) {
                    // 8 channels an MMA: 8 columns of A, 32 bytes (2 units of 16) of B's rows; B's lo rows lie behind its hi rows
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_tf32_ts(d, hi + 8 * k, b + 2 * k, idesc, !fresh || k != 0);
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_tf32_ts(small, hi + 8 * k, b + lo_units + 2 * k, idesc, i != 0 || k != 0);
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_tf32_ts(small, hi + 32 + 8 * k, b + 2 * k, idesc, 1);
                    bw::umma_commit(tfree0 + 8 * tst);
                    bw::umma_commit(xfree0 + 8 * xst);
                    if (last) bw::umma_commit(sum_full0 + 8 * buf);
                }
                __syncwarp();
                if (last) ++p;
                if (++tst == ts) { tst = 0; tph ^= 1; }
                if (++xst == xs) { xst = 0; xph ^= 1; }
            }
        }
    } else if (warp >= 4 && warp < 4 + 4 * SPLIT_GROUPS) {
        const int quarter = warp & 3, row = quarter * 32 + lane;
        const uint32_t tmem_a = tmem + 3 * acc_cols(bn) + ((uint32_t)(quarter * 32) << 16);
        const int group = (warp - 4) / 4;
        const int mine = (tiles_m - (int)blockIdx.y + (int)gridDim.y - 1) / (int)gridDim.y;            // tiles of tokens
        const long long all = (cut.begin(blockIdx.x + 1) - cut.begin(blockIdx.x)) * mine;         // stages of all items
        int s = group, ph = 0, slot = group, tph = 1, xst = group, xph = 0;
        int at = group, before = 0;              // the stage within its item; the pairs of stages in the items before
        if constexpr (SPLIT_WAITS) it.next();
        for (long long i = group; i < all; i += SPLIT_GROUPS) {
            if (!__all_sync(0xffffffffu, bw::mbar_wait(wfull0 + 8 * s, ph, &g_status, 7))) break;
            const uint8_t* src = smem + s * A_BYTES + row * 128;
            uint32_t hi[2][16];
#pragma unroll
            for (int j = 0; j < 8; ++j) {           // 16-byte pieces of the row where the 128-byte swizzle put them
                const uint4 v = *reinterpret_cast<const uint4*>(src + ((j ^ (row & 7)) << 4));
                uint32_t* to = &hi[j >> 2][4 * (j & 3)];
                to[0] = v.x; to[1] = v.y; to[2] = v.z; to[3] = v.w;
            }
            // Before the stage is handed back, every lane's reads must be done: an arrive behind loads that are still queued does not wait
            // for them, and the stage's next tile, written by TMA (the async proxy), may overtake them.  Without the fence 0.4 % of the
            // products of 301 x 6144 x 4096 that follow a norm had a weight's 16 bytes from a later stage in some row.
            bw::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) bw::mbar_arrive(wfree0 + 8 * s);
            if (!__all_sync(0xffffffffu, bw::mbar_wait(tfree0 + 8 * slot, tph, &g_status, 8))) break;
            bw::tc_fence_after();
            const uint32_t dst = tmem_a + slot * 64;
#pragma unroll
            for (int h = 0; h < 2; ++h) {           // 16 channels at a time
                uint32_t lo[16];
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    const float x = __uint_as_float(hi[h][c]), h32 = tf32_hi(x);
                    lo[c] = __float_as_uint(x - h32);
                    hi[h][c] = __float_as_uint(h32);
                }
                bw::tmem_st_32x16(dst + 16 * h, hi[h]);
                bw::tmem_st_32x16(dst + 32 + 16 * h, lo);
            }
            bw::tmem_st_wait();
            if constexpr (SPLIT_WAITS) {
                while (at >= it.n) { at -= it.n; before += (it.n + SUM_STAGES - 1) / SUM_STAGES; if (!it.next()) break; }
                const int p = before + at / SUM_STAGES;
                bool ok = bw::mbar_wait(xfull0 + 8 * xst, xph, &g_status, 4);
                if (at % SUM_STAGES == 0) ok = ok && bw::mbar_wait(sum_free0 + 8 * (p & 1), ((p >> 1) & 1) ^ 1, &g_status, 6);
                if (!__all_sync(0xffffffffu, ok)) break;
                bw::tc_fence_after();
                at += SPLIT_GROUPS;
                xst += SPLIT_GROUPS;
                if (xst >= xs) { xst -= xs; xph ^= 1; }
            }
            bw::tc_fence_before();
            __syncwarp();
            if (lane == 0) bw::mbar_arrive(ready0 + 8 * slot);
            s += SPLIT_GROUPS;
            if (s >= ws) { s -= ws; ph ^= 1; }
            slot += SPLIT_GROUPS;
            if (slot >= ts) { slot -= ts; tph ^= 1; }
        }
    } else if (warp >= 4 + 4 * SPLIT_GROUPS) {
        constexpr int COLS = MAX_BN / SUM_GROUPS;
        const int quarter = warp & 3, first = ((warp - 4 - 4 * SPLIT_GROUPS) / 4) * COLS, cols = min(bn - first, COLS);
        const uint32_t mine = tmem + first + ((uint32_t)(quarter * 32) << 16);
        bool ok = true, waited = false;
        int p = 0;
        while (ok && it.next()) {
            float sum[COLS];
#pragma unroll
            for (int c = 0; c < COLS; ++c) sum[c] = 0.f;
            auto add_up = [&](uint32_t from) {
#pragma unroll
                for (int c0 = 0; c0 < COLS; c0 += 16) {
                    if (c0 >= cols) continue;
                    uint32_t v[16];
                    bw::tmem_ld_32x16(from + c0, v);
                    bw::tmem_ld_wait();
#pragma unroll
                    for (int c = 0; c < 16; ++c) sum[c0 + c] += __uint_as_float(v[c]);
                }
                bw::tc_fence_before();
                __syncwarp();
            };
            for (int i = 0; i < it.n; i += SUM_STAGES, ++p) {
                const int buf = p & 1;
                ok = __all_sync(0xffffffffu, bw::mbar_wait(sum_full0 + 8 * buf, (p >> 1) & 1, &g_status, 9));
                if (!ok) break;
                bw::tc_fence_after();
                add_up(mine + (1 + buf) * acc_cols(bn));
                if (lane == 0) bw::mbar_arrive(sum_free0 + 8 * buf);
            }
            if (!ok) break;
            add_up(mine);              // the small products: complete with the piece's last stage
            if (lane == 0) bw::mbar_arrive(small_free);
            if (!waited) { BW_PDL_WAIT(); waited = true; }      // the result belongs to earlier kernels until here
            const int n = it.tile * BM + quarter * 32 + lane, t0 = it.mt * bn + first;
            const bool in = n < o.N;
            const bool whole = it.n == cut.kb_total;
            const long long ld = whole ? o.ldo : BM;
            const float b = whole && in ? bias_at(o, n) : 0.f;
            const bool add = whole && o.accumulate;
            float* dst = whole ? o.out + (size_t)t0 * ld + n
                               : o.part + ((size_t)cut.piece(blockIdx.x, it.tile) * o.M + t0) * BM + quarter * 32 + lane;
            unsigned again = 0;          // the tokens whose results chain() makes
#pragma unroll
            for (int c0 = 0; c0 < COLS; c0 += 16) {       // sixteen tokens' old values in flight
                if (c0 >= cols) continue;
                float old[16];
#pragma unroll
                for (int c = 0; c < 16; ++c) old[c] = add && in && t0 + c0 + c < o.M ? dst[(size_t)(c0 + c) * ld] : 0.f;
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    if (!in || t0 + c0 + c >= o.M) continue;
                    if (whole && sum[c0 + c] != sum[c0 + c]) again |= 1u << (c0 + c);
                    else dst[(size_t)(c0 + c) * ld] = add ? sum[c0 + c] + b + old[c] : sum[c0 + c] + b;
                }
                asm volatile("" ::: "memory");
            }
            __syncwarp();
            for (unsigned any = __reduce_or_sync(0xffffffffu, again); any; any &= any - 1) {
                const int c = __ffs(any) - 1;
                const bool wanted = again >> c & 1;
                const float v = chains(o, wanted, 0.f, t0 + c, n) + b;
                if (wanted) dst[(size_t)c * ld] = add ? v + dst[(size_t)c * ld] : v;
            }
        }
    }
    bw::tc_fence_before();
    __syncthreads();
    bw::tc_fence_after();
    if (warp == 1) bw::tmem_dealloc(tmem, 512);
}

// The parts of the tiles that several ranges share, in their order; V features of SUM_TOKENS tokens a thread.  Where the parts lie takes
// some 64-bit divisions, made before the wait for the products and once for the tokens (the whole product, x 6144 x 4096, with a token a
// thread and so: 301 tokens 106 and 101 us, 1 token 29.6 and 27.9).  V 4: rows of the result begin on 16 bytes.
constexpr int SUM_TOKENS = 4;
template <int V>
__global__ void __launch_bounds__(256)
sum_kernel(Out o, Cut cut) {
    BW_PDL_TRIGGER();
    const int n = (blockIdx.x * blockDim.x + threadIdx.x) * V, m0 = blockIdx.y * SUM_TOKENS, tokens = min(SUM_TOKENS, o.M - m0);
    const bool in = n < o.N;
    const int tile = min(n, o.N - 1) / BM, parts = cut.parts(tile), first = cut.first_part(tile);
    // The loads of the first parts are in flight together, those of the rest two by two (one part after another, a weight of 4096 features,
    // five or six parts a tile, waited for L2 as often: the whole product with K 4096, 4 and 64 tokens 25.5 and 31.0 us, 23.6 and 29.1 so).
    constexpr int KNOWN = 6;
    size_t at[KNOWN];                // of the first parts; a weight of few features and many channels has more
#pragma unroll
    for (int i = 0; i < KNOWN; ++i) at[i] = i < parts ? (size_t)cut.piece(first + i, tile) * o.M * BM : 0;
    float bias[V];
#pragma unroll
    for (int e = 0; e < V; ++e) bias[e] = in ? bias_at(o, n + e) : 0.f;
    BW_PDL_WAIT();
    if (parts == 1) return;          // (a warp's features lie in one tile)
    const float* p = o.part + (size_t)m0 * BM + (n - tile * BM);
    float* dst = o.out + m0 * o.ldo + n;
    auto load = [&](const float* from, bool there, float (&v)[V]) {
        if constexpr (V == 4) {
            const float4 t = there ? *reinterpret_cast<const float4*>(from) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
        } else v[0] = there ? *from : 0.f;
    };
    float s[SUM_TOKENS][V], old[SUM_TOKENS][V], v[KNOWN - 1][SUM_TOKENS][V];
#pragma unroll
    for (int t = 0; t < SUM_TOKENS; ++t) {
        load(dst + t * o.ldo, o.accumulate && in && t < tokens, old[t]);
        load(p + at[0] + t * BM, in && t < tokens, s[t]);
    }
#pragma unroll
    for (int i = 1; i < KNOWN; ++i)
#pragma unroll
        for (int t = 0; t < SUM_TOKENS; ++t) load(p + at[i] + t * BM, in && t < tokens && i < parts, v[i - 1][t]);
    auto add = [&](const float (&w)[SUM_TOKENS][V]) {
#pragma unroll
        for (int t = 0; t < SUM_TOKENS; ++t)
#pragma unroll
            for (int e = 0; e < V; ++e) s[t][e] += w[t][e];
    };
#pragma unroll
    for (int i = 1; i < KNOWN; ++i) if (i < parts) add(v[i - 1]);
    for (int i = KNOWN; i < parts; i += 2) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const size_t from = i + j < parts ? (size_t)cut.piece(first + i + j, tile) * o.M * BM : 0;
#pragma unroll
            for (int t = 0; t < SUM_TOKENS; ++t) load(p + from + t * BM, in && t < tokens && i + j < parts, v[j][t]);
        }
        add(v[0]);
        if (i + 1 < parts) add(v[1]);
    }
    unsigned again = 0;              // the results that chain() makes
#pragma unroll
    for (int t = 0; t < SUM_TOKENS; ++t) {
        if (!in || t >= tokens) continue;
        unsigned nan = 0;
#pragma unroll
        for (int e = 0; e < V; ++e) {
            nan |= s[t][e] != s[t][e] ? 1u << e : 0u;
            s[t][e] += bias[e];
            if (o.accumulate) s[t][e] += old[t][e];
        }
        again |= nan << (t * V);
        if (V == 4 && !nan) *reinterpret_cast<float4*>(dst + t * o.ldo) = make_float4(s[t][0], s[t][1 % V], s[t][2 % V], s[t][3 % V]);
        else {
#pragma unroll
            for (int e = 0; e < V; ++e) if (!(nan >> e & 1)) dst[t * o.ldo + e] = s[t][e];
        }
    }
    for (unsigned any = __reduce_or_sync(0xffffffffu, again); any; any &= any - 1) {
        const int k = __ffs(any) - 1, t = k / V, e = k % V;
        const bool wanted = again >> k & 1;
        const float v = chains(o, wanted, 0.f, m0 + t, n + e) + (wanted ? bias_at(o, n + e) : 0.f);
        if (wanted) dst[t * o.ldo + e] = o.accumulate ? v + dst[t * o.ldo + e] : v;
    }
}

bool encode(CUtensorMap* m, const void* base, long long rows, long long cols, int box_rows) {
    typedef CUresult (*Fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                           const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static Fn fn = nullptr;
    if (!fn) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            return false;
        fn = (Fn)ptr;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)cols * 4};
    const cuuint32_t box[2] = {BK, (cuuint32_t)box_rows}, estr[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

static Cut cut_of(int N, int K) {
    Cut c = {(K + BK - 1) / BK, (N + BM - 1) / BM, 1};
    const long long most = c.total() / 8;        // eight stages or more each: less would be all filling and draining
    c.ctas = most < 1 ? 1 : most < bw::num_sms() ? (int)most : bw::num_sms();
    return c;
}

// The floats of scratch that bw_gemm_f32_tc needs per token for the tiles that several ranges share (0: there are none).
BW_EXPORT int bw_gemm_f32_tc_part_floats(int N, int K) {
    if (N <= 0 || K <= 0) return BW_ERR_BAD_ARG;
    const Cut c = cut_of(N, K);
    return c.shared() ? 2 * c.ctas * BM : 0;
}

// xs: float32 [2 * M * K] for the tokens' parts; part: `part_floats` of scratch, M times bw_gemm_f32_tc_part_floats at least.
// K % 4 == 0, rows of x and w begin on 16 bytes; at most 65,535 tokens.
BW_EXPORT int bw_gemm_f32_tc(const float* x, const float* w, const void* bias, int bias_type, float* out, int M, int N, int K, long long ldx,
                             long long ldo, int accumulate, float* xs, float* part, long long part_floats, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4 || ldx % 4 || ldx < K || ldo < N || M > 65535 || cut_of(N, K).total() > 0x7fffffff || (((uintptr_t)x | (uintptr_t)w | (uintptr_t)xs) & 15)) return BW_ERR_BAD_ARG;
    const Cut cut = cut_of(N, K);
    const bool shared = cut.shared();
    if (shared && (!part || ((uintptr_t)part & 15) || part_floats < 2ll * cut.ctas * BM * M)) return BW_ERR_BAD_ARG;
    // tiles of tokens as even as they can be, a multiple of 16
    const int tiles = (M + MAX_BN - 1) / MAX_BN, bn = ((M + tiles - 1) / tiles + 15) / 16 * 16, tiles_m = (M + bn - 1) / bn;
    cudaStream_t s = (cudaStream_t)stream;
    CUtensorMap tm_w, tm_x;
    if (!encode(&tm_w, w, N, K, BM) || !encode(&tm_x, xs, 2ll * M, K, bn)) return BW_ERR_DRIVER;
    bw::launch(split_kernel, dim3(M, K < 65536 ? (K + 1023) / 1024 : 64), dim3(256), 0, s, x, xs, M, K, ldx);
    BW_LAUNCH_CHECK();
    static bool done[2][bw::MAX_DEVICES] = {};
    const auto kernel = split_waits(bn) ? gemm_f32_tc_kernel<true> : gemm_f32_tc_kernel<false>;
    const cudaError_t e = bw::allow_dynamic_smem(kernel, SMEM_BUDGET + 1024, done[split_waits(bn)]);
    if (e != cudaSuccess) return (int)e;
    const Out o = {out, bias, part, x, w, ldo, ldx, bias_type, accumulate, M, N, K};
    // a small weight's ranges leave SMs idle: they take tiles of tokens (300 tokens x 1024 x 256: 23.6 us without, 11.2
    // so, 17.4 in gemm_simt.cu; 1,000 tokens: 62.6 with launches of 512, 12.1 so, 27.0)
    const int rows = bw::num_sms() / cut.ctas < tiles_m ? bw::num_sms() / cut.ctas : tiles_m;
    bw::launch(kernel, dim3(cut.ctas, rows < 1 ? 1 : rows), dim3(THREADS), (size_t)ring_bytes(bn) + 1024, s, tm_w, tm_x, o, bn, cut,
               tiles_m);
    BW_LAUNCH_CHECK();
    if (shared) {
        const int groups = (M + SUM_TOKENS - 1) / SUM_TOKENS;
        if (N % 4 == 0 && ldo % 4 == 0 && ((uintptr_t)out & 15) == 0) bw::launch(sum_kernel<4>, dim3((N / 4 + 255) / 256, groups), dim3(256), 0, s, o, cut);
        else bw::launch(sum_kernel<1>, dim3((N + 255) / 256, groups), dim3(256), 0, s, o, cut);
        BW_LAUNCH_CHECK();
    }
    return 0;
}

// 0 if no bounded wait ever gave up (synchronises the device)
BW_EXPORT int bw_gemm_f32_tc_status() {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_status, sizeof(int)) != cudaSuccess) return -1;
    return v;
}
