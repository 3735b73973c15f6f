// Paged causal grouped-query attention in float32, tiled: the 32-bit path's attention where scores need nothing but a scale
// and a causal, windowed or block mask (attention_simt.cu takes every other option).  All arithmetic is float32 FMAs on the
// CUDA cores, as there; a key and a value are read once for all query heads of their group and for all tokens of a tile.
//
// A block of eight warps takes a tile of ROWS stacked query rows (token-major, then the heads of the group) of one request and
// kv head and walks its keys (cp.async).  ROWS = 64 for prompt portions: 64 keys at a time (32 for heads above 128) in two stages, each
// thread scores 4 rows times 4 keys (2 times 4), a warp owns eight neighbouring rows.  ROWS = 16 for the few rows of a decoding request: 32 keys at
// a time in three stages, a warp owns a row or two, which share the key that a lane scores.  In the softmax, 32 keys at a time, and the
// values a lane has four channels (twice that for heads above 128), so probabilities pass through shared memory inside the warp only.  The
// keys of a tile are one block's, or dealt out by slices to several, whose results a second kernel adds up.
// A row's result is the same bits whatever else is in the batch: both forms make a softmax per slice of keys, counted from position 0,
// in the same order of operations, and fold the slices in their order (fold()).  A slice has SLICE keys, or as many times SLICE that a
// row sees MOST slices or hardly more: what a row sees decides, and no batch.  (So a decoding request has at most MOST + 2 blocks and
// partial results per kv head at any context: 64 requests of 8 kv heads and groups of 4 at 131,072 tokens 69 MB.)
// What bounds it: decode, the bytes of keys and values; prompts, shared-memory reads (eight 16-byte reads per 64 FMAs, for
// heads above 128 six per 32); few keys, latency.
// Measured at head size 128, groups of 4, 8 kv heads, against attention_simt.cu (a block per token and head, a lane a key): 4 requests
// at 1,000 keys 18 us with the merge against 167, 4 portions of 200 tokens 109 against 1,402, 64 requests at 300 keys, groups of 1, 8 kv
// heads of 64, 54 against 66.
#include <type_traits>
#include "common.cuh"

namespace {

constexpr int THREADS = 256, WARPS = 8, KEYS = 32, SLICE_ROWS = 16, SLICE = 128, MOST = 64;

struct Params {
    const float *q, *k_pages, *v_pages;
    float* out;
    const int *cu_q, *q_start, *block_table;
    int max_blocks, nh, nkv, hd, page_size, num_pages, window, chunk;
    float scale;
    float *part_o, *part_ml;      // [row of a tile and slice][hd] and [..][2] (maximum, sum), see part_row()
};

__device__ __forceinline__ void copy16(float* dst, const float* src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// Tiles of keys in flight or at work: prompts work on a tile for longer than the next one takes to come; a decoding request's few rows do not.
__host__ __device__ constexpr int stages(int rows) { return rows == 64 ? 2 : 3; }
// Keys that a block fetches and scores at once (the softmax takes KEYS of them at a time).  Of a prompt's 64 rows a thread scores 4 x 4 with
// 64 keys, eight 16-byte reads of shared memory per 64 FMAs; with 32 keys 2 x 4, six reads per 32, which the reads bound.  One such block an
// SM, slices dealt out or not (two of 128 registers with 32 keys each took 56 us for a slice of 128 keys, one of this kind 30).
__host__ __device__ constexpr int fetched(int rows, int ch) { return rows == 64 && ch == 1 ? 64 : KEYS; }
__host__ __device__ constexpr int smem_floats(int rows, int hd, int kt) {
    return rows * (hd + 4) + stages(rows) * (kt * (hd + 4) + kt * hd + kt) + rows * (kt + 4);
}

// One more slice (maximum m, sum l) of a row: the factors of what was there (M, L) and of the slice; M and L are updated.  A slice in
// which the row sees no key changes nothing.
__device__ __forceinline__ float2 fold(float& M, float& L, float m, float l) {
    if (m == -INFINITY) return make_float2(1.f, 0.f);
    const float to = fmaxf(M, m), a = M == -INFINITY ? 0.f : expf(M - to), b = expf(m - to);
    L = fmaf(L, a, __fmul_rn(l, b));
    M = to;
    return make_float2(a, b);
}
__device__ __forceinline__ float folded(float O, float o, float2 f) { return fmaf(O, f.x, __fmul_rn(o, f.y)); }
// The keys of a slice for the row at a position, and the slices from a key on.
__device__ __forceinline__ int slice_keys(const Params& p, int pos) {
    const int sees = pos + 1 - bw::first_visible(pos, p.window, p.chunk);
    return SLICE * ((sees + SLICE * MOST - 1) / (SLICE * MOST));
}
__device__ __forceinline__ int slices_from(const Params& p, int pos, int keys) { return bw::first_visible(pos, p.window, p.chunk) / keys * keys; }
__device__ __forceinline__ int slices_of(int base, int end, int keys) { return (end - base + keys - 1) / keys; }

// Where a tile of `rows` stacked rows leaves a slice's results: `where` rows per kv head lie before its own.
__device__ __forceinline__ size_t part_row(const Params& p, int where, int slice, int rows, int kvh) {
    return (size_t)(where + slice * rows) * p.nkv + (size_t)kvh * rows;
}

// Work items (request, first token); SLICES: (request, first token, block | blocks << 16, where), a block of the `blocks` that share
// the tile's slices, whose rows have slices of one size.  Of a single slice the block writes the tile's result (its fold is it).
// CH: groups of four channels of a lane.
template <int ROWS, int CH, bool SLICES>
__global__ void __launch_bounds__(THREADS, ROWS == 64 ? 1 : 2)
attention_f32_kernel(Params p, const int4* __restrict__ work) {
    BW_PDL_TRIGGER();
    extern __shared__ float4 smem4[];
    const int hd = p.hd, ldk = hd + 4, G = p.nh / p.nkv;
    float* qs = reinterpret_cast<float*>(smem4);          // [ROWS][ldk]
    constexpr int STAGES = stages(ROWS), KT = fetched(ROWS, CH), PARTS = KT / KEYS, LDP = KT + 4;
    float* ks = qs + ROWS * ldk;                          // [STAGES][KT][ldk]
    float* vs = ks + STAGES * KT * ldk;                   // [STAGES][KT][hd]
    float* ps = vs + STAGES * KT * hd;                    // [ROWS][LDP]
    int* known = reinterpret_cast<int*>(ps + ROWS * LDP); // [STAGES][KT]: the key has a page
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, kvh = blockIdx.y;
    const int4 item = work[blockIdx.x];
    const int r = item.x;
    const int row0 = p.cu_q[r], q_len = p.cu_q[r + 1] - row0;
    const int t0 = item.y;
    const int tokens = min(ROWS / G, q_len - t0), rows = tokens * G;
    const int pos0 = p.q_start[r] + t0, end = pos0 + tokens;
    const int* bt = p.block_table + (size_t)r * p.max_blocks;
    const int keys = slice_keys(p, pos0), per = keys / KEYS;      // of the first row's slices: keys, tiles
    const int base = slices_from(p, pos0, SLICES ? keys : SLICE);
    const int all = (end - base + KEYS - 1) / KEYS;
    int first = 0, last = all;
    bool whole = !SLICES;                                 // this block makes the tile's result
    if constexpr (SLICES) {
        const int block = item.z & 0xffff, blocks = item.z >> 16, slices = slices_of(base, end, keys), share = (slices + blocks - 1) / blocks;
        whole = slices == 1;
        first = block * share * per;
        last = min(first + share * per, all);
        if (first >= last) return;                        // (the list is as long as the longest context may get)
    }
    // a portion's rows may differ in the size of their slices (it never shrinks, except where a block of positions begins)
    const bool same = !SLICES && slice_keys(p, end - 1) == keys && (p.chunk <= 0 || p.chunk <= SLICE * MOST);
    // Page and place in it of the warp's keys that are fetched next, looked up before: a lane a key (all lanes for every key were half of
    // a decoding block's instructions)
    constexpr int MINE = KT / WARPS;
    int my_page = -1, my_slot = 0;
    auto look_up = [&](int tile) {
        const int kp = base + tile * KEYS + warp * MINE + lane, block = kp / p.page_size;
        my_slot = kp - block * p.page_size;
        my_page = lane < MINE && tile < last && kp < end ? bt[block] : -1;
    };
    look_up(first);      // (block tables are on the device before the step's first kernel, as the work lists are)
    BW_PDL_WAIT();

    for (int i = warp; i < ROWS; i += WARPS) {      // with the first tile of keys; rows beyond the tile's are zeros
        const float* src = p.q + (i < rows ? ((size_t)(row0 + t0 + i / G) * p.nh + (size_t)kvh * G + i % G) * hd : 0);
        for (int c = lane * 4; c < hd; c += 128) copy16(qs + i * ldk + c, src + c, i < rows);
    }
    auto fetch = [&](int tile, int st) {            // the KT keys from this tile on: a warp brings some and their values
        const bool mine = my_page >= 0 && my_page < p.num_pages;
        const long long mine_at = mine ? (((long long)my_page * p.nkv + kvh) * p.page_size + my_slot) * hd : -1;
#pragma unroll
        for (int j = 0; j < MINE; ++j) {
            const int key = warp * MINE + j;
            const long long there = __shfl_sync(0xffffffffu, mine_at, j);
            const bool ok = there >= 0;
            const size_t at = ok ? there : 0;
            for (int c = lane * 4; c < hd; c += 128) {
                copy16(ks + (st * KT + key) * ldk + c, p.k_pages + at + c, ok);
                copy16(vs + (st * KT + key) * hd + c, p.v_pages + at + c, ok);
            }
        }
        if (lane < MINE) known[st * KT + warp * MINE + lane] = mine;
        asm volatile("cp.async.commit_group;" ::: "memory");
        look_up(tile + PARTS);
    };
    // Rows that a warp takes through the softmax and the values: side by side in a tile of 64; of few rows one each for as many warps
    // as there are (with their neighbours, and all warps through the products of empty rows, two stages and a page looked up where it was
    // needed: 4 requests at 1,000 keys, groups of 4, 8 kv heads of 128, 30.4 us with the merge, 20.3 so; 16 at 1,500 155 and 105; 64 at
    // 20 17.3 and 11.6; with a key's look-up by one lane and no empty rows 18.0, 81 and 9.9)
    auto row_of = [&](int i) { return ROWS == 64 ? warp * (ROWS / WARPS) + i : warp + i * WARPS; };

    constexpr int RW = ROWS / WARPS;                // rows of a warp
    float o[RW][CH * 4], m[RW], l[RW];
#pragma unroll
    for (int i = 0; i < RW; ++i) {
        m[i] = -INFINITY; l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < CH * 4; ++c) o[i][c] = 0.f;
    }
    constexpr int FOLDED = SLICES ? 1 : RW;         // rows of a portion fold their slices here
    float O[FOLDED][CH * 4], M[FOLDED], L[FOLDED];
#pragma unroll
    for (int i = 0; i < FOLDED; ++i) {
        M[i] = -INFINITY; L[i] = 0.f;
#pragma unroll
        for (int c = 0; c < CH * 4; ++c) O[i][c] = 0.f;
    }
    constexpr int TX = KT / 4, RPT = KT / 16, KPT = 4, TY = THREADS / TX;      // (64 rows)
    const int tx = tid % TX, ty = tid / TX;
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i)
        if (first + i * PARTS < last) fetch(first + i * PARTS, i);
    for (int from = first, st = 0; from < last; from += PARTS, st = st + 1 == STAGES ? 0 : st + 1) {
        const int next = from + (STAGES - 1) * PARTS;
        if (next < last) fetch(next, st == 0 ? STAGES - 1 : st - 1);
        // these keys have come, however many of those behind them have not
        if (next < last) asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
        else if (STAGES > 2 && from + PARTS < last) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const float* kt = ks + st * KT * ldk;
        if constexpr (ROWS == 16) {
            // a warp a row or two, a lane a key
            static_assert(ROWS == 2 * WARPS || ROWS == 64, "two rows a warp at most");
            auto score = [&](auto both) {
                const float *q0 = qs + warp * ldk, *q1 = qs + (warp + WARPS) * ldk, *key = kt + lane * ldk;
                float s0 = 0.f, s1 = 0.f;
#pragma unroll 8
                for (int c = 0; c < hd; c += 4) {
                    const float4 a = *reinterpret_cast<const float4*>(q0 + c), b = *reinterpret_cast<const float4*>(key + c);
                    s0 = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s0))));
                    if constexpr (decltype(both)::value) {
                        const float4 d = *reinterpret_cast<const float4*>(q1 + c);
                        s1 = fmaf(d.w, b.w, fmaf(d.z, b.z, fmaf(d.y, b.y, fmaf(d.x, b.x, s1))));
                    }
                }
                auto put = [&](int row, float s) {
                    const int q_pos = pos0 + row / G, kp = base + from * KEYS + lane;
                    const bool seen = kp <= q_pos && kp >= bw::first_visible(q_pos, p.window, p.chunk) && known[st * KT + lane];
                    ps[row * LDP + lane] = seen ? s * p.scale : -INFINITY;
                };
                put(warp, s0);
                if constexpr (decltype(both)::value) put(warp + WARPS, s1);
            };
            if (warp + WARPS < rows) score(std::true_type{});
            else if (warp < rows) score(std::false_type{});
            __syncwarp();
        } else {
            float s[RPT][KPT];
#pragma unroll
            for (int i = 0; i < RPT; ++i)
#pragma unroll
                for (int j = 0; j < KPT; ++j) s[i][j] = 0.f;
            for (int c = 0; c < hd; c += 4) {
                float4 a[RPT], b[KPT];
#pragma unroll
                for (int i = 0; i < RPT; ++i) a[i] = *reinterpret_cast<const float4*>(qs + (ty + i * TY) * ldk + c);
#pragma unroll
                for (int j = 0; j < KPT; ++j) b[j] = *reinterpret_cast<const float4*>(kt + (tx + j * TX) * ldk + c);
#pragma unroll
                for (int i = 0; i < RPT; ++i)
#pragma unroll
                    for (int j = 0; j < KPT; ++j)
                        s[i][j] = fmaf(a[i].w, b[j].w, fmaf(a[i].z, b[j].z, fmaf(a[i].y, b[j].y, fmaf(a[i].x, b[j].x, s[i][j]))));
            }
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const int row = ty + i * TY, q_pos = pos0 + row / G;
                const int lo = bw::first_visible(q_pos, p.window, p.chunk);
#pragma unroll
                for (int j = 0; j < KPT; ++j) {
                    const int key = tx + j * TX, kp = base + from * KEYS + key;
                    const bool seen = row < rows && kp <= q_pos && kp >= lo && known[st * KT + key];
                    ps[row * LDP + key] = seen ? s[i][j] * p.scale : -INFINITY;
                }
            }
            __syncthreads();
        }
#pragma unroll 1
        for (int part = 0; part < PARTS; ++part) {
            const int tile = from + part;
            if (tile >= last) break;
            float* pt = ps + part * KEYS;
            auto softmax_and_values = [&](auto taken) {
                constexpr int N = decltype(taken)::value;     // of the warp's rows
                // (a warp's rows side by side: one after another their shuffles and exponentials are the kernel's latency at few keys)
                float sc[N], m_new[N], e[N], sum[N];
                bool zero = false;
#pragma unroll
                for (int i = 0; i < N; ++i) sc[i] = ROWS == 64 || row_of(i) < rows ? pt[row_of(i) * LDP + lane] : -INFINITY;
#pragma unroll
                for (int i = 0; i < N; ++i) m_new[i] = fmaxf(m[i], bw::warp_max(sc[i]));
#pragma unroll
                for (int i = 0; i < N; ++i) e[i] = sc[i] == -INFINITY ? 0.f : expf(sc[i] - m_new[i]);
#pragma unroll
                for (int i = 0; i < N; ++i) sum[i] = bw::warp_sum(e[i]);
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    const float corr = m[i] == -INFINITY ? 0.f : expf(m[i] - m_new[i]);
                    l[i] = l[i] * corr + sum[i];
                    m[i] = m_new[i];
                    pt[row_of(i) * LDP + lane] = e[i];
                    zero |= e[i] == 0.f && row_of(i) < rows;
#pragma unroll
                    for (int c = 0; c < CH * 4; ++c) o[i][c] *= corr;
                }
                __syncwarp();
                // A key without weight (masked, or too far below the largest score) must not add its value, which may be no number: 0 times an
                // infinity is none.  Rare beside the diagonal and a window's edges, so a warp asks once per tile.
                const float* vt = vs + (st * KT + part * KEYS) * hd;
                auto add_values = [&](auto skip) {
#pragma unroll 2
                    for (int k4 = 0; k4 < KEYS; k4 += 4) {
                        float4 w[N];
#pragma unroll
                        for (int i = 0; i < N; ++i) w[i] = *reinterpret_cast<const float4*>(pt + row_of(i) * LDP + k4);
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                            for (int h = 0; h < CH; ++h) {
                                const int c = lane * 4 + 128 * h;
                                if (c >= hd) continue;
                                const float4 v = *reinterpret_cast<const float4*>(vt + (k4 + kk) * hd + c);
#pragma unroll
                                for (int i = 0; i < N; ++i) {
                                    const float e = kk == 0 ? w[i].x : kk == 1 ? w[i].y : kk == 2 ? w[i].z : w[i].w;
                                    if (decltype(skip)::value && e == 0.f) continue;
                                    o[i][4 * h] = fmaf(e, v.x, o[i][4 * h]);
                                    o[i][4 * h + 1] = fmaf(e, v.y, o[i][4 * h + 1]);
                                    o[i][4 * h + 2] = fmaf(e, v.z, o[i][4 * h + 2]);
                                    o[i][4 * h + 3] = fmaf(e, v.w, o[i][4 * h + 3]);
                                }
                            }
                    }
                };
                if (__any_sync(0xffffffffu, zero)) add_values(std::true_type{});
                else add_values(std::false_type{});
            };
            if constexpr (ROWS == 64) softmax_and_values(std::integral_constant<int, RW>{});
            else if (warp + WARPS < rows) softmax_and_values(std::integral_constant<int, 2>{});
            else if (warp < rows) softmax_and_values(std::integral_constant<int, 1>{});
            if constexpr (SLICES) {
                if (!whole && ((tile + 1) % per == 0 || tile + 1 == last)) {
                    const size_t at = part_row(p, item.w, tile / per, rows, kvh);
#pragma unroll
                    for (int i = 0; i < RW; ++i) {
                        const int row = row_of(i);
                        if (row >= rows) continue;
                        if (lane == 0) *reinterpret_cast<float2*>(p.part_ml + 2 * (at + row)) = make_float2(m[i], l[i]);
#pragma unroll
                        for (int h = 0; h < CH; ++h) {
                            const int c = lane * 4 + 128 * h;
                            if (c < hd) *reinterpret_cast<float4*>(p.part_o + (at + row) * hd + c) = make_float4(o[i][4 * h], o[i][4 * h + 1], o[i][4 * h + 2], o[i][4 * h + 3]);
                        }
#pragma unroll
                        for (int c = 0; c < CH * 4; ++c) o[i][c] = 0.f;
                        m[i] = -INFINITY; l[i] = 0.f;
                    }
                }
            } else {
                const int done = base / KEYS + tile + 1;      // tiles from position 0
                if (same ? done % per == 0 || tile + 1 == last : done % (SLICE / KEYS) == 0 || tile + 1 == last) {
#pragma unroll
                    for (int i = 0; i < RW; ++i) {
                        if (!same && tile + 1 < last && done % (slice_keys(p, pos0 + row_of(i) / G) / KEYS)) continue;
                        const float2 f = fold(M[i], L[i], m[i], l[i]);
#pragma unroll
                        for (int c = 0; c < CH * 4; ++c) { O[i][c] = folded(O[i][c], o[i][c], f); o[i][c] = 0.f; }
                        m[i] = -INFINITY; l[i] = 0.f;
                    }
                }
            }
        }
        __syncthreads();        // (the next fetch overwrites this stage, the next scores the probabilities)
    }
    if (!whole) return;
#pragma unroll
    for (int i = 0; i < RW; ++i) {
        const int row = row_of(i);
        if (row >= rows) continue;
        const float sum = SLICES ? l[i] : L[i], f = sum > 0.f ? 1.f / sum : 0.f;
        float* dst = p.out + ((size_t)(row0 + t0 + row / G) * p.nh + (size_t)kvh * G + row % G) * hd;
        float res[CH * 4];
#pragma unroll
        for (int c = 0; c < CH * 4; ++c) {
            if constexpr (SLICES) res[c] = o[i][c] * f;
            else res[c] = O[i][c] * f;
        }
#pragma unroll
        for (int h = 0; h < CH; ++h) {
            const int c = lane * 4 + 128 * h;
            if (c < hd) *reinterpret_cast<float4*>(dst + c) = make_float4(res[4 * h], res[4 * h + 1], res[4 * h + 2], res[4 * h + 3]);
        }
    }
}

// Slices of one (tile, kv head, row) of several, in slice order; a thread four channels.  Items (request, first token, rows, where).
__global__ void __launch_bounds__(64)
attention_f32_merge_kernel(Params p, const int4* __restrict__ work) {
    BW_PDL_TRIGGER();
    const int4 item = work[blockIdx.x];
    const int r = item.x, t0 = item.y, kvh = blockIdx.y, row = blockIdx.z, G = p.nh / p.nkv, hd = p.hd, c = threadIdx.x * 4;
    const int row0 = p.cu_q[r] + t0, tokens = min(item.z / G, p.cu_q[r + 1] - row0), rows = tokens * G, pos0 = p.q_start[r] + t0;
    if (row >= rows || c >= hd) return;
    const int keys = slice_keys(p, pos0), slices = slices_of(slices_from(p, pos0, keys), pos0 + tokens, keys);
    BW_PDL_WAIT();            // (also where nothing is left to do: who waits for this kernel waits for the slices')
    if (slices == 1) return;
    float M = -INFINITY, L = 0.f, O[4] = {0.f, 0.f, 0.f, 0.f};
    constexpr int AHEAD = 8;             // slices whose loads are in flight together
    for (int s0 = 0; s0 < slices; s0 += AHEAD) {
        float4 v[AHEAD];
        float2 ml[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            const size_t at = part_row(p, item.w, min(s0 + i, slices - 1), rows, kvh) + row;
            ml[i] = *reinterpret_cast<const float2*>(p.part_ml + 2 * at);
            v[i] = *reinterpret_cast<const float4*>(p.part_o + at * hd + c);
        }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            if (s0 + i >= slices) break;
            const float2 f = fold(M, L, ml[i].x, ml[i].y);
            O[0] = folded(O[0], v[i].x, f); O[1] = folded(O[1], v[i].y, f); O[2] = folded(O[2], v[i].z, f); O[3] = folded(O[3], v[i].w, f);
        }
    }
    const float inv = L > 0.f ? 1.f / L : 0.f;
    *reinterpret_cast<float4*>(p.out + ((size_t)(row0 + row / G) * p.nh + (size_t)kvh * G + row % G) * hd + c) =
        make_float4(O[0] * inv, O[1] * inv, O[2] * inv, O[3] * inv);
}

template <int ROWS, int CH, bool SLICES>
int go(const Params& p, const int* work, int n, cudaStream_t s) {
    static bool done[bw::MAX_DEVICES] = {};
    constexpr int KT = fetched(ROWS, CH);
    const cudaError_t e = bw::allow_dynamic_smem(attention_f32_kernel<ROWS, CH, SLICES>, 4 * smem_floats(ROWS, CH * 128, KT), done);
    if (e != cudaSuccess) return (int)e;
    bw::launch(attention_f32_kernel<ROWS, CH, SLICES>, dim3(n, p.nkv), dim3(THREADS), 4 * (size_t)smem_floats(ROWS, p.hd, KT), s, p, (const int4*)work);
    BW_LAUNCH_CHECK();
    return 0;
}

}  // namespace

// The keys of a slice, and the slices that a row sees before its slices grow (the work lists count with them).
BW_EXPORT int bw_attention_f32_slice() { return SLICE; }
BW_EXPORT int bw_attention_f32_slices() { return MOST; }

// rows_w: int32 [n_rows][4] (request, first token, 0, 0), tiles of 64 / (nh / nkv) tokens; wide_w: such tiles, and keys_w: segments of at
// most 16 stacked rows, whose slices are dealt out to blocks: [..][4] (request, first token, block | blocks << 16, where), every row's
// slices of one size; merge_w: [n_merge][4] (request, first token, rows, where), at most merge_rows rows each.  part_o, part_ml: float32
// [part_rows * nkv][hd] and [..][2] (null without merge items), part_rows at least the sum of slices times rows of the merged tiles,
// of which `where` counts those before.  hd % 4 == 0, hd <= 256, nh / nkv <= 64.
BW_EXPORT int bw_attention_f32(const float* q, const float* k_pages, const float* v_pages, float* out, const int* cu_q,
                               const int* q_start, const int* block_table, int max_blocks, const int* rows_w, int n_rows,
                               const int* wide_w, int n_wide, const int* keys_w, int n_keys, const int* merge_w, int n_merge,
                               int merge_rows, float* part_o, float* part_ml, int nh, int nkv, int hd, int page_size, int num_pages,
                               int window, int chunk, float scale, void* stream) {
    if (nkv <= 0 || nh % nkv || nh / nkv > 64 || hd <= 0 || hd % 4 || hd > 256) return BW_ERR_UNSUPPORTED;
    if (n_merge && (!part_o || !part_ml || merge_rows <= 0 || merge_rows > 64)) return BW_ERR_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    const Params p = {q, k_pages, v_pages, out, cu_q, q_start, block_table, max_blocks, nh, nkv, hd, page_size, num_pages, window, chunk,
                      scale, part_o, part_ml};
    int rc = 0;
    if (n_rows) rc = hd <= 128 ? go<64, 1, false>(p, rows_w, n_rows, s) : go<64, 2, false>(p, rows_w, n_rows, s);
    if (rc == 0 && n_wide) rc = hd <= 128 ? go<64, 1, true>(p, wide_w, n_wide, s) : go<64, 2, true>(p, wide_w, n_wide, s);
    if (rc == 0 && n_keys) rc = hd <= 128 ? go<SLICE_ROWS, 1, true>(p, keys_w, n_keys, s) : go<SLICE_ROWS, 2, true>(p, keys_w, n_keys, s);
    if (rc == 0 && n_merge) {
        bw::launch(attention_f32_merge_kernel, dim3(n_merge, nkv, merge_rows), dim3(64), 0, s, p, (const int4*)merge_w);
        BW_LAUNCH_CHECK();
    }
    return rc;
}
