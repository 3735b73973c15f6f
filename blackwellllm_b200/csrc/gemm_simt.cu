// out[M,N] (=|+=) x[M,K] . w[N,K]^T (+ bias[N])  on the CUDA cores with float32
// fused multiply-adds: the true 32-bit matrix product (no tensor cores, no reduced
// precision mode).  It is also the fallback for bfloat16 shapes the tensor-core
// kernel refuses (K not a multiple of 8).  Any M, N, K.
//
// Each output element is the sum over k in ascending order of 16-wide slices, so a
// row's result does not depend on what other rows are in the batch.
#include "common.cuh"

using bf16 = __nv_bfloat16;

namespace {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename XT, typename WT, typename BT, typename OT, bool ACCUM>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const XT* __restrict__ x, const WT* __restrict__ w, const BT* __restrict__ bias,
                 OT* __restrict__ out, int M, int N, int K, int ldx, int ldo) {
    __shared__ float xs[BK][BM + 4];
    __shared__ float ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = tid & 15, ty = tid >> 4;  // 16 x 16 threads, each TM x TN outputs
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    // each thread loads 4 elements of each tile per slice: row = tid / 4, k = (tid % 4) * 4 ..+3
    const int lr = tid >> 2, lk = (tid & 3) * 4;
    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int k = k0 + lk + q;
            const int gm = m0 + lr, gn = n0 + lr;
            xs[lk + q][lr] = (gm < M && k < K) ? bw::to_f32(x[(size_t)gm * ldx + k]) : 0.f;
            ws[lk + q][lr] = (gn < N && k < K) ? bw::to_f32(w[(size_t)gn * K + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = xs[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = ws[kk][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty * TM + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx * TN + j;
            if (gn >= N) continue;
            float v = acc[i][j];
            if (bias) v += bw::to_f32(bias[gn]);
            OT* o = out + (size_t)gm * ldo + gn;
            if (ACCUM) v += bw::to_f32(*o);
            *o = bw::from_f32<OT>(v);
        }
    }
}

// ---------------------------------------------------------------- a few tokens (float32)
// Up to 16 tokens (above eight only where gemm_f32_tc.cu does not take the form): bound by the bytes of the weights, which every
// block reads once, straight into registers (16 bytes a lane, a warp 512 contiguous bytes of a row, eight warps side by side along
// K), FEW_ROWS features at a time; the tokens' channels come through L1, where the blocks of an SM find them again.  The 64 x 64
// tiles above read the same bytes with N / 64 blocks, four channels a lane.  Measured at 4 tokens, eight layers of the 8B shape and
// its head: 23.2 ms on the tiles, 1.84 ms here (4096 x 14336: 53 us, 28672 x 4096: 84 us; at 1 token 37 and 69 us).
// A token's result is the same sum in the same order whatever the number of tokens: the even and the odd channels of a lane's
// chunks in ascending order, then lanes, then warps.
constexpr int FEW_TOKENS = 16;
constexpr int FEW_WARPS = 8, FEW_ROWS = 4, FEW_CHUNK = 128;    // channels of a warp's step

// Sums N values (a power of two) over the lanes; each lane is left with max(N / 32, 1) of them, from value `off` on.
template <int N, int SIZE, int O = 16>
__device__ __forceinline__ void lane_sums(float (&v)[SIZE], int& off) {
    if constexpr (O > 0) {
        if constexpr (N > 1) {
            const bool up = threadIdx.x & O;
#pragma unroll
            for (int i = 0; i < N / 2; ++i) {
                const float give = up ? v[i] : v[i + N / 2], keep = up ? v[i + N / 2] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, O);
            }
            if (up) off += N / 2;
            lane_sums<N / 2, SIZE, O / 2>(v, off);
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
            lane_sums<1, SIZE, O / 2>(v, off);
        }
    }
}

template <int TOKENS, bool ACCUM>
__global__ void __launch_bounds__(FEW_WARPS * 32, TOKENS <= 2 ? 4 : (TOKENS <= 4 ? 3 : (TOKENS <= 8 ? 2 : 1)))
gemm_few_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias_f,
                const bf16* __restrict__ bias_h, float* __restrict__ out, int M, int N, int K, int ldx, int ldo) {
    BW_PDL_TRIGGER();
    constexpr int VALUES = FEW_ROWS * TOKENS;
    __shared__ float part[FEW_WARPS][VALUES];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n0 = blockIdx.x * FEW_ROWS;
    const float* wr[FEW_ROWS];
#pragma unroll
    for (int r = 0; r < FEW_ROWS; ++r) wr[r] = w + (size_t)min(n0 + r, N - 1) * K;    // (rows beyond the last: its values, not written)
    bw::f32x2 acc[FEW_ROWS][TOKENS];
#pragma unroll
    for (int r = 0; r < FEW_ROWS; ++r)
#pragma unroll
        for (int t = 0; t < TOKENS; ++t) acc[r][t] = 0ull;
    const int step = FEW_WARPS * FEW_CHUNK;
    int k = warp * FEW_CHUNK + lane * 4;
    // steps whose weights are on their way: with 8 tokens two blocks fit on an SM, which need two steps to keep 64 KB in flight
    constexpr int AHEAD = TOKENS == 8 ? 2 : 1;
    float4 next[AHEAD][FEW_ROWS];
#pragma unroll
    for (int d = 0; d < AHEAD; ++d)
#pragma unroll
        for (int r = 0; r < FEW_ROWS; ++r)
            next[d][r] = k + d * step < K ? __ldcs(reinterpret_cast<const float4*>(wr[r] + k + d * step)) : make_float4(0.f, 0.f, 0.f, 0.f);
    BW_PDL_WAIT();        // the weights are nobody's output; the tokens are
    for (; k < K; k += step) {
        float4 a[FEW_ROWS];
#pragma unroll
        for (int r = 0; r < FEW_ROWS; ++r) {
            a[r] = next[0][r];
            if constexpr (AHEAD == 2) next[0][r] = next[1][r];
        }
        if (k + AHEAD * step < K) {
#pragma unroll
            for (int r = 0; r < FEW_ROWS; ++r) next[AHEAD - 1][r] = __ldcs(reinterpret_cast<const float4*>(wr[r] + k + AHEAD * step));
        }
#pragma unroll
        for (int t = 0; t < TOKENS; ++t) {
            if (t < M) {
                const float4 b = *reinterpret_cast<const float4*>(x + (size_t)t * ldx + k);
                const bw::f32x2 b0 = bw::pack2(b.x, b.y), b1 = bw::pack2(b.z, b.w);
#pragma unroll
                for (int r = 0; r < FEW_ROWS; ++r) {
                    acc[r][t] = bw::fma2(bw::pack2(a[r].x, a[r].y), b0, acc[r][t]);
                    acc[r][t] = bw::fma2(bw::pack2(a[r].z, a[r].w), b1, acc[r][t]);
                }
            }
        }
    }
    float v[VALUES];
#pragma unroll
    for (int r = 0; r < FEW_ROWS; ++r)
#pragma unroll
        for (int t = 0; t < TOKENS; ++t) v[r * TOKENS + t] = bw::sum2(acc[r][t]);
    int off = 0;
    lane_sums<VALUES>(v, off);
#pragma unroll
    for (int i = 0; i < (VALUES > 32 ? VALUES / 32 : 1); ++i) part[warp][off + i] = v[i];
    __syncthreads();
    for (int i = threadIdx.x; i < VALUES; i += blockDim.x) {
        const int n = n0 + i / TOKENS, t = i % TOKENS;
        if (n >= N || t >= M) continue;
        float s = part[0][i];
#pragma unroll
        for (int p = 1; p < FEW_WARPS; ++p) s += part[p][i];
        if (bias_f) s += bias_f[n];
        if (bias_h) s += bw::to_f32(bias_h[n]);
        float* o = out + (size_t)t * ldo + n;
        *o = ACCUM ? s + *o : s;
    }
}

int launch_few(const float* x, const float* w, const void* bias, int bias_type, float* out, int M, int N, int K, int ldx, int ldo,
               int accumulate, cudaStream_t s) {
    const float* bf = bias && bias_type != BW_BF16 ? (const float*)bias : nullptr;
    const bf16* bh = bias && bias_type == BW_BF16 ? (const bf16*)bias : nullptr;
    const dim3 grid((N + FEW_ROWS - 1) / FEW_ROWS), block(FEW_WARPS * 32);
#define BW_FEW(T) (accumulate ? bw::launch(gemm_few_kernel<T, true>, grid, block, 0, s, x, w, bf, bh, out, M, N, K, ldx, ldo) \
                              : bw::launch(gemm_few_kernel<T, false>, grid, block, 0, s, x, w, bf, bh, out, M, N, K, ldx, ldo))
    if (M <= 1) BW_FEW(1);
    else if (M <= 2) BW_FEW(2);
    else if (M <= 4) BW_FEW(4);
    else if (M <= 8) BW_FEW(8);
    else BW_FEW(16);
#undef BW_FEW
    BW_LAUNCH_CHECK();
    return 0;
}

template <typename XT, typename WT, typename OT>
int launch(const void* x, const void* w, const void* bias, int bias_type, void* out, int M, int N, int K,
           int ldx, int ldo, int accumulate, cudaStream_t s) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    const XT* xp = (const XT*)x; const WT* wp = (const WT*)w; OT* op = (OT*)out;
#define BW_GO(BT, ACC) gemm_simt_kernel<XT, WT, BT, OT, ACC><<<grid, 256, 0, s>>>(xp, wp, (const BT*)bias, op, M, N, K, ldx, ldo)
    if (bias && bias_type == BW_BF16) { if (accumulate) BW_GO(bf16, true); else BW_GO(bf16, false); }
    else { if (accumulate) BW_GO(float, true); else BW_GO(float, false); }
#undef BW_GO
    BW_LAUNCH_CHECK();
    return 0;
}

}  // namespace

// in_type: type of x and w (both the same); out_type: type of out.
// accumulate != 0: out += product (out must be float32: the residual stream).
BW_EXPORT int bw_gemm_simt(const void* x, const void* w, int in_type, const void* bias, int bias_type,
                           void* out, int out_type, int M, int N, int K, int ldx, int ldo,
                           int accumulate, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || ldx < K || ldo < N) return BW_ERR_BAD_ARG;
    if (accumulate && out_type != BW_F32) return BW_ERR_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    // 16-byte loads: channels in fours, rows that begin on 16 bytes
    const bool vec = K % 4 == 0 && ldx % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0;
    if (in_type == BW_F32 && out_type == BW_F32 && vec && M <= FEW_TOKENS)
        return launch_few((const float*)x, (const float*)w, bias, bias_type, (float*)out, M, N, K, ldx, ldo, accumulate, s);
    if (in_type == BW_F32 && out_type == BW_F32)
        return launch<float, float, float>(x, w, bias, bias_type, out, M, N, K, ldx, ldo, accumulate, s);
    if (in_type == BW_BF16 && out_type == BW_F32)
        return launch<bf16, bf16, float>(x, w, bias, bias_type, out, M, N, K, ldx, ldo, accumulate, s);
    if (in_type == BW_BF16 && out_type == BW_BF16)
        return launch<bf16, bf16, bf16>(x, w, bias, bias_type, out, M, N, K, ldx, ldo, accumulate, s);
    return BW_ERR_BAD_ARG;
}
