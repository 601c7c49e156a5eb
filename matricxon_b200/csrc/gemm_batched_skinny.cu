// Many small independent products with at most 16 rows each (the per-head and per-block products of a
// decode step): out[m][b][n] = sum_k A[m][b][k] * W[b][n][k], bfloat16 in, float accumulation.
//
// K a multiple of 32: a block of four warps forms 16 columns of a member on the tensor cores (mma.sync, the columns'
// weight rows as its 16 rows, the rows of A as its 8 columns, one or two of them). Warp w takes the blocks of 32 k
// numbered w, w + 4, ..., every thread 16 contiguous bytes of two weight rows and of a row of A a block, the
// contraction permuted the same way on both sides, and the warps' sums are added in a fixed order, so a row's
// result does not depend on the other rows. The products are a few microseconds of launches and latencies (16 heads of
// 512 x 128 are 2 MB): the first weights set out for L2 before the wait on the kernels before.
// Other K: one warp per output column (b, n): the weight row is read once with 16-byte loads (lane l takes the
// elements 8l .. 8l+7 of every block of 256), every row of A against it, and the lanes' partial sums are
// added by shuffles in a fixed order. Sixteen requests decoding with four latent
// attentions and two gated recurrences (ten of these products) took 801 us a step that way, on the tensor cores 691: a
// multiply-add a lane and element, half of the lanes idle at K = 128, and eighty shuffles a column were 17 us a product.
// The operands of the batch members may interleave (heads side by side in a row): rows are lda / ldo apart, members
// a_batch / w_batch / o_batch apart. Takes part in chained launches. K must be a multiple of 8 and every row 16-byte aligned.
#include "common.cuh"

namespace {

constexpr int BS_ROWS = 16;
constexpr int BS_WARPS = 8;

template <typename TOut>
__global__ void __launch_bounds__(BS_WARPS * 32)
batched_skinny_kernel(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ W,
                      TOut* __restrict__ out, int M, int N, int K, int lda, int ldw, int ldo, int batch,
                      long long a_batch, long long w_batch, long long o_batch) {
    pdl_trigger();
    pdl_wait();
    A = after_wait(A);
    const long long column = (long long)blockIdx.x * BS_WARPS + (threadIdx.x >> 5);
    if (column >= (long long)batch * N) return;
    const int b = (int)(column / N), n = (int)(column - (long long)b * N);
    const int lane = threadIdx.x & 31;
    const __nv_bfloat16* w = W + (size_t)b * w_batch + (size_t)n * ldw;
    const __nv_bfloat16* a = A + (size_t)b * a_batch;
    float acc[BS_ROWS];
#pragma unroll
    for (int m = 0; m < BS_ROWS; ++m) acc[m] = 0.f;
    for (int k = lane * 8; k < K; k += 256) {
        const uint4 wraw = *reinterpret_cast<const uint4*>(w + k);
        const __nv_bfloat162* w2 = reinterpret_cast<const __nv_bfloat162*>(&wraw);
        float wf[8];
#pragma unroll
        for (int e = 0; e < 4; ++e) { wf[2 * e] = __low2float(w2[e]); wf[2 * e + 1] = __high2float(w2[e]); }
#pragma unroll
        for (int m = 0; m < BS_ROWS; ++m) {
            if (m < M) {
                const uint4 araw = *reinterpret_cast<const uint4*>(a + (size_t)m * lda + k);
                const __nv_bfloat162* a2 = reinterpret_cast<const __nv_bfloat162*>(&araw);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    acc[m] = fmaf(__low2float(a2[e]), wf[2 * e], acc[m]);
                    acc[m] = fmaf(__high2float(a2[e]), wf[2 * e + 1], acc[m]);
                }
            }
        }
    }
#pragma unroll
    for (int m = 0; m < BS_ROWS; ++m) {
        if (m < M) {
            const float total = warp_sum(acc[m]);
            if (lane == 0) out[(size_t)m * ldo + (size_t)b * o_batch + n] = from_float<TOut>(total);
        }
    }
}

__device__ __forceinline__ void bs_mma(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0,
                                       unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The sum of a block of 32 k to a float's last digits. The tensor cores cut off what lies below the digits of the sum
// they form: each product of 16 k is formed a second time on top of its negated first result, which leaves what was
// lost. Results against 64 bits at 16 heads of 128 x 512: 6.1e-8 off (a lane's multiply-adds, the other kernel: 6.2e-8;
// one chain of mma a warp: 12.6e-8) for 2.7 us with 4 rows and 4.2 with 16 (the chain 2.8 and 3.3). Only for results
// that stay float: rounding to bfloat16 hides the difference.
__device__ __forceinline__ void bs_mma_exact(float (&sum)[4], const uint4& w0, const uint4& w1, const uint4& a) {
    float d[2][4] = {}, lost[2][4];
    bs_mma(d[0], w0.x, w1.x, w0.y, w1.y, a.x, a.y);
    bs_mma(d[1], w0.z, w1.z, w0.w, w1.w, a.z, a.w);
#pragma unroll
    for (int e = 0; e < 4; ++e) lost[0][e] = -d[0][e], lost[1][e] = -d[1][e];
    bs_mma(lost[0], w0.x, w1.x, w0.y, w1.y, a.x, a.y);
    bs_mma(lost[1], w0.z, w1.z, w0.w, w1.w, a.z, a.w);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float back = lost[0][e] + lost[1][e];
        sum[e] = (d[0][e] + d[1][e]) + (back == back ? back : 0.f);      // an infinite sum has lost nothing: inf - inf
    }
}

constexpr int BM_WARPS = 4, BM_AHEAD = 4;      // BM_AHEAD: blocks of 32 k whose weights a thread holds at a time

template <typename TOut, int MB>
__global__ void __launch_bounds__(BM_WARPS * 32)
batched_mma_kernel(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ W, TOut* __restrict__ out, int M,
                   int N, int K, int lda, int ldw, int ldo, int tiles, long long a_batch, long long w_batch,
                   long long o_batch) {
    __shared__ float sums[BM_WARPS][16][8 * MB];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int b = blockIdx.x / tiles, n0 = (blockIdx.x - b * tiles) * 16;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    const __nv_bfloat16* w_row[2];
    bool w_in[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        w_in[i] = n0 + g + 8 * i < N;
        w_row[i] = W + (size_t)b * w_batch + (size_t)min(n0 + g + 8 * i, N - 1) * ldw + 8 * t;
    }
    const int blocks = K / 32;
    uint4 wf[BM_AHEAD][2];
    auto weights = [&](int kb0) {
#pragma unroll
        for (int u = 0; u < BM_AHEAD; ++u)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int kb = kb0 + u * BM_WARPS;
                wf[u][i] = kb < blocks && w_in[i] ? *reinterpret_cast<const uint4*>(w_row[i] + 32 * kb) : zero;
            }
    };
    // The weights may be what the kernel before wrote, as any operand of a product may: before the wait they are only
    // asked into L2 (16 heads of 512 x 128, 4 and 16 rows: 2.6 and 3.4 us; read into registers there 2.6 and 3.5).
#pragma unroll
    for (int u = 0; u < BM_AHEAD; ++u)
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (w_in[i] && warp + u * BM_WARPS < blocks) prefetch_l2(w_row[i] + 32 * (warp + u * BM_WARPS));
    pdl_trigger();
    pdl_wait();
#pragma unroll
    for (int i = 0; i < 2; ++i) w_row[i] = after_wait(w_row[i]);
    weights(warp);
    const __nv_bfloat16* a_row[MB];
    bool a_in[MB];
#pragma unroll
    for (int mb = 0; mb < MB; ++mb) {
        a_in[mb] = 8 * mb + g < M;
        a_row[mb] = after_wait(A) + (size_t)b * a_batch + (size_t)min(8 * mb + g, M - 1) * lda + 8 * t;
    }
    float acc[MB][4];
#pragma unroll
    for (int mb = 0; mb < MB; ++mb) acc[mb][0] = acc[mb][1] = acc[mb][2] = acc[mb][3] = 0.f;
    for (int kb0 = warp; kb0 < blocks; kb0 += BM_AHEAD * BM_WARPS) {
        if (kb0 != warp) weights(kb0);
        uint4 af[BM_AHEAD][MB];
#pragma unroll
        for (int u = 0; u < BM_AHEAD; ++u)
#pragma unroll
            for (int mb = 0; mb < MB; ++mb) {
                const int kb = kb0 + u * BM_WARPS;
                af[u][mb] = kb < blocks && a_in[mb] ? *reinterpret_cast<const uint4*>(a_row[mb] + 32 * kb) : zero;
            }
#pragma unroll
        for (int mb = 0; mb < MB; ++mb) {
            float part[BM_AHEAD][4];                          // float results: the blocks' sums, what they lost added back
#pragma unroll
            for (int u = 0; u < BM_AHEAD; ++u) {
                if constexpr (sizeof(TOut) == 4) {
                    bs_mma_exact(part[u], wf[u][0], wf[u][1], af[u][mb]);
                } else {
                    bs_mma(acc[mb], wf[u][0].x, wf[u][1].x, wf[u][0].y, wf[u][1].y, af[u][mb].x, af[u][mb].y);
                    bs_mma(acc[mb], wf[u][0].z, wf[u][1].z, wf[u][0].w, wf[u][1].w, af[u][mb].z, af[u][mb].w);
                }
            }
            if constexpr (sizeof(TOut) == 4)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[mb][e] += (part[0][e] + part[1][e]) + (part[2][e] + part[3][e]);
        }
    }
    // this thread holds columns g and g + 8 for rows 8 mb + 2t, + 1
#pragma unroll
    for (int mb = 0; mb < MB; ++mb)
#pragma unroll
        for (int e = 0; e < 4; ++e) sums[warp][g + 8 * (e >> 1)][8 * mb + 2 * t + (e & 1)] = acc[mb][e];
    __syncthreads();
    for (int idx = threadIdx.x; idx < 16 * 8 * MB; idx += BM_WARPS * 32) {
        const int f = idx % 16, m = idx / 16;
        if (n0 + f >= N || m >= M) continue;
        const float v = (sums[0][f][m] + sums[1][f][m]) + (sums[2][f][m] + sums[3][f][m]);
        out[(size_t)m * ldo + (size_t)b * o_batch + n0 + f] = from_float<TOut>(v);
    }
}

template <typename TOut>
cudaError_t launch_mma(const void* A, const void* W, void* out, int M, int N, int K, int lda, int ldw, int ldo, int batch,
                       long long a_batch, long long w_batch, long long o_batch, cudaStream_t stream) {
    const int tiles = (N + 15) / 16;
    return mx_launch_chained(M <= 8 ? batched_mma_kernel<TOut, 1> : batched_mma_kernel<TOut, 2>,
                             dim3((unsigned)(tiles * (long long)batch)), dim3(BM_WARPS * 32), 0, stream,
                             (const __nv_bfloat16*)A, (const __nv_bfloat16*)W, (TOut*)out, M, N, K, lda, ldw, ldo, tiles,
                             a_batch, w_batch, o_batch);
}

}  // namespace

extern "C" int mx_gemm_batched_skinny(const void* A, const void* W, void* out, int out_dtype, int M, int N, int K,
                                      int lda, int ldw, int ldo, int batch, long long a_batch, long long w_batch,
                                      long long o_batch, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || batch <= 0) return MX_OK;
    if (M > BS_ROWS) MX_REFUSE("batched skinny product: %d rows exceed %d", M, BS_ROWS);
    if (K <= 0 || K % 8 || lda % 8 || ldw % 8 || a_batch % 8 || w_batch % 8)
        MX_REFUSE("batched skinny product: K = %d and the strides must be multiples of 8", K);
    if (K % 32 == 0) {
        const cudaError_t e = out_dtype == MX_DTYPE_F32
                                  ? launch_mma<float>(A, W, out, M, N, K, lda, ldw, ldo, batch, a_batch, w_batch, o_batch, stream)
                                  : launch_mma<__nv_bfloat16>(A, W, out, M, N, K, lda, ldw, ldo, batch, a_batch, w_batch, o_batch, stream);
        if (e != cudaSuccess) mx_set_error("batched skinny product: launch failed: %s", cudaGetErrorString(e));
        return (int)e;
    }
    const long long columns = (long long)batch * N;
    const unsigned blocks = (unsigned)((columns + BS_WARPS - 1) / BS_WARPS);
    if (out_dtype == MX_DTYPE_F32)
        mx_launch_chained(batched_skinny_kernel<float>, dim3(blocks), dim3(BS_WARPS * 32), 0, stream,
                          (const __nv_bfloat16*)A, (const __nv_bfloat16*)W, (float*)out, M, N, K, lda, ldw, ldo, batch,
                          a_batch, w_batch, o_batch);
    else
        mx_launch_chained(batched_skinny_kernel<__nv_bfloat16>, dim3(blocks), dim3(BS_WARPS * 32), 0, stream,
                          (const __nv_bfloat16*)A, (const __nv_bfloat16*)W, (__nv_bfloat16*)out, M, N, K, lda, ldw, ldo,
                          batch, a_batch, w_batch, o_batch);
    return mx_launch_status();
}
