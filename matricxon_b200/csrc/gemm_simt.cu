// out[M,N] = epilogue(A[M,K] . W[N,K]^T + bias[N]) on the FP32 cores.
//
// This is the plain 32-bit matrix product of the engine (inputs, products and sums are
// float), and the twin that the tensor-core products are checked against, those of floats
// in three parts (gemm_f32_split.cu, which takes the larger products of three rows and
// more) among them. Each output element is one fixed-order sum over K, whatever M is, so a
// row's result does not depend on what else is in the batch: four chains over a quarter of K
// each, added as (p0 + p1) + (p2 + p3) (gemm_f32.cuh; one chain over all of K leaves few
// threads to a decoding row, and its rounding errors are twice as large). Float operands
// that can be read 16 bytes at a time go to gemm_f32.cu, which forms the same sums. The
// reference runs these products through nn.Linear (app/architectures/qwen_layers.py:50-53,
// app/architectures/starcoder2_layers.py:19-23).
//
// Epilogue modes: 0 out(T) = v; 1 out(T) = gelu_tanh(v); 2 out(f32) = residual + v;
// 3 out(f32) = v; 4 out(T) = max(v, 0)^2, where v = acc + bias.
#include "common.cuh"
#include "gemm_f32.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;
constexpr int THREADS = (BM / TM) * (BN / TN);  // 256

// Bound by latency where a block has an SM to itself and by what shared memory hands to registers where blocks fill the
// SMs. A k-tile's operands are on their way in registers while the one before is worked on, and the pieces that are done
// wait in shared memory: 64 registers, four blocks an SM. 389 x 2,048 x 2,047: 166 us, 16 members of 2,048 x 512 x 128:
// 185, 16 x 2,048 x 2,047: 95 (the pieces in registers, 102 of them, two blocks an SM: 195, 224 and 159; one chain over
// K in 40 registers without the loads ahead: 238, 179 and 247). Five blocks an SM leave the loads ahead no registers
// (205, 203 and 159).
template <typename TIn, typename TOut>
__global__ void __launch_bounds__(THREADS, 4)
gemm_simt_kernel(const TIn* __restrict__ A, const TIn* __restrict__ W,
                 const float* __restrict__ bias, const float* residual, TOut* out,
                 int M, int N, int K, int lda, int ldw, int ldo, int mode,
                 long long a_batch, long long w_batch, long long o_batch, long long bias_batch) {
    // blockIdx.z: one of several independent products (a head, a block of a block-diagonal matrix)
    A += (size_t)blockIdx.z * a_batch;
    W += (size_t)blockIdx.z * w_batch;
    out += (size_t)blockIdx.z * o_batch;
    if (bias) bias += (size_t)blockIdx.z * bias_batch;
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = tid % (BN / TN), ty = tid / (BN / TN);

    float acc[TM][TN];                                   // the piece in hand
    __shared__ float4 saved[2][TM][THREADS];             // p0, then p0 + p1; p2
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    const int piece = f32_piece(K);
    int left = piece, ended = 0;                         // k to the end of the piece; pieces behind it

    // each thread stages 4 elements of A and 4 of W per k-tile: row = tid / 4, 4 k's at (tid % 4) * 4; rows of the upper
    // eight k are moved by eight floats, so that a warp's writes of four k fall on different banks
    const int lrow = tid >> 2, lk = (tid & 3) << 2;
    const bool a_in = m0 + lrow < M, w_in = n0 + lrow < N;
    const TIn* a_row = A + (size_t)(a_in ? m0 + lrow : 0) * lda;
    const TIn* w_row = W + (size_t)(w_in ? n0 + lrow : 0) * ldw;
    const int put = lrow ^ (lk & 8);
    float na[4], nw[4];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int k = k0 + lk + e;
            na[e] = (a_in && k < K) ? to_float(a_row[k]) : 0.f;
            nw[e] = (w_in && k < K) ? to_float(w_row[k]) : 0.f;
        }
    };
    fetch(0);
    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            As[lk + e][put] = na[e];
            Ws[lk + e][put] = nw[e];
        }
        __syncthreads();
        fetch(k0 + BK);
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], w[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[kk][((ty * TM) ^ (kk & 8)) + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = Ws[kk][((tx * TN) ^ (kk & 8)) + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
        left -= BK;
        if (left == 0 && k0 + BK < K) {                      // a piece ends (its length is a multiple of BK)
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                float4 v = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
                if (ended == 1) {
                    const float4 p0 = saved[0][i][tid];
                    v = make_float4(p0.x + v.x, p0.y + v.y, p0.z + v.z, p0.w + v.w);
                }
                saved[ended == 2][i][tid] = v;
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
            }
            ++ended;
            left = piece;
        }
    }
    // the last piece that has any k: p0 or p2 stands alone, p1 or p3 joins the one before it
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 p2 = ended == 3 ? saved[1][i][tid] : none, sum = ended > 0 ? saved[0][i][tid] : none;
        acc[i][0] = sum.x + (p2.x + acc[i][0]);
        acc[i][1] = sum.y + (p2.y + acc[i][1]);
        acc[i][2] = sum.z + (p2.z + acc[i][2]);
        acc[i][3] = sum.w + (p2.w + acc[i][3]);
    }

#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx * TN + j;
            if (n >= N) continue;
            float v = acc[i][j];
            if (bias) v += bias[n];
            v = mode_activation(v, mode);
            const size_t o = (size_t)m * ldo + n;
            if (mode == 2) v += residual[o];
            out[o] = from_float<TOut>(v);
        }
    }
}

}  // namespace

extern "C" int mx_gemm_simt(const void* A, const void* W, int in_dtype, const float* bias,
                            const float* residual, void* out, int out_dtype, int M, int N, int K,
                            int lda, int ldw, int ldo, int mode, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return MX_OK;
    if (K <= 0) MX_REFUSE("gemm: K must be positive, got %d", K);
    if (mode < 0 || mode > MX_MODE_LAST) MX_REFUSE("gemm: unknown epilogue mode %d", mode);
    if (mode == 2 && residual == nullptr) MX_REFUSE("gemm: residual mode without a residual");
    const int expected_out = (mx_mode_is_float(mode) || in_dtype == MX_DTYPE_F32) ? MX_DTYPE_F32 : MX_DTYPE_BF16;
    if (out_dtype != expected_out)
        MX_REFUSE("gemm: epilogue mode %d with input dtype %d writes dtype %d, not %d", mode,
                  in_dtype, expected_out, out_dtype);
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) MX_REFUSE("gemm: M = %d is beyond this kernel's grid", M);
    if (in_dtype == MX_DTYPE_F32 && mx_gemm_f32_takes((const float*)A, lda, (const float*)W, ldw, M, N, K))
        return mx_gemm_f32((const float*)A, lda, (const float*)W, ldw, bias, residual, (float*)out, ldo, M, N, K, mode, stream);
#define MX_GEMM(TI, TO) \
    gemm_simt_kernel<TI, TO><<<grid, THREADS, 0, stream>>>((const TI*)A, (const TI*)W, bias, residual, (TO*)out, M, N, K, lda, ldw, ldo, mode, 0, 0, 0, 0)
    if (in_dtype == MX_DTYPE_F32 && out_dtype == MX_DTYPE_F32) MX_GEMM(float, float);
    else if (in_dtype == MX_DTYPE_BF16 && out_dtype == MX_DTYPE_F32) MX_GEMM(__nv_bfloat16, float);
    else if (in_dtype == MX_DTYPE_BF16 && out_dtype == MX_DTYPE_BF16) MX_GEMM(__nv_bfloat16, __nv_bfloat16);
    else MX_REFUSE("gemm: float inputs with a bfloat16 output are not used by any path");
#undef MX_GEMM
    return mx_launch_status();
}

// `batch` independent products of the same shape in one launch: product b reads A + b * a_batch
// (rows lda apart) and W + b * w_batch, adds bias + b * bias_batch and writes out + b * o_batch (rows
// ldo apart). The operands of a batch may interleave (heads side by side in one row). mode 0 writes
// the input dtype, mode 3 float.
extern "C" int mx_gemm_batched_simt(const void* A, const void* W, int in_dtype, const float* bias, void* out,
                                    int out_dtype, int M, int N, int K, int lda, int ldw, int ldo, int batch,
                                    long long a_batch, long long w_batch, long long o_batch,
                                    long long bias_batch, int mode, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || batch <= 0) return MX_OK;
    if (K <= 0) MX_REFUSE("batched gemm: K must be positive, got %d", K);
    if (mode != 0 && mode != 3) MX_REFUSE("batched gemm: epilogue mode %d", mode);
    const int expected_out = (mode == 3 || in_dtype == MX_DTYPE_F32) ? MX_DTYPE_F32 : MX_DTYPE_BF16;
    if (out_dtype != expected_out) MX_REFUSE("batched gemm: mode %d writes dtype %d, not %d", mode, expected_out, out_dtype);
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batch);
    if (grid.y > 65535 || batch > 65535) MX_REFUSE("batched gemm: M = %d, batch = %d is beyond this kernel's grid", M, batch);
#define MX_GEMM(TI, TO) \
    gemm_simt_kernel<TI, TO><<<grid, THREADS, 0, stream>>>((const TI*)A, (const TI*)W, bias, nullptr, (TO*)out, M, N, K, lda, ldw, ldo, mode, a_batch, w_batch, o_batch, bias_batch)
    if (in_dtype == MX_DTYPE_F32) MX_GEMM(float, float);
    else if (out_dtype == MX_DTYPE_F32) MX_GEMM(__nv_bfloat16, float);
    else MX_GEMM(__nv_bfloat16, __nv_bfloat16);
#undef MX_GEMM
    return mx_launch_status();
}
