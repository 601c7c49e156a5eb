// out[M,N] = epilogue(A[M,K] . W[N,K]^T + bias[N]), all float, on the FP32 cores: the products of the 32-bit path
// whose operands can be read 16 bytes at a time. gemm_simt.cu holds the general kernel and the order of the sum,
// which both kernels here keep: K is cut into four pieces of f32_piece(K), each piece is one chain of fused
// multiply-adds in the order of k, and the result is (p0 + p1) + (p2 + p3). A row's result is therefore the same
// bit for bit whichever of the kernels forms it and whatever else is in the batch. The reference runs these products
// through nn.Linear (app/architectures/qwen_layers.py:50-53, app/architectures/starcoder2_layers.py:19-23).
#include <cooperative_groups.h>

#include "common.cuh"
#include "gemm_f32.cuh"

namespace {

namespace cg = cooperative_groups;

__device__ __forceinline__ void copy16(float* dst, const float* src, bool in) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int bytes = in ? 16 : 0;                    // the rest is filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// ------------------------------------------------------------------------------------------- few rows
// Decoding: the product is a stream of W from HBM. A block owns up to 32 weight rows (a lane each) and its four
// warps take one piece of K each, so the four chains of an output are four threads. A warp keeps a ring of its own
// of [32 rows][32 floats] of W and [rows of A][32 floats], filled by cp.async (a 128-byte line per row, chunks
// permuted so that the 32 lanes' 16-byte reads spread over all banks): no block-wide barrier in the loop. A row of A is
// read as a broadcast. Weights of 3072 x 12288 / 12288 x 3072 / 49152 x 3072: 38 / 32 / 96 us for one row (4.0, 4.7, 6.2 TB/s),
// 52 / 38 / 105 us for four; the general kernel, which walks tiles of 64 rows, takes 569 us for the first (one column of
// K less). What is in flight bounds it: five chunks of 128 bytes a warp and weight row, so 54 KB an SM in the first (147
// blocks of 21 rows, one an SM), 143 KB in the second while two blocks share an SM and 72 KB in its last round (439
// blocks of 28), 159 KB in the third (31 rows); two blocks fit an SM up to four rows of A (99 to 108 KB of ring each), one
// above. From about eight rows on the reads of A from shared memory bound it (128 bytes a cycle and SM go to registers,
// broadcast or not): 67 us for eight in the first.
constexpr int FR_ROWS = 32, FR_K = 32, FR_STAGES = 6, FR_THREADS = 128;

template <int MB>
__global__ void __launch_bounds__(FR_THREADS)
gemm_f32_rows_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                     const float* __restrict__ bias, const float* residual, float* out, int ldo, int M, int N, int K,
                     int piece, int rows, int mode) {
    extern __shared__ float4 fr_smem4[];
    constexpr int W_FLOATS = FR_ROWS * FR_K, STAGE = W_FLOATS + MB * FR_K;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* ring = reinterpret_cast<float*>(fr_smem4) + (size_t)warp * FR_STAGES * STAGE;
    const int n0 = blockIdx.x * rows, m0 = blockIdx.y * MB;
    const int n_rows = min(rows, N - n0), m_rows = min(MB, M - m0);
    const int k_begin = min(warp * piece, K), k_end = min(k_begin + piece, K);
    const int chunks = (k_end - k_begin + FR_K - 1) / FR_K;

    // the weights are nobody's output: their first lines set out for L2 while the kernel before this one ends
    if (lane < n_rows)
        for (int c = 0; c < min(chunks, FR_STAGES - 1); ++c)
            prefetch_l2(W + (size_t)(n0 + lane) * ldw + k_begin + c * FR_K);
    pdl_wait();
    A = after_wait(A);
    residual = after_wait(residual);

    const int col = 4 * (lane & 7), sub = lane >> 3;
    auto fetch = [&](int c) {
        float* stage = ring + (c % FR_STAGES) * STAGE;
        const int k = k_begin + c * FR_K + col;
        const bool k_in = k < k_end;                  // K and the pieces are multiples of 4
#pragma unroll
        for (int i = 0; i < FR_ROWS / 4; ++i) {
            const int r = 4 * i + sub;
            if (r < n_rows)
                copy16(stage + r * FR_K + (col ^ (4 * (r & 7))), k_in ? W + (size_t)(n0 + r) * ldw + k : W, k_in);
        }
#pragma unroll
        for (int i = 0; i < (MB + 3) / 4; ++i) {
            const int m = 4 * i + sub;
            if (m < m_rows)
                copy16(stage + W_FLOATS + m * FR_K + col, k_in ? A + (size_t)(m0 + m) * lda + k : A, k_in);
        }
    };
    float acc[MB];
#pragma unroll
    for (int m = 0; m < MB; ++m) acc[m] = 0.f;
    for (int c = 0; c < FR_STAGES - 1; ++c) {
        if (c < chunks) fetch(c);
        copy_commit();
    }
    for (int c = 0; c < chunks; ++c) {
        copy_wait<FR_STAGES - 2>();
        __syncwarp();                                 // chunk c is in place, and everyone is done with chunk c - 1
        if (c + FR_STAGES - 1 < chunks) fetch(c + FR_STAGES - 1);
        copy_commit();
        const float* stage = ring + (c % FR_STAGES) * STAGE;
        // a warp has few others beside it to hide behind: the chunk's weights and the first rows of A are read
        // ahead of the arithmetic, which then runs one vector of A behind its loads (two weight rows a lane, so that
        // a value of A is read by half as many lanes, took 63 us for 3072 x 12288 and four rows instead of 52)
        float4 w[FR_K / 4], a[2][MB];
#pragma unroll
        for (int q = 0; q < FR_K / 4; ++q)
            w[q] = *reinterpret_cast<const float4*>(stage + lane * FR_K + ((4 * q) ^ (4 * (lane & 7))));
#pragma unroll
        for (int m = 0; m < MB; ++m) a[0][m] = *reinterpret_cast<const float4*>(stage + W_FLOATS + m * FR_K);
#pragma unroll
        for (int q = 0; q < FR_K / 4; ++q) {
            if (q + 1 < FR_K / 4) {
#pragma unroll
                for (int m = 0; m < MB; ++m)
                    a[(q + 1) & 1][m] = *reinterpret_cast<const float4*>(stage + W_FLOATS + m * FR_K + 4 * (q + 1));
            }
#pragma unroll
            for (int m = 0; m < MB; ++m) acc[m] = fmaf(a[q & 1][m].x, w[q].x, acc[m]);
#pragma unroll
            for (int m = 0; m < MB; ++m) acc[m] = fmaf(a[q & 1][m].y, w[q].y, acc[m]);
#pragma unroll
            for (int m = 0; m < MB; ++m) acc[m] = fmaf(a[q & 1][m].z, w[q].z, acc[m]);
#pragma unroll
            for (int m = 0; m < MB; ++m) acc[m] = fmaf(a[q & 1][m].w, w[q].w, acc[m]);
        }
    }
    copy_wait<0>();
    pdl_trigger();
    __syncthreads();                                  // the rings are read: they hold the pieces' sums from here on
    float* sums = reinterpret_cast<float*>(fr_smem4);                // [piece][row of A][weight row]
#pragma unroll
    for (int m = 0; m < MB; ++m) sums[(warp * MB + m) * FR_ROWS + lane] = acc[m];
    __syncthreads();
    for (int i = threadIdx.x; i < MB * FR_ROWS; i += FR_THREADS) {
        const int f = i % FR_ROWS, m = i / FR_ROWS;
        if (f >= n_rows || m >= m_rows) continue;
        float v = (sums[i] + sums[MB * FR_ROWS + i]) + (sums[2 * MB * FR_ROWS + i] + sums[3 * MB * FR_ROWS + i]);
        const int n = n0 + f;
        if (bias) v += bias[n];
        v = mode_activation(v, mode);
        const size_t o = (size_t)(m0 + m) * ldo + n;
        if (mode == MX_MODE_RESIDUAL) v += residual[o];
        out[o] = v;
    }
}

// ------------------------------------------------------------------------------------------- many rows
// Prompts: bound by the FP32 pipes (128 multiply-adds a cycle and SM) and beside them by what shared memory hands to
// registers, 128 bytes a cycle. A block of 128 threads forms 64 rows x 128 features of one piece of K, 8 x 8 outputs a
// thread as 8 x 4 packed pairs of features (fma.rn.f32x2: half the issue slots). Shared memory holds a step of 16 k
// with k outermost, so that 16 bytes of W are two pairs as the instruction wants them; the other operand, a value of A
// twice, is formed in registers. The next step's operands are on their way in registers meanwhile. The four pieces of K are
// the four blocks of a cluster (a 3,072-wide product of some hundred rows has too few tiles for 148 SMs otherwise);
// each leaves its sums in its shared memory and finishes a quarter of the tile from all four. 128 registers (28 bytes a
// thread wait in local memory), four blocks an SM: issue slots 54 % and L1 74 % busy. Measured at 389 rows (the four
// products of a 3B layer): 1.94 ms, 38 TFLOP/s; with A's values twice each in shared memory, 162 registers and three
// blocks an SM, 2.28; unpacked from rows as they lie in memory, by cp.async, 2.38; 56 rows x 256 features with 7 x 16
// outputs a thread, two blocks an SM, 2.36; 64 x 192 unpacked 3.04; the general kernel (a column of K less) 3.40.
constexpr int FT_M = 64, FT_N = 128, FT_K = 16, FT_THREADS = 128;
constexpr int FT_LDA = FT_M + 4, FT_LDW = FT_N + 4;              // floats from one k to the next
constexpr int FT_BUFFER = FT_K * (FT_LDA + FT_LDW);
constexpr int FT_OUT_LD = FT_N + 4;
constexpr int FT_FLOATS = 2 * FT_BUFFER > FT_M * FT_OUT_LD ? 2 * FT_BUFFER : FT_M * FT_OUT_LD;

typedef unsigned long long pair_t;                               // two floats, low word first
__device__ __forceinline__ void fma_pair(pair_t& acc, pair_t a, pair_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(acc) : "l"(a), "l"(b));
}

__device__ __forceinline__ pair_t both(float v) {
    pair_t p;
    asm("mov.b64 %0, {%1, %1};\n" : "=l"(p) : "f"(v));
    return p;
}

__global__ void __cluster_dims__(F32_PIECES, 1, 1) __launch_bounds__(FT_THREADS, 4)
gemm_f32_tile_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                     const float* __restrict__ bias, const float* residual, float* out, int ldo, int M, int N, int K,
                     int piece, int mode) {
    __shared__ __align__(16) float smem[FT_FLOATS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = blockIdx.x % F32_PIECES;
    const int m0 = (blockIdx.x / F32_PIECES) * FT_M, n0 = blockIdx.y * FT_N;
    const int k_begin = min(rank * piece, K), k_end = min(k_begin + piece, K);
    const int steps = (k_end - k_begin + FT_K - 1) / FT_K;
    // this thread's outputs: rows m_lane + 16 i + {0 .. 3}, features n_lane + 32 j + {0 .. 3}
    const int m_lane = (warp & 1) * 32 + 4 * (lane >> 3), n_lane = (warp >> 1) * 64 + 4 * (lane & 7);

    // this thread brings k = col .. col + 3 of rows row + 32 i
    const int col = 4 * (tid & 3), row = tid >> 2;
    float4 next_a[FT_M / 32], next_w[FT_N / 32];
    auto fetch = [&](int step) {
        const int k = k_begin + step * FT_K + col;
        const bool k_in = k < k_end;                             // K and the pieces are multiples of 4
        const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < FT_M / 32; ++i) {
            const int m = m0 + row + 32 * i;
            next_a[i] = k_in && m < M ? *reinterpret_cast<const float4*>(A + (size_t)m * lda + k) : none;
        }
#pragma unroll
        for (int i = 0; i < FT_N / 32; ++i) {
            const int n = n0 + row + 32 * i;
            next_w[i] = k_in && n < N ? *reinterpret_cast<const float4*>(W + (size_t)n * ldw + k) : none;
        }
    };
    // rows of the upper eight k are moved by half a bank group: the four k that a warp writes at once then fall on
    // different banks
    const int turn = (col >> 3) & 1;
    auto put = [&](int step) {
        float* a = smem + (step & 1) * FT_BUFFER;
        float* w = a + FT_K * FT_LDA;
#pragma unroll
        for (int i = 0; i < FT_M / 32; ++i) {
            const float v[4] = {next_a[i].x, next_a[i].y, next_a[i].z, next_a[i].w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
                a[(col + e) * FT_LDA + ((row + 32 * i) ^ (8 * turn))] = v[e];
        }
#pragma unroll
        for (int i = 0; i < FT_N / 32; ++i) {
            const float v[4] = {next_w[i].x, next_w[i].y, next_w[i].z, next_w[i].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) w[(col + e) * FT_LDW + ((row + 32 * i) ^ (8 * turn))] = v[e];
        }
    };
    pair_t acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    if (steps > 0) {
        fetch(0);
        put(0);
    }
    for (int s = 0; s < steps; ++s) {
        __syncthreads();                              // step s is in place, and everyone is done with step s - 1
        if (s + 1 < steps) fetch(s + 1);
        const float* a = smem + (s & 1) * FT_BUFFER;
        const float* w = a + FT_K * FT_LDA;
#pragma unroll
        for (int k = 0; k < FT_K; ++k) {
            const int flip = k >> 3;
            pair_t av[8], wv[4];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float4 v = *reinterpret_cast<const float4*>(a + k * FT_LDA + ((m_lane + 16 * i) ^ (8 * flip)));
                av[4 * i] = both(v.x);
                av[4 * i + 1] = both(v.y);
                av[4 * i + 2] = both(v.z);
                av[4 * i + 3] = both(v.w);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(w + k * FT_LDW + ((n_lane + 32 * j) ^ (8 * flip)));
                wv[2 * j] = v.x;
                wv[2 * j + 1] = v.y;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) fma_pair(acc[i][j], av[i], wv[j]);
        }
        if (s + 1 < steps) put(s + 1);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
            *reinterpret_cast<ulonglong2*>(smem + (m_lane + 16 * (i >> 2) + (i & 3)) * FT_OUT_LD + n_lane + 32 * j) =
                make_ulonglong2(acc[i][2 * j], acc[i][2 * j + 1]);
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const float* part[F32_PIECES];
#pragma unroll
    for (int p = 0; p < F32_PIECES; ++p) part[p] = cluster.map_shared_rank(smem, p);
    constexpr int QUARTER = FT_M / F32_PIECES;
    for (int i = tid; i < QUARTER * FT_N; i += FT_THREADS) {
        const int r = rank * QUARTER + i / FT_N, f = i % FT_N;
        const int m = m0 + r, n = n0 + f;
        if (m >= M || n >= N) continue;
        const int at = r * FT_OUT_LD + f;
        float v = (part[0][at] + part[1][at]) + (part[2][at] + part[3][at]);
        if (bias) v += bias[n];
        v = mode_activation(v, mode);
        const size_t o = (size_t)m * ldo + n;
        if (mode == MX_MODE_RESIDUAL) v += residual[o];
        out[o] = v;
    }
    cluster.sync();                                   // nobody leaves while its sums are being read
}

int f32_sm_count() {
    static int count = 0;
    if (count == 0) {
        int device = 0;
        cudaGetDevice(&device);
        cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device);
        if (count <= 0) count = 148;
    }
    return count;
}

template <int MB>
cudaError_t launch_rows(const float* A, int lda, const float* W, int ldw, const float* bias, const float* residual,
                        float* out, int ldo, int M, int N, int K, int mode, cudaStream_t stream) {
    constexpr size_t smem = sizeof(float) * F32_PIECES * FR_STAGES * (FR_ROWS + MB) * FR_K;
    const cudaError_t e = cudaFuncSetAttribute(gemm_f32_rows_kernel<MB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    // as many weight rows a block as deal the matrix out evenly over whole rounds of the SMs
    const int sms = f32_sm_count();
    const int rounds = (N + sms * FR_ROWS - 1) / (sms * FR_ROWS);
    const int rows = max(1, min(FR_ROWS, (N + sms * rounds - 1) / (sms * rounds)));
    return mx_launch_chained(gemm_f32_rows_kernel<MB>, dim3((N + rows - 1) / rows, (M + MB - 1) / MB), dim3(FR_THREADS),
                             smem, stream, A, lda, W, ldw, bias, residual, out, ldo, M, N, K, f32_piece(K), rows, mode);
}

}  // namespace

// Both kernels pay for four pieces of K and for filling their rings or clusters, whatever K is: below these lengths the
// general kernel is the faster one. 2,048 columns, us here against there: 4 rows of 16 k 2.6 and 3.1; 16 of 16, 3.6 and
// 3.2; 32 of 32, 5.4 and 4.1, of 64, 5.1 and 5.6; 389 of 16, 11.3 and 4.2, of 96, 15.2 and 12.6, of 128, 15.4 and 15.9.
// 8,192 columns give the streaming kernel's blocks several rows each: 8 rows of 16 k take 4.6 and 3.3. Between 128 and 192
// the pieces are 64 long and the last block of a cluster has none: 1,024 x 1,024 x 160 takes 22.0 and 17.0.
extern "C" int mx_gemm_f32_pays(int M, int N, int K) {
    if (M > F32_FEW_ROWS) return K >= 192 || (K > 96 && K <= 128);
    const int several = N > 4096 ? 2 : 1;
    return K >= (M <= 8 ? (several > 1 ? 32 : 0) : M <= 16 ? 32 * several : 64 * several);
}

bool mx_gemm_f32_takes(const float* A, int lda, const float* W, int ldw, int M, int N, int K) {
    return mx_gemm_f32_pays(M, N, K) && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
           ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0 && (N + FT_N - 1) / FT_N <= 65535;
}

int mx_gemm_f32(const float* A, int lda, const float* W, int ldw, const float* bias, const float* residual, float* out,
                int ldo, int M, int N, int K, int mode, cudaStream_t stream) {
    cudaError_t e;
    if (M <= 1) e = launch_rows<1>(A, lda, W, ldw, bias, residual, out, ldo, M, N, K, mode, stream);
    else if (M <= 2) e = launch_rows<2>(A, lda, W, ldw, bias, residual, out, ldo, M, N, K, mode, stream);
    else if (M <= 4) e = launch_rows<4>(A, lda, W, ldw, bias, residual, out, ldo, M, N, K, mode, stream);
    else if (M <= 8) e = launch_rows<8>(A, lda, W, ldw, bias, residual, out, ldo, M, N, K, mode, stream);
    else if (M <= F32_FEW_ROWS) e = launch_rows<16>(A, lda, W, ldw, bias, residual, out, ldo, M, N, K, mode, stream);
    else {
        const dim3 grid(F32_PIECES * ((M + FT_M - 1) / FT_M), (N + FT_N - 1) / FT_N);
        gemm_f32_tile_kernel<<<grid, FT_THREADS, 0, stream>>>(A, lda, W, ldw, bias, residual, out, ldo, M, N, K,
                                                              f32_piece(K), mode);
        mx_count_launch();
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        mx_set_error("float gemm: launch failed: %s", cudaGetErrorString(e));
        return (int)e;
    }
    return MX_OK;
}
