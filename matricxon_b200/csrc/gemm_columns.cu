// out[M,N] = epilogue(x[M,K] . W[N,K]^T + bias[N]) for some hundreds of bfloat16 rows: prompts of a step and portions beside
// decoding requests. Pairs of SMs with the weight rows as the rows of tcgen05.mma and the tokens as its columns.
//
// Such a product has few tiles for 148 SMs, and what one SM takes in through TMA (about 53 bytes a cycle) bounds each of them
// more than the tensor cores do. With the tokens as rows their count is cut into steps of 256 or 512 (543 rows are computed
// as 768). As columns they are cut into tiles of any multiple of 16 up to 256 that fills the rounds of the SMs: 543 are three
// tiles of 192. A pair of blocks owns 256 weight rows of a tile (cta_group::2: each block its 128 rows and half of the
// tokens, so 16 KB + 64 bytes a token for 64 of K), a ring of TMA stages feeds it through its tiles without a break, and two
// accumulators let the eight epilogue warps of a block store one tile under the next one's products. Where the result is a
// sum added to the stream in place, K is also shared out: every part leaves its sums in scratch memory, and whoever reads the
// stream next (the norm: mx_layernorm_sum, mx_rmsnorm_pending), or else a kernel of its own, adds them in order, so a product
// repeats bit by bit. Product and norm, us, against adding to memory in the order in which the parts end, which does not
// repeat: 367 x 3,072 x 12,288 35.2 and 33.1, 512 rows 40.6 and 39.3, 1,024 x 1,024 x 6,144 21.2 and 21.2, 2,048 rows 30.0 and
// 30.7 (35 to 44 with K in one piece); parts that meet in the shared memory of clusters of four or six blocks take 3 to 7 us
// more, since 66 pairs run at a time then instead of 74.
// The reference runs these products through nn.Linear (app/architectures/qwen_layers.py:50-53,
// app/architectures/starcoder2_layers.py:19-23).
#include <stdlib.h>

#include "common.cuh"
#include "tcgen05_helpers.cuh"

namespace {

constexpr int CL_ROWS = 256, CL_TOKENS = 256;           // weight rows of a pair's tile; tokens of it at most
constexpr int CL_EPI_WARPS = 8, CL_THREADS = 32 * (CL_EPI_WARPS + 2);
constexpr int CL_MAX_STAGES = 8, CL_SMEM = 220 * 1024;
constexpr int CL_MAX_SPLITS = MX_SUM_PARTS;             // parts of K

struct ClPlan {
    int tokens, token_tiles;    // a multiple of 16; how many such tiles
    int splits;                 // parts of K
    int stages;
};

struct ClShared {
    unsigned long long full[CL_MAX_STAGES];             // used in the first block of the pair
    unsigned long long empty[CL_MAX_STAGES];            // in each block
    unsigned long long acc_full[2];                     // in each block
    unsigned long long acc_empty[2];                    // used in the first block
    unsigned tmem_base;
};

__device__ __forceinline__ unsigned cl_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cl_shared_of(const void* ptr, unsigned rank) {
    unsigned d;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(d) : "r"(smem_u32(ptr)), "r"(rank));
    return d;
}
__device__ __forceinline__ void cl_cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cl_load(void* smem_dst, const CUtensorMap* map, int x, int y, unsigned bar_cluster_addr) {
    asm volatile(
        "{\n.reg .pred q;\n"
        "elect.sync _|q, 0xffffffff;\n"
        "@q cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
        "[%4];\n}\n" ::"r"(smem_u32(smem_dst)),
        "l"(map), "r"(x), "r"(y), "r"(bar_cluster_addr)
        : "memory");
}
__device__ __forceinline__ void cl_mma(unsigned tmem_acc, unsigned long long adesc, unsigned long long bdesc, unsigned idesc,
                                       bool accumulate) {
    asm volatile(
        "{\n.reg .pred p, q;\n"
        "elect.sync _|q, 0xffffffff;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_acc),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"((unsigned)accumulate)
        : "memory");
}
// Arrives, once the products issued so far are done, on the barrier at this offset in both blocks.
__device__ __forceinline__ void cl_commit(unsigned long long* bar) {
    asm volatile(
        "{\n.reg .pred q;\n"
        "elect.sync _|q, 0xffffffff;\n"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n}\n" ::"r"(
            smem_u32(bar)),
        "h"((unsigned short)3)
        : "memory");
}
__device__ __forceinline__ void cl_arrive(unsigned bar_cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(bar_cluster_addr) : "memory");
}

template <bool F32>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(CL_THREADS, 1)
gemm_columns_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                    const float* __restrict__ bias, const float* residual, void* out, int ldo, int M, int N, int K, int mode,
                    const ClPlan plan, float* parts, int ldp, int* status) {
    extern __shared__ unsigned char cl_smem_raw[];
    unsigned char* ring = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(cl_smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ ClShared sh;
    const unsigned w_bytes = 128 * TC_BK * 2, stage_bytes = w_bytes + (unsigned)(plan.tokens / 2) * TC_BK * 2;
    const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
    const unsigned rank = cl_rank();
    const int pair = (int)(blockIdx.x >> 1), n_pairs = (int)(gridDim.x >> 1);
    const int slices = (K + TC_BK - 1) / TC_BK, per = (slices + plan.splits - 1) / plan.splits;
    const int weight_tiles = (N + CL_ROWS - 1) / CL_ROWS, items = weight_tiles * plan.token_tiles * plan.splits;
    // item -> token tile (fastest: a weight tile's tokens run at a time and read it from HBM once), part of K, weight tile
    auto place = [&](int item, int& m0, int& n0, int& first, int& count) {
        m0 = (item % plan.token_tiles) * plan.tokens;
        item /= plan.token_tiles;
        const int part = item % plan.splits;
        n0 = (item / plan.splits) * CL_ROWS;
        first = part * per;
        count = min(per, slices - first);
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < plan.stages; ++s) {
            tc_mbar_init(&sh.full[s], 1);
            tc_mbar_init(&sh.empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc_mbar_init(&sh.acc_full[b], 1);
            tc_mbar_init(&sh.acc_empty[b], 2 * CL_EPI_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == CL_EPI_WARPS + 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&sh.tmem_base)), "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    cl_cluster_barrier();                               // the peer's barriers exist from here on
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const unsigned tmem_base = sh.tmem_base;

    if (warp == CL_EPI_WARPS) {
        // ---------------- producer (in both blocks): the whole warp walks, one elected lane issues
        pdl_wait();
        int s = 0, it = 0;
        unsigned turn = 1;
        bool alive = true;
        for (int item = pair; item < items && alive; item += n_pairs) {
            int m0, n0, first, count;
            place(item, m0, n0, first, count);
            const int w_row = n0 + 128 * (int)rank, x_row = m0 + plan.tokens / 2 * (int)rank;
            for (int i = 0; i < count; ++i, ++it) {
                alive = tc_mbar_wait_warp(&sh.empty[s], turn, status);
                if (!alive) break;
                if (rank == 0) tc_mbar_expect_tx_elect(&sh.full[s], 2 * stage_bytes);
                const unsigned bar = cl_shared_of(&sh.full[s], 0);
                unsigned char* to = ring + (size_t)s * stage_bytes;
                cl_load(to, &map_w, (first + i) * TC_BK, w_row, bar);
                cl_load(to + w_bytes, &map_x, (first + i) * TC_BK, x_row, bar);
                if (++s == plan.stages) s = 0, turn ^= 1;
            }
        }
        pdl_trigger();
        if (rank == 0)                                  // nothing stays in flight (the products read both blocks' stages)
            for (int j = max(0, it - plan.stages); j < it; ++j)
                if (!tc_mbar_wait_warp(&sh.full[j % plan.stages], (unsigned)(j / plan.stages) & 1, status)) break;
    } else if (warp == CL_EPI_WARPS + 1) {
        // ---------------- MMA issuer of the pair
        if (rank == 0) {
            const unsigned idesc = umma_idesc(CL_ROWS, plan.tokens);
            int s = 0, local = 0;
            unsigned turn = 0;
            bool alive = true;
            for (int item = pair; item < items && alive; item += n_pairs, ++local) {
                int m0, n0, first, count;
                place(item, m0, n0, first, count);
                const int b = local & 1;
                alive = tc_mbar_wait_warp(&sh.acc_empty[b], ((unsigned)(local >> 1) & 1) ^ 1, status);
                if (!alive) break;
                const unsigned acc = tmem_base + (unsigned)(b * CL_TOKENS);
                for (int i = 0; i < count; ++i) {
                    alive = tc_mbar_wait_warp(&sh.full[s], turn, status);
                    if (!alive) break;
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const unsigned long long w = umma_desc(ring + (size_t)s * stage_bytes);
                    const unsigned long long x = umma_desc(ring + (size_t)s * stage_bytes + w_bytes);
#pragma unroll
                    for (int k = 0; k < TC_BK / 16; ++k) cl_mma(acc, w + 2 * k, x + 2 * k, idesc, (i | k) != 0);
                    cl_commit(&sh.empty[s]);
                    if (++s == plan.stages) s = 0, turn ^= 1;
                }
                if (alive) cl_commit(&sh.acc_full[b]);
            }
        }
    } else {
        // ---------------- epilogue: warp w has weight rows 32 (w % 4) .. of this block's 128 and half w / 4 of the tokens
        const int quarter = warp & 3, half = plan.tokens / 2, column = (warp >> 2) * half;
        pdl_wait();                                     // the residual is somebody's output
        residual = after_wait(residual);
        bias = after_wait(bias);
        int local = 0;
        for (int item = pair; item < items; item += n_pairs, ++local) {
            int m0, n0, first, count;
            place(item, m0, n0, first, count);
            const int b = local & 1, n = n0 + 128 * (int)rank + 32 * quarter + lane;
            const bool mine = n < N, shared = F32 && plan.splits > 1;       // a part of K: its sums alone, to scratch memory
            const float bias_here = mine && bias != nullptr && !shared ? bias[n] : 0.f;
            const int tokens = min(half, M - m0 - column);                  // of this warp
            // sixteen tokens at a time; what a sum in place is added to sets out sixteen tokens ahead
            const float* old = F32 && mode == MX_MODE_RESIDUAL && !shared && mine ? residual + (size_t)(m0 + column) * ldo + n : nullptr;
            float before[16];
            auto fetch = [&](int c) {
#pragma unroll
                for (int j = 0; j < 16; ++j) before[j] = old != nullptr && c + j < tokens ? __ldcg(old + (size_t)(c + j) * ldo) : 0.f;
            };
            if constexpr (F32) fetch(0);
            if (!tc_mbar_wait_warp(&sh.acc_full[b], (unsigned)(local >> 1) & 1, status)) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const unsigned from = tmem_base + (unsigned)(b * CL_TOKENS + column) + ((unsigned)(32 * quarter) << 16);
            float* const to_f32 = shared ? parts + (size_t)(first / per) * M * ldp : reinterpret_cast<float*>(out);
            const int stride = shared ? ldp : ldo;
            for (int c = 0; c < tokens; c += 16) {
                unsigned r[16];
                __syncwarp();                           // lanes beyond N have gone past the stores
                tmem_load16(from + (unsigned)c, r);
                const size_t o = (size_t)(m0 + column + c) * stride + n;
                if constexpr (F32) {
                    float* to = to_f32 + o;
                    float sum[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) sum[j] = __uint_as_float(r[j]) + bias_here + before[j];
                    fetch(c + 16);
                    if (!mine) continue;
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (c + j >= tokens) break;
                        to[(size_t)j * stride] = sum[j];
                    }
                } else {
                    if (!mine) continue;
                    __nv_bfloat16* to = reinterpret_cast<__nv_bfloat16*>(out) + o;
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (c + j < tokens)
                            to[(size_t)j * ldo] = __float2bfloat16_rn(mode_activation_fast(__uint_as_float(r[j]) + bias_here, mode));
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) cl_arrive(cl_shared_of(&sh.acc_empty[b], 0));
        }
    }
    // ---------------- teardown: neither block leaves while the other may still touch its memory
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    cl_cluster_barrier();
    if (warp == CL_EPI_WARPS + 1) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512) : "memory");
    }
}

// Pairs of SMs that run at a time (0: the kernel cannot run), looked up by the first call while others wait for it.
int cl_pairs() {
    static const int count = [] {
        int clusters = 0;
        if (cudaFuncSetAttribute(gemm_columns_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, CL_SMEM) == cudaSuccess &&
            cudaFuncSetAttribute(gemm_columns_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, CL_SMEM) == cudaSuccess) {
            int device = 0, sms = 0;
            cudaGetDevice(&device);
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
            cudaLaunchConfig_t config = {};
            config.gridDim = dim3(2 * max(1, sms / 2));
            config.blockDim = dim3(CL_THREADS);
            config.dynamicSmemBytes = CL_SMEM;
            if (cudaOccupancyMaxActiveClusters(&clusters, gemm_columns_kernel<true>, &config) != cudaSuccess) clusters = 0;
        }
        cudaGetLastError();
        return clusters;
    }();
    return count;
}

// Tiles, parts of K and the cycles that they take: a slice of 64 of K takes a pair the longer of its products (2 cycles a
// token) and its loads (53 bytes a cycle and SM); an item costs the turn from one accumulator to the next, the launch its
// start and the last item's stores; the sums of a part are 4 bytes a result to write and to read again, and less of an item's
// end is hidden (480 x 6,144 x 24,576 in three parts 117 us, in one 110; 2,048 x 1,024 x 6,144 in two 30, in one 35).
double cl_plan(int M, int N, int K, bool may_split, int pairs, ClPlan* best) {
    double best_cost = -1.0;
    const int weight_tiles = (N + CL_ROWS - 1) / CL_ROWS, slices = (K + TC_BK - 1) / TC_BK;
    const int least = (M + CL_TOKENS - 1) / CL_TOKENS;
    for (int tiles = least; tiles <= least + 4; ++tiles) {
        const int tokens = ((M + tiles - 1) / tiles + 15) / 16 * 16;
        if (tiles > least && tokens * (tiles - 1) >= M) continue;
        const double slice = max(2.0 * tokens, (16384.0 + 64.0 * tokens) / 53.0);
        for (int splits = 1; splits <= (may_split ? CL_MAX_SPLITS : 1); ++splits) {
            const int per = (slices + splits - 1) / splits;
            if (splits > 1 && (per < 8 || (splits - 1) * per >= slices)) continue;
            const long long rounds = ((long long)weight_tiles * tiles * splits + pairs - 1) / pairs;
            double cost = rounds * (per * slice + (splits > 1 ? 2500.0 : 500.0)) + 4000.0 + 20.0 * tokens;
            if (splits > 1) cost += 4.0 * M * N * (splits + 1.0) / 1400.0;
            if (best_cost < 0.0 || cost < best_cost) {
                best_cost = cost;
                best->tokens = tokens;
                best->token_tiles = (M + tokens - 1) / tokens;
                best->splits = splits;
            }
        }
    }
    best->stages = min(CL_MAX_STAGES, (CL_SMEM - 1024) / (128 * TC_BK * 2 + best->tokens / 2 * TC_BK * 2));
    return best_cost;
}

}  // namespace

// Whether a product of more than 256 rows that fills the SMs is better off here than on the kernels with 128, 256 or 512
// tokens to a tile (gemm_tcgen05.cu). Us there against here, weights from HBM: with GELU 367 x 12,288 x 3,072 36.1 and 27.8,
// 512 38.9 and 33.2, 543 x 18,432 x 4,608 104 and 72, 1,023 x 12,288 x 3,072 75.7 and 60.0, 1,777 x 16,384 x 2,048 106 and 88;
// 8,192 x 12,288 x 3,072 459 and 385; added to the stream, with the norm that reads it, 367 x 3,072 x 12,288 43.7 and 34.8, 512
// 42.0 and 40.6, 633 x 2,048 x 8,192 37.5 and 29.4, 543 x 4,608 x 18,432 99 and 72, 1,024 x 1,024 x 6,144 26.3 and 21.2, 1,400 x
// 3,072 x 3,072 39.9 and 32.4, 2,048 x 1,024 x 6,144 54.6 and 30.0 (in two parts of K; in one 35), 2,048 x 2,048 x 8,192 76 and
// 57. From 2,048 rows on 512-row tiles are as good where K is long and the result narrow: 2,048 x 4,608 x 18,432 221 and 232, 2,500 x 3,072 x 12,288
// 127 and 134, 4,096 x 2,048 x 8,192 96 and 100, 8,192 x 1,024 x 6,144 75 and 84.
extern "C" int mx_gemm_columns_pays(int M, int N, int K) {
    return M > 256 && !(M >= 2048 && N < K && K >= (M >= 8192 ? 6144 : M >= 4096 ? 8192 : 12288));
}

namespace {

// The plan of a product; `in_place`: its result is a sum added to the stream in place. MATRICXON_GEMM_SPLIT_K=0 keeps every
// tile's K in one pair.
ClPlan cl_plan_of(int M, int N, int K, bool in_place, int pairs) {
    static const bool split_allowed = [] {
        const char* env = getenv("MATRICXON_GEMM_SPLIT_K");
        return env == nullptr || env[0] != '0';
    }();
    ClPlan plan = {};
    cl_plan(M, N, K, in_place && split_allowed, pairs, &plan);
    return plan;
}

}  // namespace

// Parts of K that a product added to the stream in place is cut into (1: none), each [M][N rounded up to 4] floats of scratch.
extern "C" int mx_gemm_columns_parts(int M, int N, int K) {
    const int pairs = M > 0 && N > 0 && K > 0 ? cl_pairs() : 0;
    return pairs > 0 ? cl_plan_of(M, N, K, true, pairs).splits : 1;
}

// `parts`: the scratch memory of a product that is added to the stream in place and cut into parts of K; null otherwise. With
// `finish` 0 the sums stay there (out and bias are not touched) for mx_layernorm_sum or mx_add_parts.
extern "C" int mx_gemm_columns(const void* x, const void* W, const float* bias, const float* residual, void* out, int out_dtype,
                               float* parts, int finish, int M, int N, int K, int ldx, int ldw, int ldo, int mode, int* status,
                               cudaStream_t stream) {
    if (M <= 0 || N <= 0) return MX_OK;
    if (K <= 0 || K % 8 != 0) MX_REFUSE("column gemm: K = %d is not a positive multiple of 8", K);
    if (ldx % 8 != 0 || ldw % 8 != 0) MX_REFUSE("column gemm: row strides %d, %d are not multiples of 8", ldx, ldw);
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(W)) & 15)
        MX_REFUSE("column gemm: operands must start on 16-byte boundaries");
    if (mode < 0 || mode > MX_MODE_LAST) MX_REFUSE("column gemm: unknown epilogue mode %d", mode);
    if (mode == MX_MODE_RESIDUAL && residual == nullptr) MX_REFUSE("column gemm: residual mode without a residual");
    if (mx_mode_is_float(mode) != (out_dtype == MX_DTYPE_F32))
        MX_REFUSE("column gemm: epilogue mode %d does not write dtype %d", mode, out_dtype);
    if (status == nullptr) MX_REFUSE("column gemm: a status word is needed for its bounded waits");
    const int pairs = cl_pairs();
    if (pairs <= 0) MX_REFUSE("column gemm: pairs of SMs cannot run %d bytes of shared memory", CL_SMEM);
    const ClPlan plan = cl_plan_of(M, N, K, mode == MX_MODE_RESIDUAL && residual == out, pairs);
    if (plan.splits > 1 && (parts == nullptr || (reinterpret_cast<uintptr_t>(parts) & 15)))
        MX_REFUSE("column gemm: %d parts of K need scratch on a 16-byte boundary", plan.splits);
    CUtensorMap map_w, map_x;
    int rc = mx_tensor_map_2d(&map_w, W, N, K, ldw, 128);
    if (rc != MX_OK) return rc;
    rc = mx_tensor_map_2d(&map_x, x, M, K, ldx, plan.tokens / 2);
    if (rc != MX_OK) return rc;
    const long long items = (long long)((N + CL_ROWS - 1) / CL_ROWS) * plan.token_tiles * plan.splits;
    if (items > 0x3fffffffLL) MX_REFUSE("column gemm: %d x %d is beyond this kernel's grid", M, N);
    const int grid = 2 * (int)(items < pairs ? items : pairs);
    const size_t smem = 1024 + (size_t)plan.stages * (128 + plan.tokens / 2) * TC_BK * 2;
    const int ldp = (N + 3) / 4 * 4;
    const cudaError_t e = out_dtype == MX_DTYPE_F32
                              ? mx_launch_chained(gemm_columns_kernel<true>, dim3(grid), dim3(CL_THREADS), smem, stream, map_w,
                                                  map_x, bias, residual, out, ldo, M, N, K, mode, plan, parts, ldp, status)
                              : mx_launch_chained(gemm_columns_kernel<false>, dim3(grid), dim3(CL_THREADS), smem, stream, map_w,
                                                  map_x, bias, residual, out, ldo, M, N, K, mode, plan, parts, ldp, status);
    if (e != cudaSuccess) {
        mx_set_error("column gemm: launch failed: %s", cudaGetErrorString(e));
        return (int)e;
    }
    if (plan.splits > 1 && finish)
        return mx_add_parts(parts, ldp, plan.splits, bias, reinterpret_cast<float*>(out), ldo, M, N, stream);
    return MX_OK;
}
