// out[M,N] = epilogue(A[M,K] . W[N,K]^T + bias[N]), all float, on the tensor cores: products of the 32-bit path.
//
// A float of 2^-110 or more is the sum of three bfloat16 numbers, exactly: x = h + m + l with h = bf16(x), m = bf16(x - h),
// l = x - h - m (8 + 8 + 8 bits of significand and the signs); of smaller ones what lies below bfloat16's smallest number,
// 2^-133, is lost. Of the nine products of two such sums the six largest are formed, h h, h m, m h, m m, h l, l h; what is left
// out is at most 2^-24 of a term (|m| reaches 2^-8 of a float, |l| 2^-17). The tensor cores add in float but cut sums off
// instead of rounding them, so an accumulator only ever holds 32 values of k, the small products first and h h last; it is
// then added to float registers, rounded to nearest (96 additions for K = 3,072, where the FP32 cores' chains make 768 to a
// piece).
// Root mean square error against 64 bits, of the result's, here and on the FP32 cores, K = 512 / 3,072 / 12,288:
//   operands of both signs        8.1e-8 and 2.1e-7    1.1e-7 and 5.0e-7    1.5e-7 and 9.9e-7
//   of one sign (|normal|)        6.3e-8 and 8.5e-8    7.2e-8 and 2.1e-7    7.9e-8 and 4.1e-7
//   relu^2 times |normal|         7.0e-8 and 7.3e-8    7.5e-8 and 1.5e-7    8.2e-8 and 3.1e-7
//   one term 10,000 x the others  9.3e-8 and 2.1e-7    1.1e-7 and 4.7e-7    1.5e-7 and 9.7e-7
//   one value in fifty not zero   6.8e-8 and 5.3e-8    8.8e-8 and 8.3e-8    1.2e-7 and 1.5e-7
//   one value alone               4.5e-8 and 2.6e-8    4.5e-8 and 2.5e-8    4.6e-8 and 2.5e-8
// So sums of many terms come closer, of one sign too; rows of few terms do not, since the FP32 cores then round little.
// The order of a row's sums, and the unit that forms them, follow the number of rows: FP32 cores up to two, mma.sync up to
// eight, tcgen05 above, with shares of K that depend on the tiles. The same row in another batch differs in its last bits, as
// in bfloat16; gemm_backend "simt" keeps every product on the FP32 cores, where it does not.
// A result that is not finite (an operand that is not, an overflow on the way, a float above bfloat16's largest) is formed
// again from the operands by plain multiply-adds, which decide what it is, unless its row of A holds a NaN, which decides it:
// a warp looks at the row first (one such row among 4 of 3,072 x 12,288 took 558 us as chains and takes 40, the product 40;
// 389 of 389 rows of 12,288 x 3,072 61,200 and 183, the product 169). An infinity or an overflow in a row still costs the
// chains (245 us at 4 rows of 12,288, 501 at 389 of 3,072). The reference runs these products through
// nn.Linear (app/architectures/qwen_layers.py:50-53, app/architectures/starcoder2_layers.py:19-23).
//
// Weight rows are the tensor cores' 128 rows, tokens the columns (up to 208). The weights come as floats by TMA, since a
// split copy would be 1.5 times the bytes of a matrix that is read once; two groups of four warps split them, a stage each
// in turn and a row a thread, into tensor memory, from where the products take them (through shared memory, whose 128 bytes
// a cycle then bound products of few tokens, a stage took 1,000 cycles). Up to 64 tokens of a tile are split
// beside them; more are split once, by a kernel of their own, and come by TMA as parts. Eight more warps add up the
// accumulators, of which there are two to four. K is dealt out to the blocks of a cluster where tiles alone leave SMs idle;
// each block finishes a share of the tokens from all sums, in the order of K. 389 rows x 12,288 x 3,072 and 3,072 x 12,288 take
// 170 and 166 us (the FP32 cores 701 and 790), 1,024 rows 362 and 352 (1,589 and 1,625), 64 rows 69 and 61 (136 and 298): 172 to
// 220 TFLOP/s of the 278 that six products leave of the measured rate. What is left is a tile's start and end, about 13,000
// cycles beside 96 stages of 1,300. With splitting and adding in the same eight warps a stage took 1,600 to 1,850 cycles
// whatever its size, with one issuer 5 % more than with two.
#include <cooperative_groups.h>

#include "common.cuh"
#include "gemm_f32.cuh"
#include "tcgen05_helpers.cuh"

namespace {

namespace cg = cooperative_groups;

// ------------------------------------------------------------------------------------------- three parts of a float
__device__ __forceinline__ unsigned pack_bf16(float low, float high) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(low, high);
    return *reinterpret_cast<const unsigned*>(&p);
}
__device__ __forceinline__ float low_of(unsigned p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float high_of(unsigned p) { return __uint_as_float(p & 0xffff0000u); }

__device__ __forceinline__ void split_pair(float x, float y, unsigned& h, unsigned& m, unsigned& l) {
    h = pack_bf16(x, y);
    x -= low_of(h);
    y -= high_of(h);
    m = pack_bf16(x, y);
    x -= low_of(m);
    y -= high_of(m);
    l = pack_bf16(x, y);
}
__device__ __forceinline__ void split_eight(const float4& u, const float4& v, uint4& h, uint4& m, uint4& l) {
    split_pair(u.x, u.y, h.x, m.x, l.x);
    split_pair(u.z, u.w, h.y, m.y, l.y);
    split_pair(v.x, v.y, h.z, m.z, l.z);
    split_pair(v.z, v.w, h.w, m.w, l.w);
}

// parts [3][M][ldp] of A [M][K]; columns from K to ldp (a multiple of 8) are zeros. A thread splits eight values.
constexpr int FS_SPLIT_THREADS = 256;
__global__ void __launch_bounds__(FS_SPLIT_THREADS)
f32_split_kernel(const float* __restrict__ A, int lda, __nv_bfloat16* __restrict__ parts, int ldp, int M, int K) {
    pdl_trigger();
    pdl_wait();
    A = after_wait(A);
    const long long eighths = ldp / 8, i = (long long)blockIdx.x * FS_SPLIT_THREADS + threadIdx.x;
    if (i < eighths * M) {
        const int row = (int)(i / eighths), k = (int)(i - row * eighths) * 8;
        const float* a = A + (size_t)row * lda + k;
        const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 u = *reinterpret_cast<const float4*>(a);                          // K is a multiple of 4
        const float4 v = k + 4 < K ? *reinterpret_cast<const float4*>(a + 4) : none;
        uint4 h, m, l;
        split_eight(u, v, h, m, l);
        const size_t at = (size_t)row * ldp + k, plane = (size_t)M * ldp;
        *reinterpret_cast<uint4*>(parts + at) = h;
        *reinterpret_cast<uint4*>(parts + plane + at) = m;
        *reinterpret_cast<uint4*>(parts + 2 * plane + at) = l;
    }
}

// ------------------------------------------------------------------------------------------- the product
constexpr int FS_K = 32;                                // k of a stage: 128 bytes of float, 64 bytes of each part
constexpr int FS_ROWS = 128;                            // weight rows of a tile
constexpr int FS_ADDERS = 8, FS_GROUP = 4, FS_GROUPS = 2;         // warps: adding up; a group that splits, and how many
constexpr int FS_THREADS = 32 * (FS_ADDERS + FS_GROUPS * FS_GROUP + 4);
constexpr int FS_MAX_TOKENS = 208, FS_INLINE_TOKENS = 64;
constexpr int FS_MAX_STAGES = 8;
constexpr unsigned FS_RAW_BYTES = FS_ROWS * FS_K * 4;   // a stage of weights as they lie in memory
constexpr int FS_A_COLUMNS = 3 * FS_K / 2;              // of tensor memory for the parts of a stage of weights
constexpr int FS_TMEM = 512;
constexpr int FS_SMEM = 224 * 1024;
// Registers a thread, by warpgroup: 640 threads are launched with 96 each, 61,440 together, and share them anew as
// 8 warps x 168 + 8 x 56 + 4 x 32.
constexpr int FS_ADDER_REGS = 168, FS_SPLIT_REGS = 56, FS_ISSUE_REGS = 32;

struct FsPlan {
    int tokens;                 // of a tile: a multiple of 16
    int token_tiles;
    int splits;                 // blocks of a cluster
    int inlined;                // tokens are split in this kernel
    int accumulators;           // of `tokens` columns of tensor memory
    int raw_stages, part_stages, x_stages;
    unsigned raw_bytes;         // of a stage, tokens that are split here included
};

struct FsShared {
    unsigned long long raw_full[FS_MAX_STAGES], raw_empty[FS_MAX_STAGES];
    unsigned long long x_full[FS_MAX_STAGES], x_empty[FS_MAX_STAGES];
    unsigned long long part_full[FS_MAX_STAGES], part_empty[FS_MAX_STAGES];
    unsigned long long acc_full[FS_MAX_STAGES], acc_empty[FS_MAX_STAGES];
    unsigned tmem_base;
};

// K-major operand in rows of 64 bytes, 64-byte swizzle, groups of eight rows 512 bytes apart
__device__ __forceinline__ unsigned long long umma_desc_64(const void* smem_tile) {
    unsigned long long desc = 0;
    desc |= (unsigned long long)((smem_u32(smem_tile) & 0x3FFFF) >> 4);
    desc |= (unsigned long long)1 << 16;
    desc |= (unsigned long long)(512 >> 4) << 32;
    desc |= (unsigned long long)1 << 46;
    desc |= (unsigned long long)4 << 61;                // SWIZZLE_64B
    return desc;
}

__device__ __forceinline__ void tmem_load32(unsigned taddr, unsigned (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

__device__ __forceinline__ void tmem_store8(unsigned taddr, const unsigned (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

// A from tensor memory: lane r holds row r, a column two values of k.
__device__ __forceinline__ void umma_bf16_ts_elect(unsigned tmem_acc, unsigned tmem_a, unsigned long long bdesc, unsigned idesc,
                                                   bool accumulate) {
    asm volatile(
        "{\n.reg .pred p, q;\n"
        "elect.sync _|q, 0xffffffff;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_acc),
        "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"((unsigned)accumulate)
        : "memory");
}

// ---- results that are not finite
// Whether a row of A holds a NaN (its results are then NaN): a whole warp looks at it.
__device__ __noinline__ bool row_has_nan(const float* a, int K) {
    const int lane = threadIdx.x & 31;
    bool found = false;
    for (int k0 = 0; k0 < K; k0 += 16 * 32) {
        float4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + 4 * (i * 32 + lane);
            v[i] = k < K ? *reinterpret_cast<const float4*>(a + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) found = found || isnan(v[i].x) || isnan(v[i].y) || isnan(v[i].z) || isnan(v[i].w);
        if (__any_sync(0xffffffffu, found)) return true;
    }
    return false;
}

// What the FP32 cores give for one result, in the order of gemm_simt.cu: its four chains side by side, 16 bytes at a time.
__device__ __noinline__ float plain_product(const float* a, const float* w, int K) {
    const int piece = f32_piece(K);                     // a multiple of 32, as K is one of 4
    float total[F32_PIECES] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
    for (int k = 0; k < piece; k += 4) {
        float4 x[F32_PIECES], y[F32_PIECES];
#pragma unroll
        for (int i = 0; i < F32_PIECES; ++i) {
            const bool in = i * piece + k < K;
            x[i] = in ? *reinterpret_cast<const float4*>(a + i * piece + k) : make_float4(0.f, 0.f, 0.f, 0.f);
            y[i] = in ? *reinterpret_cast<const float4*>(w + i * piece + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < F32_PIECES; ++i)
            total[i] = fmaf(x[i].w, y[i].w, fmaf(x[i].z, y[i].z, fmaf(x[i].y, y[i].y, fmaf(x[i].x, y[i].x, total[i]))));
    }
    return (total[0] + total[1]) + (total[2] + total[3]);
}

// Splits eight k (chunk c of four) of a token: rows of 128 bytes of floats with their 16-byte chunks at c ^ (row & 7), rows
// of 64 bytes of each part with theirs at c ^ ((row >> 1) & 3).
__device__ __forceinline__ void split_token(const float4* from, unsigned char* to, unsigned part, int row, int c) {
    const float4 u = from[8 * row + ((2 * c) ^ (row & 7))];
    const float4 v = from[8 * row + ((2 * c + 1) ^ (row & 7))];
    uint4 h, m, l;
    split_eight(u, v, h, m, l);
    to += 64 * row + 16 * (c ^ ((row >> 1) & 3));
    *reinterpret_cast<uint4*>(to) = h;
    *reinterpret_cast<uint4*>(to + part) = m;
    *reinterpret_cast<uint4*>(to + 2 * part) = l;
}

// All threads of the cluster's blocks, warp by warp and not at one place: roles that have registers of their own end here.
__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

__global__ void __launch_bounds__(FS_THREADS, 1)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                      const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                      const float* __restrict__ bias, const float* residual, float* out, int ldo, int M, int N, int K,
                      int mode, const FsPlan plan, int* status) {
    constexpr int NH = (FS_MAX_TOKENS / 2 + 31) / 32 * 32;             // columns a thread adds up at most
    extern __shared__ unsigned char fs_smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(fs_smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* raw = smem;
    unsigned char* xs = raw + plan.raw_stages * plan.raw_bytes;
    const unsigned x_part = (unsigned)plan.tokens * FS_K * 2, x_stage = 3 * x_part;
    // tensor memory: the accumulators, then the stages of weights in parts
    const unsigned a_columns = (unsigned)(plan.accumulators * plan.tokens);
    __shared__ FsShared sh;

    const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x % plan.splits, tile = (int)blockIdx.x / plan.splits;
    const int m0 = (tile % plan.token_tiles) * plan.tokens, n0 = (tile / plan.token_tiles) * FS_ROWS;
    const int all_stages = (K + FS_K - 1) / FS_K;
    const int first = (int)((long long)all_stages * rank / plan.splits);
    const int stages = (int)((long long)all_stages * (rank + 1) / plan.splits) - first;

    if (warp == 0) {
        if (lane < FS_MAX_STAGES) {
            tc_mbar_init(&sh.raw_full[lane], 1);
            tc_mbar_init(&sh.raw_empty[lane], FS_GROUP);
            tc_mbar_init(&sh.x_full[lane], 1);
            tc_mbar_init(&sh.x_empty[lane], 1);
            tc_mbar_init(&sh.part_full[lane], FS_GROUP);
            tc_mbar_init(&sh.part_empty[lane], 1);
            tc_mbar_init(&sh.acc_full[lane], 1);
            tc_mbar_init(&sh.acc_empty[lane], FS_ADDERS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    constexpr int PRODUCER = FS_ADDERS + FS_GROUPS * FS_GROUP, ISSUER = PRODUCER + 1;
    if (warp == ISSUER) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&sh.tmem_base)),
                     "r"(FS_TMEM)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    } else if (warp == PRODUCER) {
        // the weights' first stages towards L2 (they may be the output of the kernel before, whose end is waited for)
        for (int i = 0; i < min(stages, plan.raw_stages); ++i) tma_prefetch_2d_elect(&map_w, (first + i) * FS_K, n0);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const unsigned tmem_base = sh.tmem_base;

    if (warp >= PRODUCER) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(FS_ISSUE_REGS));
        if (warp == PRODUCER) {
            // ---------------- producer: the whole warp walks the loop, one elected lane issues
            pdl_wait();
            int r = 0, x = 0;
            unsigned r_turn = 1, x_turn = 1;            // parities of the waits for room: the first round passes
            for (int i = 0; i < stages; ++i) {
                if (!tc_mbar_wait_warp(&sh.raw_empty[r], r_turn, status)) break;
                tc_mbar_expect_tx_elect(&sh.raw_full[r], plan.raw_bytes);
                unsigned char* to = raw + r * plan.raw_bytes;
                tma_load_2d_elect(to, &map_w, (first + i) * FS_K, n0, &sh.raw_full[r]);
                if (plan.inlined) {
                    tma_load_2d_elect(to + FS_RAW_BYTES, &map_x, (first + i) * FS_K, m0, &sh.raw_full[r]);
                } else {
                    if (!tc_mbar_wait_warp(&sh.x_empty[x], x_turn, status)) break;
                    tc_mbar_expect_tx_elect(&sh.x_full[x], x_stage);
                    for (int p = 0; p < 3; ++p)         // rows beyond M are the next part's: columns that nobody reads
                        tma_load_2d_elect(xs + x * x_stage + p * x_part, &map_x, (first + i) * FS_K, p * M + m0, &sh.x_full[x]);
                    if (++x == plan.x_stages) x = 0, x_turn ^= 1;
                }
                if (++r == plan.raw_stages) r = 0, r_turn ^= 1;
            }
            pdl_trigger();
            // no copy may be in flight when the block ends
            for (int i = max(0, stages - plan.raw_stages); i < stages; ++i)
                if (!tc_mbar_wait_warp(&sh.raw_full[i % plan.raw_stages], (unsigned)(i / plan.raw_stages) & 1, status)) break;
            if (!plan.inlined)
                for (int i = max(0, stages - plan.x_stages); i < stages; ++i)
                    if (!tc_mbar_wait_warp(&sh.x_full[i % plan.x_stages], (unsigned)(i / plan.x_stages) & 1, status)) break;
        } else if (warp < ISSUER + 2) {
            // ---------------- two MMA issuers, a stage each in turn: one's waits (some 100 cycles each, also for what has
            // long arrived) pass while the other's products run
            const unsigned idesc = umma_idesc(FS_ROWS, plan.tokens);
            for (int i = warp - ISSUER; i < stages; i += 2) {
                const int p = i % plan.part_stages, x = plan.inlined ? p : i % plan.x_stages, b = i % plan.accumulators;
                if (!plan.inlined && !tc_mbar_wait_warp(&sh.x_full[x], (unsigned)(i / plan.x_stages) & 1, status)) break;
                if (!tc_mbar_wait_warp(&sh.acc_empty[b], ((unsigned)(i / plan.accumulators) & 1) ^ 1, status)) break;
                if (!tc_mbar_wait_warp(&sh.part_full[p], (unsigned)(i / plan.part_stages) & 1, status)) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const unsigned w = tmem_base + a_columns + p * FS_A_COLUMNS, acc = tmem_base + b * plan.tokens;
                const unsigned long long t = umma_desc_64(xs + x * x_stage);
                // small products first: l h, h l, m m, m h, h m, h h
                constexpr int OF_W[6] = {2, 0, 1, 1, 0, 0}, OF_X[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
                for (int q = 0; q < 6; ++q)
#pragma unroll
                    for (int k = 0; k < FS_K / 16; ++k)  // 16 values are 8 columns, and 32 bytes
                        umma_bf16_ts_elect(acc, w + OF_W[q] * (FS_K / 2) + 8 * k, t + OF_X[q] * (x_part >> 4) + 2 * k, idesc,
                                           (q | k) != 0);
                umma_commit_elect(&sh.part_empty[p]);
                if (!plan.inlined) umma_commit_elect(&sh.x_empty[x]);
                umma_commit_elect(&sh.acc_full[b]);
            }
        }
    } else if (warp >= FS_ADDERS) {
        // ---------------- two groups of four warps split the stages in turn
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(FS_SPLIT_REGS));
        const int group = (warp - FS_ADDERS) / FS_GROUP, thread = (int)threadIdx.x % (32 * FS_GROUP);
        const unsigned a_of_warp = tmem_base + a_columns + ((unsigned)(32 * (warp & 3)) << 16);
        for (int i = group; i < stages; i += FS_GROUPS) {
            const int r = i % plan.raw_stages, p = i % plan.part_stages;
            if (!tc_mbar_wait_warp(&sh.part_empty[p], ((unsigned)(i / plan.part_stages) & 1) ^ 1, status)) break;
            if (!tc_mbar_wait_warp(&sh.raw_full[r], (unsigned)(i / plan.raw_stages) & 1, status)) break;
            const float4* from = reinterpret_cast<const float4*>(raw + r * plan.raw_bytes);
            const unsigned to = a_of_warp + p * FS_A_COLUMNS;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
            for (int half = 0; half < 2; ++half) {      // 16 k of this thread's row: chunk c lies at c ^ (row & 7)
                unsigned h[8], m[8], l[8];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float4 u = from[8 * thread + ((4 * half + c) ^ (thread & 7))];
                    split_pair(u.x, u.y, h[2 * c], m[2 * c], l[2 * c]);
                    split_pair(u.z, u.w, h[2 * c + 1], m[2 * c + 1], l[2 * c + 1]);
                }
                tmem_store8(to + 8 * half, h);
                tmem_store8(to + FS_K / 2 + 8 * half, m);
                tmem_store8(to + FS_K + 8 * half, l);
            }
            if (plan.inlined) {
                for (int t = thread >> 2; t < plan.tokens; t += 32)
                    split_token(from + FS_RAW_BYTES / 16, xs + p * x_stage, x_part, t, thread & 3);
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            }
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                tc_mbar_arrive(&sh.part_full[p]);
                tc_mbar_arrive(&sh.raw_empty[r]);
            }
        }
    } else {
        // ---------------- eight warps add up the accumulators: 32 weight rows and half the tokens each
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(FS_ADDER_REGS));
        const int half = plan.tokens / 2, quarter = warp & 3, column = (warp >> 2) * half;
        float acc[NH];
#pragma unroll
        for (int j = 0; j < NH; ++j) acc[j] = 0.f;
        for (int i = 0; i < stages; ++i) {
            const int b = i % plan.accumulators;
            if (!tc_mbar_wait_warp(&sh.acc_full[b], (unsigned)(i / plan.accumulators) & 1, status)) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const unsigned from = tmem_base + b * plan.tokens + column + ((unsigned)(32 * quarter) << 16);
#pragma unroll
            for (int g = 0; g < NH / 32; ++g) {
                if (32 * g >= half) break;              // columns from `half` on are added up for nobody
                unsigned r[32];
                tmem_load32(from + 32 * g, r);
#pragma unroll
                for (int j = 0; j < 32; ++j) acc[32 * g + j] += __uint_as_float(r[j]);
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) tc_mbar_arrive(&sh.acc_empty[b]);
        }
        // the last product has read all stages: their place holds the sums from here on, [token][128 weight rows]
        float* sums = reinterpret_cast<float*>(smem);
#pragma unroll
        for (int j = 0; j < NH; ++j)
            if (j < half) sums[(column + j) * FS_ROWS + 32 * quarter + lane] = acc[j];
        cluster_sync();                                 // every block's sums are in place
        pdl_wait();                                     // the residual is somebody's output
        A = after_wait(A);
        W = after_wait(W);
        bias = after_wait(bias);
        const int n = n0 + 4 * lane;
        const bool wide = ldo % 4 == 0 && n + 4 <= N && ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(residual)) & 15) == 0;
        float b[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) b[e] = bias != nullptr && n + e < N ? bias[n + e] : 0.f;
        // four tokens at a time, so that their reads are out together (lanes beyond N go along)
        for (int j0 = rank + plan.splits * warp; j0 < plan.tokens; j0 += plan.splits * FS_ADDERS * 4) {
            float4 v[4], res[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                v[t] = res[t] = make_float4(0.f, 0.f, 0.f, 0.f);
                const int j = j0 + t * plan.splits * FS_ADDERS;
                if (mode == MX_MODE_RESIDUAL && j < plan.tokens && m0 + j < M && n < N) {
                    const float* from = residual + (size_t)(m0 + j) * ldo + n;
                    if (wide) {
                        res[t] = *reinterpret_cast<const float4*>(from);
                    } else {
                        res[t].x = from[0];
                        if (n + 1 < N) res[t].y = from[1];
                        if (n + 2 < N) res[t].z = from[2];
                        if (n + 3 < N) res[t].w = from[3];
                    }
                }
            }
            for (int s = 0; s < plan.splits; ++s) {
                const float* peer = cg::this_cluster().map_shared_rank(sums, s);
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const int j = min(j0 + t * plan.splits * FS_ADDERS, plan.tokens - 1);
                    const float4 part = *reinterpret_cast<const float4*>(peer + j * FS_ROWS + 4 * lane);
                    v[t].x += part.x;
                    v[t].y += part.y;
                    v[t].z += part.z;
                    v[t].w += part.w;
                }
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int j = j0 + t * plan.splits * FS_ADDERS, m = m0 + j;
                if (j >= plan.tokens || m >= M) break;
                float y[4] = {v[t].x, v[t].y, v[t].z, v[t].w};
                const float z[4] = {res[t].x, res[t].y, res[t].z, res[t].w};
                const bool finite = n >= N || (isfinite(y[0]) && isfinite(y[1]) && isfinite(y[2]) && isfinite(y[3]));
                if (!__all_sync(0xffffffffu, finite)) {
                    const bool nan = row_has_nan(A + (size_t)m * lda, K);
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (!isfinite(y[e]) && n + e < N)
                            y[e] = nan ? NAN : plain_product(A + (size_t)m * lda, W + (size_t)(n + e) * ldw, K);
                }
                float* to = out + (size_t)m * ldo + n;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    y[e] = mode_activation(y[e] + b[e], mode);
                    if (mode == MX_MODE_RESIDUAL) y[e] += z[e];
                }
                if (wide) {
                    *reinterpret_cast<float4*>(to) = make_float4(y[0], y[1], y[2], y[3]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (n + e < N) to[e] = y[e];
                }
            }
        }
        cluster_sync();                                 // nobody leaves while its sums are being read
    }
    if (warp >= FS_ADDERS) {
        cluster_sync();
        cluster_sync();
    }
    if (warp == ISSUER) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(FS_TMEM) : "memory");
    }
}

// ------------------------------------------------------------------------------------------- up to eight rows
// Decoding: a stream of the weights. A block of eight warps owns 16 weight rows, the rows of mma.sync.m16n8k16, with the
// tokens as its columns; the warps deal out K, 32 values at a time. A lane loads floats of two weight rows (64 bytes of a
// row to a quad) and of a token, splits them where they are and multiplies: nothing passes through shared memory. Three
// pieces are in flight a warp, two blocks an SM.
constexpr int FK_WARPS = 8, FK_THREADS = 32 * FK_WARPS, FK_ROWS = 16, FK_TOKENS = 8, FK_UNROLL = 3;

__device__ __forceinline__ void mma_parts(float (&d)[4], const unsigned (&a)[2][4], const unsigned (&b)[4], int j) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0][2 * j]), "r"(a[1][2 * j]), "r"(a[0][2 * j + 1]), "r"(a[1][2 * j + 1]), "r"(b[2 * j]), "r"(b[2 * j + 1]));
}

__device__ __forceinline__ float4 load_once(const float* p) {
    float4 v;
    asm volatile("ld.global.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}

__global__ void __launch_bounds__(FK_THREADS, 2)
gemm_f32_skinny_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                       const float* __restrict__ bias, const float* residual, float* out, int ldo, int M, int N, int K,
                       int mode) {
    __shared__ float sums[FK_WARPS][FK_TOKENS][FK_ROWS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int n0 = blockIdx.x * FK_ROWS, pieces = (K + 31) / 32;
    const float* w_row[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) w_row[i] = W + (size_t)min(n0 + g + 8 * i, N - 1) * ldw;
    // the weights' first lines set out for L2 while the kernel before this one ends
    for (int u = 0; u < FK_UNROLL; ++u) {
        const int k = 32 * (warp + FK_WARPS * u);
        if (t == 0 && k < K) {
            prefetch_l2(w_row[0] + k);
            prefetch_l2(w_row[1] + k);
        }
    }
    pdl_wait();
    A = after_wait(A);
    W = after_wait(W);
    bias = after_wait(bias);
    const float* x_row = A + (size_t)min(g, M - 1) * lda;
#pragma unroll
    for (int i = 0; i < 2; ++i) w_row[i] = after_wait(w_row[i]);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int first = warp; first < pieces; first += FK_WARPS * FK_UNROLL) {
        float4 w[FK_UNROLL][2][2], x[FK_UNROLL][2];
#pragma unroll
        for (int u = 0; u < FK_UNROLL; ++u)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int k = 32 * (first + FK_WARPS * u) + 16 * e + 4 * t;              // K is a multiple of 4
                const bool in = k < K;
                const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
                w[u][0][e] = in ? load_once(w_row[0] + k) : none;
                w[u][1][e] = in ? load_once(w_row[1] + k) : none;
                x[u][e] = in ? *reinterpret_cast<const float4*>(x_row + k) : none;
            }
#pragma unroll
        for (int u = 0; u < FK_UNROLL; ++u) {
            unsigned wh[2][4], wm[2][4], wl[2][4], xh[4], xm[4], xl[4];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    split_pair(w[u][i][e].x, w[u][i][e].y, wh[i][2 * e], wm[i][2 * e], wl[i][2 * e]);
                    split_pair(w[u][i][e].z, w[u][i][e].w, wh[i][2 * e + 1], wm[i][2 * e + 1], wl[i][2 * e + 1]);
                }
                split_pair(x[u][e].x, x[u][e].y, xh[2 * e], xm[2 * e], xl[2 * e]);
                split_pair(x[u][e].z, x[u][e].w, xh[2 * e + 1], xm[2 * e + 1], xl[2 * e + 1]);
            }
            float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                mma_parts(c, wl, xh, j);
                mma_parts(c, wh, xl, j);
                mma_parts(c, wm, xm, j);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                mma_parts(c, wm, xh, j);
                mma_parts(c, wh, xm, j);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) mma_parts(c, wh, xh, j);
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i] += c[i];
        }
    }
    pdl_trigger();
#pragma unroll
    for (int i = 0; i < 4; ++i) sums[warp][2 * t + (i & 1)][g + 8 * (i >> 1)] = acc[i];
    __syncthreads();
    const int f = threadIdx.x % FK_ROWS, m = threadIdx.x / FK_ROWS, n = n0 + f;
    if (warp >= FK_TOKENS / 2) return;                  // a warp has the 16 columns of two tokens
    const bool mine = m < M && n < N;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < FK_WARPS; ++w) v += sums[w][m][f];
    for (int half = 0; half < 2; ++half) {
        const bool again = mine && (lane >> 4) == half && !isfinite(v);
        if (!__any_sync(0xffffffffu, again)) continue;
        const bool nan = row_has_nan(A + (size_t)(2 * warp + half) * lda, K);
        if (again) v = nan ? NAN : plain_product(A + (size_t)m * lda, W + (size_t)n * ldw, K);
    }
    if (!mine) return;
    v = mode_activation(v + (bias != nullptr ? bias[n] : 0.f), mode);
    const size_t o = (size_t)m * ldo + n;
    if (mode == MX_MODE_RESIDUAL) v += residual[o];
    out[o] = v;
}

// ------------------------------------------------------------------------------------------- the host's side
constexpr int FS_MAX_SPLITS = 8;

void fs_config(cudaLaunchConfig_t& config, cudaLaunchAttribute (&attribute)[2], int blocks, int splits, size_t smem,
               cudaStream_t stream) {
    config = {};
    config.gridDim = dim3(blocks);
    config.blockDim = dim3(FS_THREADS);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = splits;
    attribute[0].val.clusterDim.y = attribute[0].val.clusterDim.z = 1;
    attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[1].val.programmaticStreamSerializationAllowed = mx_chained_launch_enabled() ? 1 : 0;
    config.attrs = attribute;
    config.numAttrs = 2;
}

// Lets the kernel use its shared memory on the current device.
bool fs_ready() {
    return cudaFuncSetAttribute(gemm_f32_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FS_SMEM) == cudaSuccess;
}

// Clusters of `splits` blocks that run at a time: what the device's groups of SMs leave room for.
int fs_clusters(int splits) {
    static int known[FS_MAX_SPLITS + 1];                // the same on every GPU this library is built for
    if (known[splits] == 0) {
        cudaLaunchConfig_t config;
        cudaLaunchAttribute attribute[2];
        fs_config(config, attribute, splits * 148, splits, FS_SMEM, nullptr);
        config.numAttrs = 1;
        int n = 0;
        if (!fs_ready() || cudaOccupancyMaxActiveClusters(&n, gemm_f32_split_kernel, &config) != cudaSuccess) {
            cudaGetLastError();
            n = 148 / splits;
        }
        known[splits] = max(1, n);
    }
    return known[splits];
}

// The stages that a tile of plan.tokens leaves room for; returns the bytes of shared memory.
size_t fs_stages(FsPlan& plan) {
    const int room = FS_SMEM - 1024, x_raw = plan.tokens * FS_K * 4, x_parts = 3 * plan.tokens * FS_K * 2;
    plan.inlined = plan.tokens <= FS_INLINE_TOKENS;
    plan.accumulators = max(2, min(4, (FS_TMEM - 3 * FS_A_COLUMNS) / plan.tokens));
    plan.part_stages = min(4, (FS_TMEM - plan.accumulators * plan.tokens) / FS_A_COLUMNS);
    plan.raw_bytes = FS_RAW_BYTES + (plan.inlined ? x_raw : 0);
    plan.x_stages = plan.inlined ? plan.part_stages : max(2, min(4, (room - 4 * (int)plan.raw_bytes) / x_parts));
    plan.raw_stages = max(2, min(FS_MAX_STAGES, (room - plan.x_stages * x_parts) / (int)plan.raw_bytes));
    return 1024 + (size_t)plan.x_stages * x_parts + (size_t)plan.raw_stages * plan.raw_bytes;
}

// The tiles and shares of K of a product. A stage takes the longest of its products (12 MMAs of `tokens` / 2 cycles, 40 at
// least), of splitting, and of its weights' way from HBM; a tile costs its start, the exchange of the sums
// and its end. The plan with the fewest cycles over the rounds that the SMs need is taken.
FsPlan fs_plan(int M, int N, int K) {
    FsPlan best = {};
    double best_cost = -1.0;
    const int weight_tiles = (N + FS_ROWS - 1) / FS_ROWS, stages = (K + FS_K - 1) / FS_K;
    const int least = (M + FS_MAX_TOKENS - 1) / FS_MAX_TOKENS;
    for (int tiles = least; tiles <= least + 3; ++tiles) {
        const int tokens = ((M + tiles - 1) / tiles + 15) / 16 * 16;
        if (tiles > least && tokens * (tiles - 1) >= M) continue;
        const double stage = max(max(12.0 * max(40.0, tokens / 2.0), 600.0), 750.0 / tiles);
        for (int splits = 1; splits <= FS_MAX_SPLITS && (splits == 1 || splits * 4 <= stages); ++splits) {
            const long long rounds = ((long long)weight_tiles * tiles + fs_clusters(splits) - 1) / fs_clusters(splits);
            const double cost = rounds * ((double)((stages + splits - 1) / splits) * stage + 9000.0 + 20.0 * tokens);
            if (best_cost < 0.0 || cost < best_cost) {
                best_cost = cost;
                best.tokens = tokens;
                best.token_tiles = (M + tokens - 1) / tokens;
                best.splits = splits;
            }
        }
    }
    return best;
}

}  // namespace

// Whether a float product is better off here than on the FP32 cores (gemm_f32.cu): K long enough for what a tile costs
// beside its stages (some 9 us with the launch). Us there against here: 17 rows x 256 x 256 6.7 and 9.4, 17 x 4,096 x 512
// 10.6 and 13.1, 33 x 4,096 x 512 16.9 and 13.5, 17 x 1,024 x 1,024 17.2 and 12.7, 512 x 256 x 256 11.4 and 15.1, 512 x 512 x
// 512 16.4 and 15.8; 16 rows x 4,096 x 512 6.1 and 11.6, 9 x 2,048 x 2,048 16.5 and 15.5, 16 x 3,072 x 12,288 82 and 52; 4 rows
// x 3,072 x 12,288 50 and 51.
// Up to eight rows, on the kernel for them: 4 rows x 3,072 x 12,288 50 and 40, 4 x 12,288 x 3,072 36 and 33, 8 x 12,288 x
// 3,072 52 and 33, 4 x 1,024 x 1,024 6.0 and 5.2; but 4 x 49,152 x 3,072 103 and 110, 4 x 4,096 x 512 4.2 and 4.7, and one or
// two rows 5 to 15 % slower everywhere (2 x 12,288 x 3,072 31.6 and 32.1).
extern "C" int mx_gemm_f32_split_pays(int M, int N, int K) {
    if (N < 256 || M <= 2) return 0;
    if (M <= 4) return K >= 1024 && N <= 16384;
    return K >= (M <= 8 ? 512 : M <= 16 ? 2048 : M <= 32 ? 1024 : 512);
}

// Bytes of scratch that a product needs (0: none, and it is one launch instead of two): the parts of A where a tile has more
// tokens than are split in passing.
extern "C" long long mx_gemm_f32_split_scratch(int M, int N, int K) {
    if (M <= FS_INLINE_TOKENS || N <= 0 || K <= 0 || fs_plan(M, N, K).tokens <= FS_INLINE_TOKENS) return 0;
    return 3LL * M * ((K + 7) / 8 * 8) * 2;
}

// K, lda and ldw are multiples of 4; A, W and the scratch start on 16-byte boundaries.
extern "C" int mx_gemm_f32_split(const float* A, const float* W, const float* bias, const float* residual, float* out,
                                 void* scratch, int M, int N, int K, int lda, int ldw, int ldo, int mode, int* status,
                                 cudaStream_t stream) {
    if (M <= 0 || N <= 0) return MX_OK;
    if (K <= 0 || K % 4 != 0) MX_REFUSE("split gemm: K = %d is not a positive multiple of 4", K);
    if (lda % 4 != 0 || ldw % 4 != 0) MX_REFUSE("split gemm: row strides %d, %d are not multiples of 4", lda, ldw);
    if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(scratch)) & 15)
        MX_REFUSE("split gemm: operands must start on 16-byte boundaries");
    if (mode < 0 || mode > MX_MODE_LAST) MX_REFUSE("split gemm: unknown epilogue mode %d", mode);
    if (mode == MX_MODE_RESIDUAL && residual == nullptr) MX_REFUSE("split gemm: residual mode without a residual");
    if (status == nullptr) MX_REFUSE("split gemm: a status word is needed for its bounded waits");
    if (3LL * M > 0x7fffffffLL) MX_REFUSE("split gemm: M = %d is beyond this kernel's coordinates", M);

    if (M <= FK_TOKENS) {
        const cudaError_t e = mx_launch_chained(gemm_f32_skinny_kernel, dim3((N + FK_ROWS - 1) / FK_ROWS), dim3(FK_THREADS), 0,
                                                stream, A, lda, W, ldw, bias, residual, out, ldo, M, N, K, mode);
        if (e != cudaSuccess) {
            mx_set_error("split gemm: launch failed: %s", cudaGetErrorString(e));
            return (int)e;
        }
        return MX_OK;
    }
    if (!fs_ready()) MX_REFUSE("split gemm: cannot reserve %d bytes of shared memory", FS_SMEM);
    FsPlan plan = fs_plan(M, N, K);
    const size_t smem = fs_stages(plan);
    const long long blocks = (long long)((N + FS_ROWS - 1) / FS_ROWS) * plan.token_tiles * plan.splits;
    if (blocks > 0x7fffffffLL) MX_REFUSE("split gemm: %d x %d is beyond this kernel's grid", M, N);
    if (!plan.inlined && scratch == nullptr) MX_REFUSE("split gemm: %d rows need scratch", M);
    CUtensorMap map_w, map_x;
    int rc = mx_tensor_map_form(&map_w, W, N, K, ldw, FS_ROWS, MX_MAP_F32_128B);
    if (rc != MX_OK) return rc;
    cudaError_t e = cudaSuccess;
    if (plan.inlined) {
        rc = mx_tensor_map_form(&map_x, A, M, K, lda, plan.tokens, MX_MAP_F32_128B);
        if (rc != MX_OK) return rc;
    } else {
        const int ldp = (K + 7) / 8 * 8;
        rc = mx_tensor_map_form(&map_x, scratch, 3LL * M, ldp, ldp, plan.tokens, MX_MAP_BF16_64B);
        if (rc != MX_OK) return rc;
        const long long eighths = (long long)M * (ldp / 8);
        e = mx_launch_chained(f32_split_kernel, dim3((unsigned)((eighths + FS_SPLIT_THREADS - 1) / FS_SPLIT_THREADS)),
                              dim3(FS_SPLIT_THREADS), 0, stream, A, lda, (__nv_bfloat16*)scratch, ldp, M, K);
    }
    if (e == cudaSuccess) {
        cudaLaunchConfig_t config;
        cudaLaunchAttribute attribute[2];
        fs_config(config, attribute, (int)blocks, plan.splits, smem, stream);
        mx_count_launch();
        e = cudaLaunchKernelEx(&config, gemm_f32_split_kernel, map_w, map_x, A, lda, W, ldw, bias, residual, out, ldo, M, N,
                               K, mode, (const FsPlan)plan, status);
    }
    if (e != cudaSuccess) {
        mx_set_error("split gemm: launch failed: %s", cudaGetErrorString(e));
        return (int)e;
    }
    return MX_OK;
}
