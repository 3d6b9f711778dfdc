// The float32 matrix product on the 5th-generation tensor cores:  C[M, N] = A[M, K] * W[N, K]^T (+ bias[N]).
//
// A float32 number is the sum of three bfloat16 ones (round to nearest, twice the remainder: 8 + 8 + 8 bits and signs), and a product of two
// float32 numbers the sum of nine products of those, each exact in float32.  Six of them are made, smallest first: m m, h l, l h, h m, m h,
// h h.  What is left out (m l, l m, l l) is at most about 2^-24 of |a||w|, and 2^-27.4 in the mean (root of the mean square, normal operands).
// bfloat16 has float32's exponents but not its smallest numbers: below 2^-110 the parts of a number would be cut off.  So both operands are
// taken times 2^16, which makes every float32 number's parts whole, and the sums times 2^-32.
// The tensor core adds the products of FS_BK = 64 columns of K into tensor memory; these sums go to registers and are added
// up there by float32 additions, since the tensor core's own additions cut off instead of rounding, which adds up over a long
// chain.  Error against 64 bits (2-norm of the difference over that of the result, normal operands): K 1,536 1.0e-7 to 1.2e-7, the
// multiply-adds of gemm_f32.cu 2.5e-7; K 3,840 1.1e-7 to 1.6e-7 and 4.0e-7; K 96 0.8e-7 and 0.8e-7.
// Numbers that this does not carry (infinities, NaN, operands from 2^111 and results from 2^95 on) leave a result that
// is not finite: such outputs are made again from the operands by the multiply-adds of gemm_f32.cu, in its order.
// A row's result depends on the row and on the cuts of K, not on the tile nor on the other rows (jk::f32_plan says who sets the cuts).
//
// The weights are on the MMA's M side (128 features a tile), tokens on its N side (BN of them), so that a prompt's odd number
// of rows costs no more than its last tile of BN.  K is cut over the blocks of a cluster where tiles alone leave SMs idle;
// the blocks' sums meet in the order of the blocks through distributed shared memory.
//
// What bounds it: the MMAs (six where bfloat16 has one; 65 cycles each up to 128 tokens, 80 at 160: a chunk takes 1,560 to 1,920) and, by a
// little more, the chain from raw weights to split ones and from tensor memory to the sums, which two stages only half hide (1.2 to 1.5 us
// a chunk; 301 x 7,680 x 1,536: the tensor pipe is active for two thirds of the cycles of an SM that has a block, issue slots are used for three quarters).  Shared memory would hold both of an MMA's operands as a rule, and 24 MMAs a chunk would read 216 KB of it at BN = 160,
// as long as they take; so the weights' three parts go to tensor memory, from where an MMA takes its A operand as well.  Splitting
// weights and tokens in registers on their way to shared memory measured 89 us for 301 x 7,680 x 1,536 where this takes 45.
//
// Roles: warps 0..7 have two tasks that take turns: the weights come by TMA into a ring of raw chunks, a thread splits half a
// chunk of one row into tensor memory; and they hold the sums (two warps a lane quarter, half the columns each).  Warps 8..13 read
// the tokens from memory as float32, a chunk ahead in registers, and write their three bfloat16 tiles, 128-byte swizzled.
// Warp 14 issues the MMAs, which keeps its thread for as long as they run, and owns tensor memory.  More warps would leave a thread 96
// registers instead of 128.  Every wait is bounded; one that runs out leaves a code in `status`.
#include "tcgen05.cuh"

#include <algorithm>

JK_DEFINE_ERROR_BUFFER(jk_gemm_f32_tcgen05)

namespace {

constexpr int FS_BK = 64, FS_ADDERS = 8, FS_LOADERS = 6, FS_THREADS = 32 * (FS_ADDERS + FS_LOADERS + 1), FS_STAGES = 2;
constexpr float FS_SCALE = 65536.f, FS_UNSCALE = 1.f / (FS_SCALE * FS_SCALE);

struct FsArgs {
    const float *A, *W, *bias;
    float *C;
    int M, N, K, lda, ldw, ldc;
    int cuts;          // blocks of a cluster: ranges of K
    int *status;
};

template <int BN> struct FsSmem {
    static constexpr int RAW = BN <= 32 ? 6 : BN <= 64 ? 5 : BN <= 128 ? 4 : 3;      // raw chunks of weights in flight
    float w[RAW][2][TG_BM * 32];                        // [128 rows][32 floats] twice, 128-byte swizzled
    __nv_bfloat16 a[FS_STAGES][3][BN * FS_BK];
    unsigned long long raw_full[RAW], raw_empty[RAW], full[FS_STAGES], empty[FS_STAGES], acc_full[2], acc_empty[2];
    unsigned tmem_base;
};

__device__ __forceinline__ void tmem_ld16(unsigned addr, unsigned (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_st8(unsigned addr, const unsigned (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n"
                 ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
// the A operand [128 lanes][16] in tensor memory, two bfloat16 a column
__device__ __forceinline__ void umma_bf16_tmem(unsigned d, unsigned a, unsigned long long bdesc, unsigned idesc, unsigned accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
                 ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ unsigned bf16_pair(float lo, float hi) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const unsigned *>(&p);
}
__device__ __forceinline__ float pair_lo(unsigned p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float pair_hi(unsigned p) { return __uint_as_float(p & 0xffff0000u); }

// two numbers times FS_SCALE in one instruction
__device__ __forceinline__ void scale_pair(float &x, float &y) {
    asm("{ .reg .b64 a, b;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %2};\n\tmul.rn.f32x2 a, a, b;\n\tmov.b64 {%0, %1}, a; }" : "+f"(x), "+f"(y) : "f"(FS_SCALE));
}
// two numbers rounded to bfloat16, and what is left of them
__device__ __forceinline__ unsigned split_pair(float &x, float &y) {
    const unsigned h = bf16_pair(x, y);
    asm("{ .reg .b64 a, b, c;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %3};\n\tmov.b64 c, {%4, %4};\n\tfma.rn.f32x2 a, b, c, a;\n\tmov.b64 {%0, %1}, a; }"
        : "+f"(x), "+f"(y) : "f"(pair_lo(h)), "f"(pair_hi(h)), "f"(-1.f));
    return h;
}
// four consecutive floats into the three tiles (`plane` bytes apart)
__device__ __forceinline__ void split_store(unsigned char *dst, int plane, float4 x) {
    scale_pair(x.x, x.y);
    scale_pair(x.z, x.w);
    const unsigned h0 = split_pair(x.x, x.y), h1 = split_pair(x.z, x.w);
    const unsigned m0 = split_pair(x.x, x.y), m1 = split_pair(x.z, x.w);
    *reinterpret_cast<uint2 *>(dst) = make_uint2(h0, h1);
    *reinterpret_cast<uint2 *>(dst + plane) = make_uint2(m0, m1);
    *reinterpret_cast<uint2 *>(dst + 2 * plane) = make_uint2(bf16_pair(x.x, x.y), bf16_pair(x.z, x.w));
}
// The outputs of row m that came out infinite or not a number (`bad`), from the operands themselves, a warp a row and a lane an output: what
// gemm_f32.cu gives, its sums in its order.  A row of A that holds a NaN, the usual cause, is known by one look at it.  301 x 7,680 x 1,536 with
// one row of NaN takes 70 us where it takes 45 without, with an infinity in one row 145, all rows NaN some 250 (a thread an output by itself: 175, 170 and 17,000).
__device__ __noinline__ void store_plain(const FsArgs &a, int m, int n, bool bad) {
    const float *x = a.A + (size_t)m * a.lda;
    bool nan = false;
    for (int k = (threadIdx.x & 31) * 4; k < a.K; k += 128) {
        const float4 v = *reinterpret_cast<const float4 *>(x + k);
        nan = nan || isnan(v.x) || isnan(v.y) || isnan(v.z) || isnan(v.w);
    }
    nan = __any_sync(0xffffffffu, nan);
    if (!bad) return;
    float sum = NAN;
    if (!nan) {
        const float *w = a.W + (size_t)n * a.ldw;
        float even[4] = {0.f, 0.f, 0.f, 0.f}, odd[4] = {0.f, 0.f, 0.f, 0.f};
        for (int k0 = 0; k0 < a.K; k0 += 64)
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int k = k0 + 4 * i, g = i / 4;
                if (k >= a.K) break;
                const float4 p = *reinterpret_cast<const float4 *>(x + k), q = *reinterpret_cast<const float4 *>(w + k);
                even[g] = fmaf(p.z, q.z, fmaf(p.x, q.x, even[g]));
                odd[g] = fmaf(p.w, q.w, fmaf(p.y, q.y, odd[g]));
            }
        sum = ((even[0] + odd[0]) + (even[1] + odd[1])) + ((even[2] + odd[2]) + (even[3] + odd[3])) + (a.bias != nullptr ? a.bias[n] : 0.f);
    }
    a.C[(size_t)m * a.ldc + n] = sum;
}
__device__ __forceinline__ float load_cluster(unsigned addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

template <int BN>
__global__ void __launch_bounds__(FS_THREADS, 1) gemm_f32_tcgen05_kernel(const __grid_constant__ CUtensorMap map_w, FsArgs a) {
    extern __shared__ unsigned char fs_raw[];
    using Smem = FsSmem<BN>;
    constexpr int RAW = Smem::RAW, HALF = BN / 2, TMEM = 2 * BN + FS_STAGES * 96 <= 256 ? 256 : 512;
    Smem &s = *reinterpret_cast<Smem *>((reinterpret_cast<uintptr_t>(fs_raw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x % a.cuts, tile = blockIdx.x / a.cuts, tiles_m = (a.M + BN - 1) / BN;
    const int m0 = tile % tiles_m * BN, n0 = tile / tiles_m * TG_BM;
    const int all = (a.K + FS_BK - 1) / FS_BK, per = (all + a.cuts - 1) / a.cuts, first = rank * per, chunks = max(0, min(per, all - first));
    if (threadIdx.x == 0) {
        for (int i = 0; i < RAW; ++i) { mbar_init(&s.raw_full[i], 1); mbar_init(&s.raw_empty[i], FS_ADDERS); }
        for (int i = 0; i < FS_STAGES; ++i) { mbar_init(&s.full[i], FS_LOADERS + FS_ADDERS); mbar_init(&s.empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&s.acc_full[i], 1); mbar_init(&s.acc_empty[i], FS_ADDERS); }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == FS_ADDERS + FS_LOADERS) tmem_alloc(&s.tmem_base, TMEM);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = s.tmem_base, tmem_w = tmem + 2 * BN;      // sums, then the weights' parts: 32 columns each, three a stage
    int failed = 0;
    pdl_trigger();      // once the block holds its tensor memory: gemm_tcgen05.cu says why
    float *share = reinterpret_cast<float *>(s.w);

    if (warp == FS_ADDERS + FS_LOADERS) {
        pdl_wait();
        if (lane == 0) {
            constexpr unsigned idesc = instr_desc_bf16(BN);
            constexpr int OF_W[6] = {1, 0, 2, 0, 1, 0}, OF_A[6] = {1, 2, 0, 1, 0, 0};      // smallest first
            for (int c = 0; c < chunks; ++c) {
                const int st = c % FS_STAGES, buf = c & 1;
                if (!mbar_wait(&s.full[st], (c / FS_STAGES) & 1) || (c >= 2 && !mbar_wait(&s.acc_empty[buf], ((c >> 1) - 1) & 1))) { failed = 1; break; }
                tc_fence_after();
#pragma unroll
                for (int t = 0; t < 6; ++t) {
                    const unsigned long long ad = smem_desc_sw128(s.a[st][OF_A[t]]);
                    const unsigned wt = tmem_w + st * 96 + OF_W[t] * 32;
#pragma unroll
                    for (int k = 0; k < FS_BK / 16; ++k) umma_bf16_tmem(tmem + buf * BN, wt + 8 * k, ad + 2 * k, idesc, (t | k) ? 1u : 0u);
                }
                umma_commit(&s.empty[st]);
                umma_commit(&s.acc_full[buf]);
            }
            if (failed) atomicExch(a.status, 31);
        }
    } else if (warp >= FS_ADDERS) {
        constexpr int STEP = FS_LOADERS * 2, ROWS = (BN + STEP - 1) / STEP;      // 16 threads a row
        const int thread = threadIdx.x - 32 * FS_ADDERS, row = thread / 16, col = thread % 16 * 4;
        float4 x[ROWS];
        auto load = [&](int c) {
            const int k = (first + c) * FS_BK + col;
#pragma unroll
            for (int i = 0; i < ROWS; ++i)
                if (row + i * STEP < BN)
                    x[i] = k < a.K ? *reinterpret_cast<const float4 *>(a.A + (size_t)min(m0 + row + STEP * i, a.M - 1) * a.lda + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        pdl_wait();
        if (chunks > 0) load(0);
        for (int c = 0; c < chunks; ++c) {
            const int st = c % FS_STAGES;
            if (c >= FS_STAGES && !__all_sync(0xffffffffu, mbar_wait(&s.empty[st], (c / FS_STAGES - 1) & 1))) { failed = 2; break; }
            unsigned char *tile_a = reinterpret_cast<unsigned char *>(s.a[st][0]);
#pragma unroll
            for (int i = 0; i < ROWS; ++i) {
                const int r = row + i * STEP;
                if (r < BN) split_store(tile_a + r * 128 + (((col >> 3) ^ (r & 7)) << 4) + (col & 7) * 2, BN * 128, x[i]);
            }
            if (c + 1 < chunks) load(c + 1);
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s.full[st]);
        }
        if (failed && lane == 0) atomicExch(a.status, 32);
    } else {
        const int quarter = warp & 3, half = warp >> 2;
        float acc[HALF];
#pragma unroll
        for (int j = 0; j < HALF; ++j) acc[j] = 0.f;
        auto bring = [&](int c) {       // one thread: a raw chunk of weights
            const int r = c % RAW;
            mbar_expect_tx(&s.raw_full[r], sizeof(s.w[0]));
            for (int h = 0; h < 2; ++h) tma_load_2d(s.w[r][h], &map_w, &s.raw_full[r], (first + c) * FS_BK + 32 * h, n0);
        };
        auto add = [&](int c) {         // the sums of chunk c
            const int buf = c & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(&s.acc_full[buf], (c >> 1) & 1))) { failed = 3; return; }
            tc_fence_after();
            const unsigned d = tmem + buf * BN + half * HALF + ((unsigned)(quarter * 32) << 16);
#pragma unroll
            for (int j = 0; j + 32 <= HALF; j += 32) {
                unsigned v[32];
                tmem_ld32(d + j, v);
#pragma unroll
                for (int i = 0; i < 32; ++i) acc[j + i] += __uint_as_float(v[i]);
            }
            if (HALF % 32) {
                unsigned v[16];
                tmem_ld16(d + HALF - 16, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[HALF - 16 + i] += __uint_as_float(v[i]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s.acc_empty[buf]);
        };
        const bool bringer = threadIdx.x == 0;
        if (bringer)                    // the weights depend on no kernel before this one
            for (int c = 0; c < RAW && c < chunks; ++c) bring(c);
        pdl_wait();
        const int row = quarter * 32 + lane;
        for (int c = 0; c < chunks; ++c) {
            const int st = c % FS_STAGES, r = c % RAW;
            bool ok = mbar_wait(&s.raw_full[r], (c / RAW) & 1);
            if (c >= FS_STAGES) ok = mbar_wait(&s.empty[st], (c / FS_STAGES - 1) & 1) && ok;
            if (!__all_sync(0xffffffffu, ok)) { failed = 3; break; }
            tc_fence_after();
            const unsigned to = tmem_w + st * 96 + half * 16 + ((unsigned)(quarter * 32) << 16);
            const unsigned char *from = reinterpret_cast<const unsigned char *>(s.w[r][half]) + row * 128;
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                float v[16];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float4 x = *reinterpret_cast<const float4 *>(from + (((4 * p + i) ^ (row & 7)) << 4));
                    scale_pair(x.x, x.y);
                    scale_pair(x.z, x.w);
                    v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
                }
#pragma unroll
                for (int part = 0; part < 3; ++part) {
                    unsigned b[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) b[i] = part < 2 ? split_pair(v[2 * i], v[2 * i + 1]) : bf16_pair(v[2 * i], v[2 * i + 1]);
                    tmem_st8(to + part * 32 + p * 8, b);
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&s.full[st]);
                mbar_arrive(&s.raw_empty[r]);
            }
            if (c >= 2) add(c - 2);
            if (bringer && c + RAW < chunks) {
                if (mbar_wait(&s.raw_empty[r], (c / RAW) & 1)) bring(c + RAW);
                else failed = 3;
            }
            __syncwarp();
            if (__any_sync(0xffffffffu, failed != 0)) { failed = 3; break; }
        }
        for (int c = max(0, chunks - 2); c < chunks && !failed; ++c) add(c);
        if (failed && lane == 0) atomicExch(a.status, 33);
        const int m = m0 + half * HALF, n = n0 + quarter * 32 + lane;
        if (a.cuts > 1) {
            // every product of this block is complete (its last sums were read), so the ring is free to hold its share
#pragma unroll
            for (int j = 0; j < HALF; ++j) share[(half * HALF + j) * TG_BM + quarter * 32 + lane] = acc[j];
        } else {
            const bool mine = n < a.N;
            const float bias = mine && a.bias != nullptr ? a.bias[n] : 0.f;
            float *to = a.C + (size_t)m * a.ldc + n;
            bool finite = true;
#pragma unroll
            for (int j = 0; j < HALF; ++j) {
                finite = finite && isfinite(acc[j]);
                if (mine && m + j < a.M) to[(size_t)j * a.ldc] = fmaf(acc[j], FS_UNSCALE, bias);
            }
            if (__any_sync(0xffffffffu, mine && !finite))
                for (int j = 0; j < HALF && m + j < a.M; ++j) {
                    const bool bad = mine && !isfinite(to[(size_t)j * a.ldc]);
                    if (__any_sync(0xffffffffu, bad)) store_plain(a, m + j, n, bad);
                }
        }
    }
    if (a.cuts > 1) {
        cluster_sync();
        constexpr int OUTPUTS = BN * TG_BM;
        const int begin = rank * OUTPUTS / a.cuts, end = (rank + 1) * OUTPUTS / a.cuts;
        for (int i = begin + threadIdx.x; i < end; i += FS_THREADS) {
            float v = load_cluster(cluster_addr(share + i, 0));
            for (int r = 1; r < a.cuts; ++r) v += load_cluster(cluster_addr(share + i, r));
            const int m = m0 + i / TG_BM, n = n0 + i % TG_BM;          // a warp: 32 features of one row
            const bool mine = m < a.M && n < a.N;
            if (mine && isfinite(v)) a.C[(size_t)m * a.ldc + n] = fmaf(v, FS_UNSCALE, a.bias != nullptr ? a.bias[n] : 0.f);
            if (__any_sync(0xffffffffu, mine && !isfinite(v))) store_plain(a, m, n, mine && !isfinite(v));
        }
        cluster_sync();      // no block leaves while another reads its share
    }
    // a role that gave up may leave copies or MMAs in flight: bounded time for them before memory is released
    if (failed && lane == 0) {
        for (int r = 0; r < RAW; ++r) mbar_wait(&s.raw_full[r], 0);
        for (int st = 0; st < FS_STAGES; ++st) mbar_wait(&s.empty[st], 0);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == FS_ADDERS + FS_LOADERS) tmem_dealloc(tmem, TMEM);
}

template <int BN> int fs_run(const FsArgs &a, cudaStream_t stream) {
    auto kernel = gemm_f32_tcgen05_kernel<BN>;
    constexpr size_t smem = sizeof(FsSmem<BN>) + 1024;
    static_assert(smem <= 227 * 1024, "shared memory");
    static_assert((size_t)BN * TG_BM * 4 <= sizeof(FsSmem<BN>::w), "a block's share fits its ring");
    CUtensorMap mw;
    if (int rc = tensor_map_2d(a.W, a.N, a.K, a.ldw, TG_BM, 32, 4, &mw)) return rc;
    cudaError_t e = cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const long long tiles = (long long)((a.M + BN - 1) / BN) * ((a.N + TG_BM - 1) / TG_BM);
    if (e == cudaSuccess) e = jk_launch_clusters(kernel, a.cuts, dim3((unsigned)(tiles * a.cuts)), dim3(FS_THREADS), smem, stream, mw, a);
    if (e != cudaSuccess) JK_FAIL(JK_CUDA_ERROR, "gemm_f32_tcgen05: %s", cudaGetErrorString(e));
    return JK_OK;
}

}  // namespace

// rows start on 16 bytes and hold whole vectors of four
JK_EXPORT int jk_gemm_f32_tcgen05_supports(const float *A, int lda, const float *W, int ldw, int M, int N, int K) {
    return M >= 1 && N >= 1 && K >= 4 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
}

// `tile` tokens (32, 64, 96, 128 or 160) and `cuts` of K (1, 2, 4 or 8)
JK_EXPORT int jk_gemm_f32_tcgen05(const float *A, int lda, const float *W, int ldw, const float *bias, float *C, int ldc, int M, int N, int K,
                                  int tile, int cuts, int *status, cudaStream_t stream) {
    if (M == 0 || N == 0) return JK_OK;
    JK_REQUIRE(jk_gemm_f32_tcgen05_supports(A, lda, W, ldw, M, N, K), "gemm_f32_tcgen05: M %d N %d K %d, rows of %d and %d", M, N, K, lda, ldw);
    JK_REQUIRE(status != nullptr && (cuts == 1 || cuts == 2 || cuts == 4 || cuts == 8), "gemm_f32_tcgen05: %d cuts, or no status word", cuts);
    const FsArgs a{A, W, bias, C, M, N, K, lda, ldw, ldc, cuts, status};
    switch (tile) {
        case 32: return fs_run<32>(a, stream);
        case 64: return fs_run<64>(a, stream);
        case 96: return fs_run<96>(a, stream);
        case 128: return fs_run<128>(a, stream);
        case 160: return fs_run<160>(a, stream);
    }
    JK_FAIL(JK_BAD_ARGUMENT, "gemm_f32_tcgen05: tiles of %d tokens are not built", tile);
}
