// The float32 matrix product on the CUDA cores:  C[M, N] = A[M, K] * W[N, K]^T (+ bias[N]).  Short sums take it, and
// operands off 16 bytes; the others go to gemm_f32_tcgen05.cu (jk::f32_plan).
//
// Fused multiply-adds in float32: no tensor cores, hence no TF32 rounding of the operands.
// (reference: the products at jiuge.cpp:200, :236, :247, :249, :264 go to a library.)
//
// K is cut into chunks of GF_BK.  Chunk c belongs to group c % GF_GROUPS, a group adds the products of even and of odd k in
// two chains of float32 multiply-adds (the two halves of fma.rn.f32x2), each in ascending order, and an output is
// (g0 + g1) + (g2 + g3) with g = even + odd.  That order depends on K alone, so a row's result does not depend on what else is
// in the batch, and every tile below gives the same bits.
//
// What bounds it: the float32 pipes.  A thread has TM x TN outputs, as two-element accumulators; per four k it reads TM + TN
// vectors of 16 bytes for TM x TN x 2 two-element multiply-adds, which at 8 x 8 leaves shared memory at 45 % of its rate (at
// 4 x 4, where reads of 16 bytes take three cycles each whatever they share, it was the bound).  The groups of a block keep
// rings and, for one warp a group, timing of their own: no barrier of the block stands in the loop.  Cutting K over the
// warps of a block gives outputs of few tiles (301 x 1,536 x 1,536: 120 tiles of 64 x 64) two warps on every scheduler where
// one tile had one chain.  Rows of a tile lie in shared memory as in memory, padded by four floats, so that eight lanes that
// read eight rows touch every bank once.
// Measured on a B200 against tiles of 64 x 64 with 4 x 4 outputs a thread, loaded element by element (us): 301 x 2,560 x
// 1,536 393 -> 72, 301 x 1,536 x 1,536 262 -> 44, 301 x 7,680 x 1,536 551 -> 195, 301 x 1,536 x 3,840 656 -> 101,
// 2,048 x 7,680 x 1,536 2,202 -> 1,065 (0.61 of the pipes' 74 TFLOP/s), 8 x 2,560 x 1,536 264 -> 15.
#include "common.cuh"
#include "host_rules.h"

#include <cmath>

namespace {

constexpr int GF_BK = 16, GF_LD = GF_BK + 4, GF_GROUPS = 4;

// `bytes` of VEC floats are copied, the rest are zeros
template <int VEC> __device__ __forceinline__ void gf_copy(unsigned dst, const float *src, int bytes) {
    if (VEC == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// A thread's share of a tile of ROWS rows of GF_BK floats: every THREADS / (GF_BK / VEC)-th row, always the same columns.
// Rows beyond the matrix are left as they are (their products are not stored), columns beyond K are zeros.
template <int ROWS, int THREADS, int VEC> struct GfLoader {
    static constexpr int PER_ROW = GF_BK / VEC, STEP = THREADS / PER_ROW, COPIES = (ROWS + STEP - 1) / STEP;
    static_assert(ROWS % STEP == 0, "every thread has the same number of copies");
    const float *src[COPIES];
    unsigned dst;
    int column, copies;
    __device__ __forceinline__ GfLoader(float *tile, const float *from, int ld, int row0, int rows, int k0, int thread) {
        column = k0 + thread % PER_ROW * VEC;
        dst = (unsigned)__cvta_generic_to_shared(tile + thread / PER_ROW * GF_LD + thread % PER_ROW * VEC);
#pragma unroll
        for (int i = 0; i < COPIES; ++i) src[i] = from + (size_t)min(row0 + thread / PER_ROW + i * STEP, rows - 1) * ld;
        copies = max(0, rows - row0 - thread / PER_ROW + STEP - 1) / STEP;
    }
    // the tile of the group's chunk s into the ring's place `slot` (bytes from its first)
    __device__ __forceinline__ void load(int s, unsigned slot, int K) const {
        const int k = column + s * GF_GROUPS * GF_BK, bytes = k < K ? VEC * 4 : 0, at = k < K ? k : 0;
#pragma unroll
        for (int i = 0; i < COPIES; ++i)
            if (i < copies) gf_copy<VEC>(dst + slot + i * STEP * GF_LD * 4, src[i] + at, bytes);
    }
};
__device__ __forceinline__ void gf_fma2(unsigned long long &acc, unsigned long long a, unsigned long long w) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(acc) : "l"(a), "l"(w));
}

// MW warps a group, one below the other; TM x TN outputs a thread; STAGES chunks in a group's ring; VEC floats a copy (4 where
// every row starts on 16 bytes and holds whole vectors, else 1).
template <int MW, int TM, int TN, int STAGES, int VEC>
__global__ void __launch_bounds__(GF_GROUPS * MW * 32, 256 / (GF_GROUPS * MW * 32))
gemm_f32_kernel(const float *__restrict__ A, const float *__restrict__ W, const float *__restrict__ bias, float *__restrict__ C,
                int M, int N, int K, int lda, int ldw, int ldc) {
    constexpr int RY = 4 * MW, BM = RY * TM, BN = 8 * TN, THREADS = MW * 32;       // a warp: 4 threads down, 8 across
    constexpr int STAGE = (BM + BN) * GF_LD;
    extern __shared__ __align__(16) float gf_smem[];
    pdl_trigger();
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int group = threadIdx.x / THREADS, thread = threadIdx.x % THREADS, lane = thread & 31;
    const int tx = lane & 7, ty = (thread >> 5) * 4 + (lane >> 3);
    float *ring = gf_smem + group * STAGES * STAGE;
    const int chunks = (K + GF_BK - 1) / GF_BK, steps = chunks > group ? (chunks - group + GF_GROUPS - 1) / GF_GROUPS : 0;
    const GfLoader<BM, THREADS, VEC> load_a(ring, A, lda, m0, M, group * GF_BK, thread);
    const GfLoader<BN, THREADS, VEC> load_w(ring + BM * GF_LD, W, ldw, n0, N, group * GF_BK, thread);
    auto sync = [&] {
        if (MW == 1) __syncwarp();
        else asm volatile("bar.sync %0, %1;\n" ::"r"(1 + group), "n"(THREADS) : "memory");
    };
    pdl_wait();
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) {
            load_w.load(s, s * STAGE * 4, K);
            load_a.load(s, s * STAGE * 4, K);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    unsigned long long acc[TM][TN] = {};
    int slot = 0, free_slot = STAGES - 1;       // of the tile that is used now, and of the one that is loaded now
    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
        sync();
        if (s + STAGES - 1 < steps) {
            load_w.load(s + STAGES - 1, free_slot * STAGE * 4, K);
            load_a.load(s + STAGES - 1, free_slot * STAGE * 4, K);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const float *a_tile = ring + slot * STAGE + ty * GF_LD, *w_tile = ring + slot * STAGE + (BM + tx) * GF_LD;
#pragma unroll
        for (int k = 0; k < GF_BK; k += 4) {
            ulonglong2 w[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const ulonglong2 *>(w_tile + j * 8 * GF_LD + k);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(a_tile + i * RY * GF_LD + k);
#pragma unroll
                for (int j = 0; j < TN; ++j) gf_fma2(acc[i][j], a.x, w[j].x);
#pragma unroll
                for (int j = 0; j < TN; ++j) gf_fma2(acc[i][j], a.y, w[j].y);
            }
        }
        slot = slot + 1 == STAGES ? 0 : slot + 1;
        free_slot = free_slot + 1 == STAGES ? 0 : free_slot + 1;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    // the groups' shares meet in shared memory, added in the order of the groups
    constexpr int LD = BN + 1;
    float *shares = gf_smem + group * BM * LD;
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j)
            shares[(ty + i * RY) * LD + tx + j * 8] = __uint_as_float((unsigned)acc[i][j]) + __uint_as_float((unsigned)(acc[i][j] >> 32));
    __syncthreads();
    for (int i = threadIdx.x; i < BM * BN; i += GF_GROUPS * THREADS) {
        const int r = i / BN, c = i % BN, m = m0 + r, n = n0 + c;
        if (m >= M || n >= N) continue;
        const float *p = gf_smem + r * LD + c;
        C[(size_t)m * ldc + n] = ((p[0] + p[BM * LD]) + (p[2 * BM * LD] + p[3 * BM * LD])) + (bias ? bias[n] : 0.f);
    }
}

struct GfCall {
    const float *A, *W, *bias;
    float *C;
    int M, N, K, lda, ldw, ldc;
    cudaStream_t stream;
};

template <int MW, int TM, int TN, int STAGES> int gf_run(const GfCall &c) {
    constexpr int BM = 4 * MW * TM, BN = 8 * TN;
    const dim3 grid((c.N + BN - 1) / BN, (c.M + BM - 1) / BM);
    const bool whole = c.K % 4 == 0 && c.lda % 4 == 0 && c.ldw % 4 == 0 && (((uintptr_t)c.A | (uintptr_t)c.W) & 15) == 0;
    constexpr int ring = GF_GROUPS * STAGES * (BM + BN) * GF_LD * 4, shares = GF_GROUPS * BM * (BN + 1) * 4, smem = ring > shares ? ring : shares;
    static_assert(smem <= 227 * 1024, "shared memory");
    auto kernel = whole ? gemm_f32_kernel<MW, TM, TN, STAGES, 4> : gemm_f32_kernel<MW, TM, TN, STAGES, 1>;
    const cudaError_t e = cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) JK_FAIL(JK_CUDA_ERROR, "gemm_f32: %s", cudaGetErrorString(e));
    jk_launch(kernel, grid, dim3(GF_GROUPS * MW * 32), smem, c.stream, c.A, c.W, c.bias, c.C, c.M, c.N, c.K, c.lda, c.ldw, c.ldc);
    JK_CHECK_LAUNCH("gemm_f32");
    return JK_OK;
}

// by jk::F32_TILES
constexpr int (*GF_RUN[])(const GfCall &) = {gf_run<1, 2, 8, 3>, gf_run<1, 4, 4, 4>, gf_run<1, 8, 8, 3>, gf_run<2, 8, 8, 2>};

}  // namespace

JK_EXPORT int jk_gemm_f32(const float *A, int lda, const float *W, int ldw, const float *bias,
                          float *C, int ldc, int M, int N, int K, cudaStream_t stream) {
    if (M == 0 || N == 0) return JK_OK;
    JK_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_f32: M %d N %d K %d", M, N, K);
    double us = 0.;
    const int tile = jk::f32_tile(M, N, 148, &us);
    JK_REQUIRE(tile >= 0, "gemm_f32: M %d is too large for one launch", M);
    return GF_RUN[tile](GfCall{A, W, bias, C, M, N, K, lda, ldw, ldc, stream});
}
