// The routed experts' products on the 5th-generation tensor cores (bfloat16), included by blocks.cu.
//
// The entries of all experts lie one after the other (route_sort), expert e's in [starts[e], starts[e + 1]).  A persistent
// block walks tiles (expert, 128 of its entries, a range of output features): the number of an expert's tiles follows from the
// counts on the device, so a step asks the host nothing.  Roles as in gemm_tcgen05.cu: a TMA producer, an MMA issuer with two
// accumulators that take turns, eight epilogue warps (two a lane quarter, every second 32 columns each).  A tile's rows behind the expert's last entry are other experts' and are
// not stored.  With GLU a tile's B rows are 128 gate rows and the 128 up rows that belong to them.
//
// What bounds it: neither the tensor cores (2,048 rows, eight experts of 1,408 of which a row takes two, width 2,048: 71 GFLOP in 141 us,
// a third of the burst rate) nor memory (138 MB of weights, 21 us), but part-filled last waves (352 and 256 tiles over 148 blocks) and
// the five launches around the two products.  All seven launches of that layer on a B200: 405 us in tiles of 64 on mma.sync -> 141.
#pragma once

#include "tcgen05.cuh"

constexpr int ET_BN = 256, ET_MAX_EXPERTS = 256, ET_EPI_WARPS = 8, ET_THREADS = 64 + 32 * ET_EPI_WARPS;

// expert_inner with its smooth activations in one form, c / (1 + e^-at) (gelu's as in gated_unit, common.cuh), so that 32 of them
// unrolled carry one exponential and one division each and no tanhf.
__device__ __forceinline__ float expert_inner_unrolled(int act, float s, float g, float u, float limit) {
    const float z = s * g, v = s * u, c = act == BACT_SWISH_CLAMP ? fminf(z, limit) : z;
    const float at = act == BACT_GELU_TANH ? 1.5957691216057308f * (z + 0.044715f * z * z * z) : act == BACT_SWISH_CLAMP ? 1.702f * c : z;
    const float smooth = (act == BACT_SIGMOID ? 1.f : c) / (1.f + expf(-at));
    if (act == BACT_SWISH_CLAMP) return smooth * (fminf(fmaxf(v, -limit), limit) + 1.f);
    if (act == BACT_SILU || act == BACT_GELU_TANH || act == BACT_SIGMOID) return smooth * v;
    return (act == BACT_RELU ? fmaxf(z, 0.f) : z) * v;
}

struct ExpertTcArgs {
    void *out;                    // GLU: bfloat16 [entries, N]; else float32 [entries, N]
    const int *starts;            // [E + 1]
    const float *entry_score;     // GLU: the score that multiplies an entry's input, or null
    int E, entries, N, K;         // N: output features (GLU: after the gate)
    int act;
    float limit;
    int *status;
};

struct ExpertTcSmem {
    __nv_bfloat16 a[TG_STAGES][TG_BM * TG_BK];
    __nv_bfloat16 b[TG_STAGES][ET_BN * TG_BK];
    unsigned long long full[TG_STAGES], empty[TG_STAGES], acc_full[2], acc_empty[2];
    unsigned tmem_base;
    int first_tile[ET_MAX_EXPERTS + 1];      // tiles ahead of each expert's
    int start[ET_MAX_EXPERTS + 1];
};

// The rows of `in` [*, K] that the entries name, one after the other.
__global__ void __launch_bounds__(256) expert_gather_kernel(const uint4 *__restrict__ in, const int *__restrict__ entry_row,
                                                            const int *__restrict__ starts, int E, uint4 *__restrict__ out, int vectors) {
    pdl_trigger();
    pdl_wait();
    const int entries = starts[E];
    for (int entry = blockIdx.x; entry < entries; entry += gridDim.x) {
        const uint4 *src = in + (size_t)entry_row[entry] * vectors;
        for (int v = threadIdx.x; v < vectors; v += 256) out[(size_t)entry * vectors + v] = src[v];
    }
}

template <bool GLU>
__global__ void __launch_bounds__(ET_THREADS)
expert_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, ExpertTcArgs a) {
    extern __shared__ unsigned char et_raw[];
    ExpertTcSmem &s = *reinterpret_cast<ExpertTcSmem *>((reinterpret_cast<uintptr_t>(et_raw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int OUT_COLS = GLU ? ET_BN / 2 : ET_BN;
    constexpr unsigned STAGE_BYTES = (TG_BM + ET_BN) * TG_BK * sizeof(__nv_bfloat16);
    if (threadIdx.x == 0) {
        for (int i = 0; i < TG_STAGES; ++i) { mbar_init(&s.full[i], 1); mbar_init(&s.empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&s.acc_full[i], 1); mbar_init(&s.acc_empty[i], ET_EPI_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) tmem_alloc(&s.tmem_base, 2 * ET_BN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // the next kernel may be scheduled only once every block holds its tensor memory (gemm_tcgen05.cu says why)
    pdl_trigger();
    pdl_wait();
    const int tiles_n = (a.N + OUT_COLS - 1) / OUT_COLS;
    for (int e = threadIdx.x; e <= a.E; e += ET_THREADS) s.start[e] = a.starts[e];
    __syncthreads();
    if (threadIdx.x == 0) {
        int tiles = 0;
        for (int e = 0; e < a.E; ++e) {
            s.first_tile[e] = tiles;
            tiles += (s.start[e + 1] - s.start[e] + TG_BM - 1) / TG_BM * tiles_n;
        }
        s.first_tile[a.E] = tiles;
    }
    __syncthreads();
    const unsigned tmem = s.tmem_base;
    const int num_tiles = s.first_tile[a.E], nk = (a.K + TG_BK - 1) / TG_BK;
    int failed = 0;
    // tile number -> expert, first entry, first output feature; down an expert's entries first, so that tiles that run at the
    // same time share their rows of W
    auto locate = [&](int tile, int &e, int &m0, int &n0) {
        e = 0;
        while (s.first_tile[e + 1] <= tile) ++e;
        const int mine = tile - s.first_tile[e], down = (s.start[e + 1] - s.start[e] + TG_BM - 1) / TG_BM;
        m0 = s.start[e] + mine % down * TG_BM;
        n0 = mine / down * OUT_COLS;
    };
    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            for (int tile = blockIdx.x; tile < num_tiles && !failed; tile += gridDim.x) {
                int e, m0, n0;
                locate(tile, e, m0, n0);
                const int w0 = GLU ? e * 2 * a.N + n0 : e * a.N + n0;
                for (int i = 0; i < nk; ++i, ++it) {
                    const int st = it % TG_STAGES;
                    if (it >= TG_STAGES && !mbar_wait(&s.empty[st], (it / TG_STAGES - 1) & 1)) { failed = 1; break; }
                    mbar_expect_tx(&s.full[st], STAGE_BYTES);
                    tma_load_2d(s.a[st], &map_a, &s.full[st], i * TG_BK, m0);
                    tma_load_2d(s.b[st], &map_w, &s.full[st], i * TG_BK, w0);
                    tma_load_2d(s.b[st] + ET_BN / 2 * TG_BK, &map_w, &s.full[st], i * TG_BK, w0 + (GLU ? a.N : ET_BN / 2));
                }
            }
            if (failed) atomicExch(a.status, 21);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr unsigned idesc = instr_desc_bf16(ET_BN);
            int it = 0, j = 0;
            for (int tile = blockIdx.x; tile < num_tiles && !failed; tile += gridDim.x, ++j) {
                const int buf = j & 1;
                if (j >= 2 && !mbar_wait(&s.acc_empty[buf], ((j >> 1) - 1) & 1)) { failed = 2; break; }
                tc_fence_after();
                for (int i = 0; i < nk; ++i, ++it) {
                    const int st = it % TG_STAGES;
                    if (!mbar_wait(&s.full[st], (it / TG_STAGES) & 1)) { failed = 2; break; }
                    tc_fence_after();
                    const unsigned long long ad = smem_desc_sw128(s.a[st]), bd = smem_desc_sw128(s.b[st]);
#pragma unroll
                    for (int k = 0; k < TG_BK / 16; ++k) umma_bf16(tmem + buf * ET_BN, ad + 2 * k, bd + 2 * k, idesc, (i | k) ? 1u : 0u);
                    umma_commit(&s.empty[st]);
                }
                if (!failed) umma_commit(&s.acc_full[buf]);
            }
            if (failed) atomicExch(a.status, 22);
        }
    } else {
        const int quarter = warp & 3, turn = (warp - 2) >> 2;
        int j = 0;
        for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x, ++j) {
            int e, m0, n0;
            locate(tile, e, m0, n0);
            const int buf = j & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(&s.acc_full[buf], (j >> 1) & 1))) { failed = 3; if (lane == 0) atomicExch(a.status, 23); break; }
            tc_fence_after();
            const unsigned acc = tmem + buf * ET_BN + ((unsigned)(quarter * 32) << 16);
            const int entry = m0 + quarter * 32 + lane;
            const bool mine = entry < s.start[e + 1];
            const float score = GLU && mine && a.entry_score != nullptr ? a.entry_score[entry] : 1.f;
#pragma unroll 1
            for (int c0 = turn * 32; c0 < OUT_COLS; c0 += 64) {
                if (n0 + c0 >= a.N) break;
                unsigned v[32];
                tmem_ld32(acc + c0, v);
                if (GLU) {
                    unsigned u[32];
                    tmem_ld32(acc + ET_BN / 2 + c0, u);
                    if (mine) {
                        __nv_bfloat16 *dst = (__nv_bfloat16 *)a.out + (size_t)entry * a.N + n0 + c0;
#pragma unroll
                        for (int i = 0; i < 32; i += 8) {
                            if (n0 + c0 + i >= a.N) break;
                            unsigned w[4];
#pragma unroll
                            for (int p = 0; p < 4; ++p) {
                                const __nv_bfloat162 b = __floats2bfloat162_rn(
                                    expert_inner_unrolled(a.act, score, __uint_as_float(v[i + 2 * p]), __uint_as_float(u[i + 2 * p]), a.limit),
                                    expert_inner_unrolled(a.act, score, __uint_as_float(v[i + 2 * p + 1]), __uint_as_float(u[i + 2 * p + 1]), a.limit));
                                w[p] = *reinterpret_cast<const unsigned *>(&b);
                            }
                            *reinterpret_cast<uint4 *>(dst + i) = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    }
                } else if (mine) {
                    float *dst = (float *)a.out + (size_t)entry * a.N + n0 + c0;
#pragma unroll
                    for (int i = 0; i < 32; i += 4)
                        if (n0 + c0 + i < a.N) *reinterpret_cast<uint4 *>(dst + i) = make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                }
                __syncwarp();           // the next pass reads tensor memory, which takes the warp as a whole
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s.acc_empty[buf]);
        }
    }
    // a role that gave up may leave copies in flight: bounded time to land before memory is released
    if (failed && lane == 0)
        for (int st = 0; st < TG_STAGES; ++st) mbar_wait(&s.full[st], 0);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem, 2 * ET_BN);
}

template <bool GLU>
static int launch_expert_tc(const __nv_bfloat16 *in, const __nv_bfloat16 *w, const ExpertTcArgs &a, int tiles, int sms, cudaStream_t stream) {
    CUtensorMap ma, mw;
    if (int rc = tensor_map_2d(in, a.entries, a.K, a.K, TG_BM, TG_BK, 2, &ma)) return rc;
    if (int rc = tensor_map_2d(w, a.E * a.N * (GLU ? 2 : 1), a.K, a.K, ET_BN / 2, TG_BK, 2, &mw)) return rc;
    const size_t smem = sizeof(ExpertTcSmem) + 1024;
    const cudaError_t e = cudaFuncSetAttribute(expert_tcgen05_kernel<GLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) JK_FAIL(JK_CUDA_ERROR, "expert products: %s", cudaGetErrorString(e));
    jk_launch(expert_tcgen05_kernel<GLU>, dim3(std::min(tiles, sms)), dim3(ET_THREADS), smem, stream, ma, mw, a);
    JK_CHECK_LAUNCH("expert products");
    return JK_OK;
}
