// Float32 attention of prompts: plain causal softmax attention over a paged cache, heads of 64 or 128, tiles of query rows.
//
// The row kernel of attention.cu gives a warp whole (row, head) pairs: a score is one lane's chain over the head, and the weighted
// values one slice of it.  Here a block takes 32 or 64 rows of one request and head and 64 keys at a time: a lane makes two or four rows x 8
// keys of scores, and two or four rows x 4 or 8 columns of every 32 of the output, so that a vector read from shared memory serves several
// multiply-adds, two of them an instruction (two rows' scores, two columns' sums).  Float32 throughout, each sum in the row kernel's order: a
// score is one chain over the head, chunks of 32 keys from position 0 on set the running maximum and add their weights as
// a warp's tree does.  So a row's result is the same bits in either kernel, and does not depend on how its prompt was cut.
// What bounds it: shared memory (a read of 16 bytes a lane takes four cycles of the SM's one port, whatever lanes share), and in short
// prompts the chain of one block's tiles.  B200, row kernel -> this (us): 24 heads of 64 over 8, a prompt of 64 rows 15.5 -> 8.2, 301 62 -> 33, 600
// 148 -> 82, 1,200 437 -> 232, 128 rows after 2,000 381 -> 191; 36 heads, 301 rows 88 -> 40; 32 heads of 128 over 2, 200 rows 64 -> 44, 301
// 113 -> 67; 8 of 128, 1,200 rows 409 -> 207.
//
// Keys that a row does not see have weight 0; where one of their values is infinite or not a number, the chunk's products leave them out.
#include "common.cuh"
#include "host_rules.h"

JK_EXPORT int jk_attention_f32_supports(int dh, int dv) { return (dh == 64 || dh == 128) && (dv == 0 || dv == dh); }

namespace {

constexpr int AF_KEYS = 64, AF_WARPS = 4, AF_P = AF_KEYS + 4;

struct AfArgs {
    const float *q, *k_pages, *v_pages;
    float *out;
    const int *tiles, *req_start, *req_pos, *block_table;
    int nh, nkvh, page_shift, max_blocks;
    float scale;
};

__device__ __forceinline__ void af_copy16(float *to, const float *from, bool valid) {
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from), "r"(bytes) : "memory");
}
__device__ __forceinline__ void af_fma2(unsigned long long &acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long af_pair(float x) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float af_lo(unsigned long long v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float af_hi(unsigned long long v) { return __uint_as_float((unsigned)(v >> 32)); }

template <int DH, int RL> struct AfSmem {
    static constexpr int LD = DH + 4;        // eight lanes that read eight rows touch every bank once
    static constexpr int LDQ = 2 * DH + 4;   // two rows of q, element by element side by side
    float q[8 * RL * LDQ], k[2][AF_KEYS * LD], v[2][AF_KEYS * DH], p[AF_WARPS][4 * RL * AF_P];
};

// RL: rows a lane
template <int DH, int RL>
__global__ void __launch_bounds__(AF_WARPS * 32) attention_f32_kernel(AfArgs a) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) unsigned char af_raw[];
    using Smem = AfSmem<DH, RL>;
    constexpr int AF_ROWS = 16 * RL, WR = 4 * RL, LD = Smem::LD, LDQ = Smem::LDQ, CHUNKS = DH / 4, PASS = AF_WARPS * 32 / CHUNKS, CN = DH / 32;
    Smem &s = *reinterpret_cast<Smem *>(af_raw);
    const int *tile = a.tiles + 2 * (blockIdx.x / (jk::TILE_ROWS / AF_ROWS));
    const int req = tile[0], row0 = tile[1] + blockIdx.x % (jk::TILE_ROWS / AF_ROWS) * AF_ROWS;
    const int first = a.req_start[req], end = a.req_start[req + 1];
    if (row0 >= end) return;
    const int rows = min(AF_ROWS, end - row0), pos0 = a.req_pos[req] + row0 - first, last = pos0 + rows - 1;
    const int h = blockIdx.y, hk = h / (a.nh / a.nkvh), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int *bt = a.block_table + (size_t)req * a.max_blocks;
    const int chunk = threadIdx.x % CHUNKS * 4, line = threadIdx.x / CHUNKS;
    // a lane looks up the page of two keys of a tile, one tile ahead of its copies
    int page[2];
    auto look = [&](int j0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) page[i] = bt[min(j0 + lane + 32 * i, last) >> a.page_shift];
    };
    auto bring = [&](int stage, int j0) {
#pragma unroll
        for (int i = 0; i < AF_KEYS / PASS; ++i) {
            const int r = line + i * PASS, j = min(j0 + r, last);
            const int where = __shfl_sync(0xffffffffu, i * PASS < 32 ? page[0] : page[1], r & 31);
            const size_t at = ((((size_t)where * a.nkvh + hk) << a.page_shift) + (j & ((1 << a.page_shift) - 1))) * DH + chunk;
            af_copy16(s.k[stage] + r * LD + chunk, a.k_pages + at, j0 + r <= last);
            af_copy16(s.v[stage] + r * DH + chunk, a.v_pages + at, j0 + r <= last);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    look(0);
    bring(0, 0);
    look(AF_KEYS);
    for (int i = line; i < AF_ROWS / 2; i += PASS) {
        const float *from = a.q + ((size_t)row0 * a.nh + h) * DH + chunk;
        const float4 x = *reinterpret_cast<const float4 *>(from + (size_t)min(2 * i, rows - 1) * a.nh * DH);
        const float4 y = *reinterpret_cast<const float4 *>(from + (size_t)min(2 * i + 1, rows - 1) * a.nh * DH);
        float4 *to = reinterpret_cast<float4 *>(s.q + i * LDQ + 2 * chunk);
        to[0] = make_float4(x.x, y.x, x.y, y.y);
        to[1] = make_float4(x.z, y.z, x.w, y.w);
    }
    const int rg = lane >> 3, cg = lane & 7, mine = warp * WR + rg * RL;      // this lane's rows of the tile, RL from here on
    float m[RL], l[RL];
    unsigned long long o[RL][2 * CN];
#pragma unroll
    for (int r = 0; r < RL; ++r) {
        m[r] = -INFINITY;
        l[r] = 0.f;
#pragma unroll
        for (int c = 0; c < 2 * CN; ++c) o[r][c] = 0ull;
    }
    float *p = s.p[warp];
    int stage = 0;
    for (int j0 = 0; j0 <= last; j0 += AF_KEYS, stage ^= 1) {
        if (j0 + AF_KEYS <= last) {
            bring(stage ^ 1, j0 + AF_KEYS);
            look(j0 + 2 * AF_KEYS);
        }
        else asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();
        const int top_pos = pos0 + warp * WR + WR - 1;      // of the warp's last row
        if (j0 <= top_pos) {
            const float *ks = s.k[stage] + cg * LD, *qs = s.q + mine / 2 * LDQ;
            unsigned long long sc[RL / 2][8];               // two rows side by side
#pragma unroll
            for (int r = 0; r < RL / 2; ++r)
#pragma unroll
                for (int j = 0; j < 8; ++j) sc[r][j] = 0ull;
#pragma unroll 2
            for (int e = 0; e < DH; e += 4) {
                ulonglong2 q[RL / 2][2];
#pragma unroll
                for (int r = 0; r < RL / 2; ++r)
#pragma unroll
                    for (int i = 0; i < 2; ++i) q[r][i] = *reinterpret_cast<const ulonglong2 *>(qs + r * LDQ + 2 * e + 4 * i);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float4 k = *reinterpret_cast<const float4 *>(ks + j * 8 * LD + e);
                    const unsigned long long k0 = af_pair(k.x), k1 = af_pair(k.y), k2 = af_pair(k.z), k3 = af_pair(k.w);
#pragma unroll
                    for (int r = 0; r < RL / 2; ++r) af_fma2(sc[r][j], q[r][0].x, k0);
#pragma unroll
                    for (int r = 0; r < RL / 2; ++r) af_fma2(sc[r][j], q[r][0].y, k1);
#pragma unroll
                    for (int r = 0; r < RL / 2; ++r) af_fma2(sc[r][j], q[r][1].x, k2);
#pragma unroll
                    for (int r = 0; r < RL / 2; ++r) af_fma2(sc[r][j], q[r][1].y, k3);
                }
            }
            // the row kernel's chunks of 32 keys, one after the other
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                const int k0 = j0 + 32 * part;
                if (k0 > top_pos) break;
                const bool masked = k0 + 31 > pos0 + warp * WR;       // some row of the warp does not see all of the chunk
#pragma unroll
                for (int r = 0; r < RL; ++r) {
                    const int pos = pos0 + mine + r;
                    float x[4], top = -INFINITY;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const unsigned long long both = sc[r / 2][4 * part + j];
                        x[j] = __fmul_rn(r % 2 ? af_hi(both) : af_lo(both), a.scale);
                        if (!masked || k0 + cg + 8 * j <= pos) top = fmaxf(top, x[j]);
                    }
#pragma unroll
                    for (int k = 4; k > 0; k >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, k));
                    const float m_new = fmaxf(m[r], top), corr = expf(__fsub_rn(m[r], m_new));
                    m[r] = m_new;
                    float w[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        w[j] = masked && k0 + cg + 8 * j > pos ? 0.f : expf(__fsub_rn(x[j], m_new));
                        p[(rg * RL + r) * AF_P + 32 * part + cg + 8 * j] = w[j];
                    }
                    float sum = (w[0] + w[2]) + (w[1] + w[3]);        // a warp's tree over the 32 keys
#pragma unroll
                    for (int k = 4; k > 0; k >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, k);
                    l[r] = fmaf(l[r], corr, sum);
                    const unsigned long long c2 = af_pair(corr);
#pragma unroll
                    for (int c = 0; c < 2 * CN; ++c) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(o[r][c]) : "l"(c2));
                }
                __syncwarp();
                const float *vs = s.v[stage] + 32 * part * DH + cg * 4, *ps = p + rg * RL * AF_P + 32 * part;
                bool whole = true;
                if (masked) {
                    float sum[4] = {0.f, 0.f, 0.f, 0.f};                 // stay 0 unless a value is infinite or not a number
#pragma unroll 8
                    for (int i = lane * 4; i < 32 * DH; i += 128) {
                        const float4 v = *reinterpret_cast<const float4 *>(s.v[stage] + 32 * part * DH + i);
                        sum[0] = fmaf(v.x, 0.f, sum[0]); sum[1] = fmaf(v.y, 0.f, sum[1]);
                        sum[2] = fmaf(v.z, 0.f, sum[2]); sum[3] = fmaf(v.w, 0.f, sum[3]);
                    }
                    whole = __all_sync(0xffffffffu, (sum[0] + sum[1]) + (sum[2] + sum[3]) == 0.f);
                }
                if (whole) {
#pragma unroll 2
                    for (int j = 0; j < 32; j += 4) {
                        float w[RL][4];
#pragma unroll
                        for (int r = 0; r < RL; ++r) *reinterpret_cast<float4 *>(w[r]) = *reinterpret_cast<const float4 *>(ps + r * AF_P + j);
#pragma unroll
                        for (int i = 0; i < 4; ++i)
#pragma unroll
                            for (int c = 0; c < CN; ++c) {
                                const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(vs + (j + i) * DH + 32 * c);
#pragma unroll
                                for (int r = 0; r < RL; ++r) {
                                    const unsigned long long w2 = af_pair(w[r][i]);
                                    af_fma2(o[r][2 * c], w2, v.x);
                                    af_fma2(o[r][2 * c + 1], w2, v.y);
                                }
                            }
                    }
                } else {
                    for (int j = 0; j < 32; ++j)
#pragma unroll
                        for (int r = 0; r < RL; ++r)
                            if (k0 + j <= pos0 + mine + r) {
                                const unsigned long long w = af_pair(ps[r * AF_P + j]);
#pragma unroll
                                for (int c = 0; c < CN; ++c) {
                                    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(vs + j * DH + 32 * c);
                                    af_fma2(o[r][2 * c], w, v.x);
                                    af_fma2(o[r][2 * c + 1], w, v.y);
                                }
                            }
                }
            }
        }
        __syncthreads();
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
    for (int r = 0; r < RL; ++r) {
        if (mine + r >= rows) continue;
        const float inv = 1.f / l[r];
        float *to = a.out + ((size_t)(row0 + mine + r) * a.nh + h) * DH + cg * 4;
#pragma unroll
        for (int c = 0; c < CN; ++c)
            *reinterpret_cast<float4 *>(to + 32 * c) = make_float4(af_lo(o[r][2 * c]) * inv, af_hi(o[r][2 * c]) * inv, af_lo(o[r][2 * c + 1]) * inv, af_hi(o[r][2 * c + 1]) * inv);
    }
}

}  // namespace

// q, out [T, nh, dh]; tiles [ntiles][2]: batch entry, first row (jk::TILE_ROWS rows each)
JK_EXPORT int jk_attention_f32(const float *q, const float *k_pages, const float *v_pages, float *out, const int *tiles, int ntiles, const int *req_start, const int *req_pos,
                               const int *block_table, int max_blocks, int page_size, int nh, int nkvh, int dh, float scale, cudaStream_t stream) {
    if (ntiles == 0) return JK_OK;
    JK_REQUIRE(q && k_pages && v_pages && out && tiles && req_start && req_pos && block_table, "attention_f32: an argument is missing");
    JK_REQUIRE(jk_attention_f32_supports(dh, dh) && ntiles > 0 && nkvh > 0 && nh % nkvh == 0 && nh <= 65535 && page_size > 0 && (page_size & (page_size - 1)) == 0 && max_blocks > 0,
               "attention_f32: heads %d/%d of %d, page size %d", nh, nkvh, dh, page_size);
    JK_REQUIRE((((uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages | (uintptr_t)out) & 15) == 0, "attention_f32: operands must be 16-byte aligned");
    int shift = 0;
    while ((1 << shift) < page_size) ++shift;
    const AfArgs a{q, k_pages, v_pages, out, tiles, req_start, req_pos, block_table, nh, nkvh, shift, max_blocks, scale};
    auto run = [&](auto kernel, size_t smem, int rows) -> int {
        const dim3 grid(ntiles * (jk::TILE_ROWS / rows), nh);
        const cudaError_t e = cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) JK_FAIL(JK_CUDA_ERROR, "attention_f32: %s", cudaGetErrorString(e));
        jk_launch(kernel, grid, dim3(AF_WARPS * 32), smem, stream, a);
        JK_CHECK_LAUNCH("attention_f32");
        return JK_OK;
    };
    if (jk::attention_f32_tall(2LL * ntiles * nh, dh)) return dh == 64 ? run(attention_f32_kernel<64, 4>, sizeof(AfSmem<64, 4>), 64) : run(attention_f32_kernel<128, 4>, sizeof(AfSmem<128, 4>), 64);
    return dh == 64 ? run(attention_f32_kernel<64, 2>, sizeof(AfSmem<64, 2>), 32) : run(attention_f32_kernel<128, 2>, sizeof(AfSmem<128, 2>), 32);
}
