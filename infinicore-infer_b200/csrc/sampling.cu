// Sampling from rows of float32 logits: greedy, temperature, top-k, top-p.
//
// The reference hands one row of raw logits plus (random_val, topp, topk, temperature) to a
// library operator, once per request (src/models/jiuge/jiuge.cpp:282-289); temperature 0 or
// topk 1 means greedy (include/infinicore_infer/models/jiuge.h:85-87).  Here one block
// samples one row:
//   greedy       the largest logit, the lowest index among equals;
//   otherwise    w_i = exp((logit_i - max) / temperature); the candidate set is the largest
//                logits down to the first one at which either topk candidates or a share
//                topp of the whole mass is reached (candidates equal to that one included);
//                the token is the first candidate, in vocabulary order, whose running mass
//                exceeds u * (mass of the candidates).
// Masses are summed as 64-bit fixed point, so the result does not depend on the order in
// which threads add: the same (logits, u) always gives the same token.
#include "common.cuh"

JK_DEFINE_ERROR_BUFFER(jk_sampling)

constexpr int SAMPLE_THREADS = 1024;

__device__ __forceinline__ unsigned ordered_key(float f) {
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

struct ArgMax { float v; int i; };
__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
    if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
    return a;
}

__device__ int block_argmax(const float *row, int V, ArgMax *scratch) {
    ArgMax best{-INFINITY, 0x7fffffff};
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
        const float v = row[i];
        if (v > best.v || (v == best.v && i < best.i)) best = ArgMax{v, i};
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ArgMax other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
        best = better(best, other);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) scratch[warp] = best;
    __syncthreads();
    if (warp == 0) {
        ArgMax t = lane < (int)(blockDim.x >> 5) ? scratch[lane] : ArgMax{-INFINITY, 0x7fffffff};
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            ArgMax other{__shfl_xor_sync(0xffffffffu, t.v, o), __shfl_xor_sync(0xffffffffu, t.i, o)};
            t = better(t, other);
        }
        if (lane == 0) scratch[32] = t;
    }
    __syncthreads();
    int idx = scratch[32].i;
    if (idx == 0x7fffffff) idx = 0;     // a row of NaN or -inf only
    return idx;
}

__global__ void __launch_bounds__(SAMPLE_THREADS)
argmax_kernel(const float *__restrict__ logits, long long ld, int V, int *__restrict__ out) {
    pdl_trigger();
    pdl_wait();
    __shared__ ArgMax scratch[33];
    const int idx = block_argmax(logits + (size_t)blockIdx.x * ld, V, scratch);
    if (threadIdx.x == 0) out[blockIdx.x] = idx;
}

// Two stages for few rows of a large vocabulary: blocks take chunks of a row, then one block per row
// picks among the chunks' winners (the lowest index among equals in both stages).
constexpr int ARGMAX_CHUNK = 8192;

__global__ void __launch_bounds__(256)
argmax_chunks_kernel(const float *__restrict__ logits, long long ld, int V, ArgMax *__restrict__ part) {
    pdl_trigger();
    pdl_wait();
    __shared__ ArgMax scratch[33];
    const int r = blockIdx.y, c = blockIdx.x;
    const int lo = c * ARGMAX_CHUNK, n = min(ARGMAX_CHUNK, V - lo);
    const int idx = block_argmax(logits + (size_t)r * ld + lo, n, scratch);
    if (threadIdx.x == 0) part[(size_t)r * gridDim.x + c] = ArgMax{logits[(size_t)r * ld + lo + idx], lo + idx};
}

__global__ void argmax_merge_kernel(const ArgMax *__restrict__ part, int nchunks, int *__restrict__ out) {
    pdl_trigger();
    pdl_wait();
    const int r = blockIdx.x;
    ArgMax best{-INFINITY, 0x7fffffff};
    for (int i = threadIdx.x; i < nchunks; i += 32) best = better(best, part[(size_t)r * nchunks + i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ArgMax other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
        best = better(best, other);
    }
    if (threadIdx.x == 0) out[r] = best.i == 0x7fffffff ? 0 : best.i;
}

// Bytes of scratch that `jk_argmax` wants for this shape (0: it runs in one stage).
JK_EXPORT long long jk_argmax_scratch_bytes(int nrows, int V) {
    const int chunks = (V + ARGMAX_CHUNK - 1) / ARGMAX_CHUNK;
    if (chunks < 2 || nrows * 1 >= 148 * 2) return 0;
    return (long long)nrows * chunks * sizeof(ArgMax);
}

JK_EXPORT int jk_argmax(const float *logits, long long ld, int nrows, int V, int *out, void *scratch,
                        cudaStream_t stream) {
    if (nrows == 0) return JK_OK;
    JK_REQUIRE(nrows > 0 && V > 0 && ld >= V, "argmax: rows %d, vocabulary %d, stride %lld", nrows, V, ld);
    if (scratch != nullptr && jk_argmax_scratch_bytes(nrows, V) > 0) {
        const int chunks = (V + ARGMAX_CHUNK - 1) / ARGMAX_CHUNK;
        JK_REQUIRE(nrows <= 65535, "argmax: %d rows exceed one launch", nrows);
        jk_launch(argmax_chunks_kernel, dim3(chunks, nrows), dim3(256), 0, stream, logits, ld, V, (ArgMax *)scratch);
        JK_CHECK_LAUNCH("argmax_chunks");
        jk_launch(argmax_merge_kernel, dim3(nrows), dim3(32), 0, stream, (const ArgMax *)scratch, chunks, out);
        JK_CHECK_LAUNCH("argmax_merge");
        return JK_OK;
    }
    jk_launch(argmax_kernel, dim3(nrows), dim3(SAMPLE_THREADS), 0, stream, logits, ld, V, out);
    JK_CHECK_LAUNCH("argmax");
    return JK_OK;
}

__device__ __forceinline__ unsigned long long fixed_mass(float z, float m) {
    return (unsigned long long)(expf(z - m) * 4294967296.f);
}

// A row by one block.  The candidates' threshold is found in one of two ways that give the same key:
//   topk up to the block's threads: the topk-th largest of the threads' maxima is a bound that at least topk logits reach, so
//     the few logits above it are listed in one pass and everything else happens in that list, in shared memory;
//   else, or if the list overflows: passes over the row with a histogram of counts and masses per 11 bits of the key.
// What bounds it: passes over the row by one SM (294 KB at 73,440 logits, 5 us each) and, in the second way, atomics that meet in
// few bins.  B200, temperature 0.8, normal logits of spread 2, against four histogram passes, thread-long stretches of the row
// and loops of one thread over the shares (us): 22 rows of 73,440, topk 50 and topp 0.9 1,256 -> 33, topp 0.9 alone 1,280 -> 267,
// neither 176 -> 59; 64 rows of 122,753, topk 50 2,216 -> 48; 4 rows of 384 46 -> 12.
constexpr int SAMPLE_LIST = 2048, SAMPLE_BINS = 2048, SAMPLE_WARPS = SAMPLE_THREADS / 32;
struct SampleList { unsigned key[SAMPLE_LIST]; int index[SAMPLE_LIST]; unsigned long long mass[SAMPLE_LIST]; };
struct SampleBins { unsigned count[SAMPLE_BINS]; unsigned long long mass[SAMPLE_BINS]; };

// Inclusive sum over a warp's lanes 0 .. lane.
template <typename T> __device__ __forceinline__ T warp_prefix(T v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T other = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += other;
    }
    return v;
}

// OCC: blocks an SM that the registers must allow.  Two for more rows than there are SMs, whose second wave would otherwise run alone: 200
// rows of 122,753, greedy ones 97 -> 59 us, 200 of 384 with topp 64 -> 54; one for fewer, whose passes have more loads in flight (one row of
// 122,753, topk 50: 45 -> 43).
template <int OCC>
__global__ void __launch_bounds__(SAMPLE_THREADS, OCC)
sample_kernel(const float *__restrict__ logits, long long ld, int V,
              const float *__restrict__ temperature, const int *__restrict__ topk,
              const float *__restrict__ topp, const float *__restrict__ uniform,
              int *__restrict__ out) {
    pdl_trigger();
    pdl_wait();
    __shared__ ArgMax am_scratch[33];
    __shared__ float f_scratch[33];
    __shared__ union { SampleList list; SampleBins bins; } sh;
    __shared__ unsigned long long warp_mass[SAMPLE_WARPS], sh_mass;
    __shared__ unsigned warp_count[SAMPLE_WARPS], sh_n, sh_key;
    __shared__ int sh_pick;

    const int r = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float *row = logits + (size_t)r * ld;
    const float temp = temperature[r];
    const int k_in = topk[r];
    const float p_in = topp[r];
    auto greedy = [&] {
        const int idx = block_argmax(row, V, am_scratch);
        if (threadIdx.x == 0) out[r] = idx;
    };
    if (temp <= 0.f || k_in == 1) {
        greedy();
        return;
    }
    const float inv_t = 1.f / temp;
    float most = -INFINITY;
#pragma unroll 8
    for (int i = threadIdx.x; i < V; i += SAMPLE_THREADS) most = fmaxf(most, row[i] * inv_t);
    const float m = block_max(most, f_scratch);
    const bool cut_k = k_in > 1 && k_in < V, cut_p = p_in < 1.f;
    const unsigned kk = cut_k ? (unsigned)k_in : (unsigned)V;

    // a key that at least kk logits reach
    const bool listed = cut_k && kk <= SAMPLE_THREADS;
    unsigned bound = 0;
    if (listed) {
        const unsigned mine = ordered_key(most);
#pragma unroll 1
        for (int bit = 31; bit >= 0; --bit) {
            const unsigned trial = bound | 1u << bit;
            if (__syncthreads_count(mine >= trial) >= (int)kk) bound = trial;
        }
    }
    if (threadIdx.x == 0) { sh_n = 0; sh_key = 0; sh_pick = 0x7fffffff; sh_mass = 0; }
    __syncthreads();

    // the whole mass where a share of it, or all of it, is asked for; and the list
    unsigned long long sum = 0;
    const bool whole = cut_p || !cut_k;
    if (whole || listed) {
#pragma unroll 4
        for (int i0 = 0; i0 < V; i0 += SAMPLE_THREADS) {
            const int i = i0 + threadIdx.x;
            const float z = i < V ? row[i] * inv_t : 0.f;
            const unsigned key = ordered_key(z);
            if (whole && i < V) sum += fixed_mass(z, m);
            const bool in = listed && i < V && key >= bound;
            const unsigned who = __ballot_sync(0xffffffffu, in);
            if (who == 0) continue;
            unsigned at = 0;
            if (lane == 0) at = atomicAdd(&sh_n, (unsigned)__popc(who));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(who & ((1u << lane) - 1u));
            if (in && at < SAMPLE_LIST) { sh.list.key[at] = key; sh.list.index[at] = i; sh.list.mass[at] = fixed_mass(z, m); }
        }
        if (whole) {
            sum = warp_prefix(sum);
            if (lane == 31) atomicAdd(&sh_mass, sum);
        }
    }
    __syncthreads();
    const unsigned long long total = sh_mass;
    const unsigned long long limit = cut_p ? (unsigned long long)((double)fmaxf(p_in, 0.f) * (double)total) : ~0ull;
    float u = uniform[r];
    u = fminf(fmaxf(u, 0.f), 0.99999994f);

    if (listed && sh_n <= SAMPLE_LIST) {
        // an entry's key is low enough if the entries at or above it are enough, or heavy enough; the threshold is the highest such key
        const int n = (int)sh_n;
        for (int i = threadIdx.x; i < n; i += SAMPLE_THREADS) {
            const unsigned key = sh.list.key[i];
            unsigned c = 0;
            unsigned long long ms = 0;
            for (int j = 0; j < n; ++j)
                if (sh.list.key[j] >= key) { ++c; ms += sh.list.mass[j]; }
            if (c >= kk || ms >= limit) atomicMax(&sh_key, key);
        }
        __syncthreads();
        const unsigned tau = sh_key;
        unsigned long long cand = 0;
        for (int j = 0; j < n; ++j)
            if (sh.list.key[j] >= tau) cand += sh.list.mass[j];
        const unsigned long long target = (unsigned long long)((double)u * (double)cand);
        for (int i = threadIdx.x; i < n; i += SAMPLE_THREADS) {
            if (sh.list.key[i] < tau) continue;
            const int index = sh.list.index[i];
            unsigned long long cum = 0;
            for (int j = 0; j < n; ++j)
                if (sh.list.key[j] >= tau && sh.list.index[j] <= index) cum += sh.list.mass[j];
            if (cum > target) atomicMin(&sh_pick, index);
        }
        __syncthreads();
        if (sh_pick == 0x7fffffff) greedy();          // no mass at all (an infinite logit)
        else if (threadIdx.x == 0) out[r] = sh_pick;
        return;
    }

    unsigned tau = 0;                       // candidates: ordered_key >= tau
    unsigned long long cand_mass = total;
    if (cut_k || cut_p) {
        unsigned above = 0;                 // logits above the range of keys that is being divided, and their mass
        unsigned long long above_mass = 0;
        const int shifts[3] = {21, 10, 0}, widths[3] = {11, 11, 10};
#pragma unroll 1
        for (int pass = 0; pass < 3; ++pass) {
            const int shift = shifts[pass], top = shift + widths[pass];
            for (int b = threadIdx.x; b < SAMPLE_BINS; b += SAMPLE_THREADS) { sh.bins.count[b] = 0; sh.bins.mass[b] = 0; }
            __syncthreads();
#pragma unroll 4
            for (int i = threadIdx.x; i < V; i += SAMPLE_THREADS) {
                const float z = row[i] * inv_t;
                const unsigned key = ordered_key(z);
                if (pass == 0 || (key >> top) == (tau >> top)) {
                    const unsigned b = (key >> shift) & ((1u << widths[pass]) - 1u);
                    atomicAdd(&sh.bins.count[b], 1u);
                    atomicAdd(&sh.bins.mass[b], fixed_mass(z, m));
                }
            }
            __syncthreads();
            // thread t has bins 2047 - 2t and 2046 - 2t: sums from the highest bin down
            const int b1 = SAMPLE_BINS - 1 - 2 * threadIdx.x, b0 = b1 - 1;
            const unsigned c1 = sh.bins.count[b1], c0 = sh.bins.count[b0];
            const unsigned long long m1 = sh.bins.mass[b1], m0 = sh.bins.mass[b0];
            unsigned c = warp_prefix(c1 + c0);
            unsigned long long ms = warp_prefix(m1 + m0);
            if (lane == 31) { warp_count[warp] = c; warp_mass[warp] = ms; }
            if (threadIdx.x == 0) sh_key = 0;
            __syncthreads();
            c -= c1 + c0;
            ms -= m1 + m0;
            for (int w = 0; w < warp; ++w) { c += warp_count[w]; ms += warp_mass[w]; }
            // the highest bin that has logits and at which enough of them, or enough mass, is reached (+ 1: 0 stands for none)
            const bool at1 = c1 > 0 && (above + c + c1 >= kk || above_mass + ms + m1 >= limit);
            const bool at0 = c0 > 0 && (above + c + c1 + c0 >= kk || above_mass + ms + m1 + m0 >= limit);
            if (at1) atomicMax(&sh_key, (unsigned)b1 + 1u);
            else if (at0) atomicMax(&sh_key, (unsigned)b0 + 1u);
            __syncthreads();
            const int sel = max((int)sh_key - 1, 0);
            __syncthreads();
            if (b1 == sel) { sh_n = c; sh_mass = ms; }
            if (b0 == sel) { sh_n = c + c1; sh_mass = ms + m1; }
            __syncthreads();
            above += sh_n;
            above_mass += sh_mass;
            tau |= (unsigned)sel << shift;
            cand_mass = above_mass + sh.bins.mass[sel];
            __syncthreads();
        }
    }

    // the candidates in vocabulary order: a warp has a stretch of the row, the stretch that holds the token is walked once more
    const int seg = ((V + SAMPLE_WARPS - 1) / SAMPLE_WARPS + 31) / 32 * 32;
    const int s0 = min(V, warp * seg), s1 = min(V, s0 + seg);
    unsigned long long mine = 0;
#pragma unroll 4
    for (int i = s0 + lane; i < s1; i += 32) {
        const float z = row[i] * inv_t;
        if (ordered_key(z) >= tau) mine += fixed_mass(z, m);
    }
    mine = warp_prefix(mine);
    if (lane == 31) warp_mass[warp] = mine;
    __syncthreads();
    const unsigned long long target = (unsigned long long)((double)u * (double)cand_mass);
    unsigned long long cum = 0;
    for (int w = 0; w < warp; ++w) cum += warp_mass[w];
    if (cum <= target && cum + warp_mass[warp] > target) {         // one warp
        for (int i0 = s0; i0 < s1; i0 += 32) {
            const int i = i0 + lane;
            const float z = i < s1 ? row[i] * inv_t : 0.f;
            const unsigned long long w = i < s1 && ordered_key(z) >= tau ? fixed_mass(z, m) : 0ull, upto = cum + warp_prefix(w);
            const unsigned past = __ballot_sync(0xffffffffu, upto > target);
            if (past != 0) {
                if (lane == 0) sh_pick = i0 + __ffs(past) - 1;
                break;
            }
            cum = __shfl_sync(0xffffffffu, upto, 31);
        }
    }
    __syncthreads();
    if (sh_pick == 0x7fffffff) greedy();          // no mass at all (an infinite logit)
    else if (threadIdx.x == 0) out[r] = sh_pick;
}

JK_EXPORT int jk_sample(const float *logits, long long ld, int nrows, int V, const float *temperature,
                        const int *topk, const float *topp, const float *uniform, int *out,
                        cudaStream_t stream) {
    if (nrows == 0) return JK_OK;
    JK_REQUIRE(nrows > 0 && V > 0 && ld >= V, "sample: rows %d, vocabulary %d, stride %lld", nrows, V, ld);
    jk_launch(nrows > 148 ? sample_kernel<2> : sample_kernel<1>, dim3(nrows), dim3(SAMPLE_THREADS), 0, stream, logits, ld, V, temperature, topk, topp, uniform, out);
    JK_CHECK_LAUNCH("sample");
    return JK_OK;
}
