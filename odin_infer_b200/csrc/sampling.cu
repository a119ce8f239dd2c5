// Sampling over rows of 32-bit logits, one thread block per sequence.
//
// Restates sampler/sampler.odin on the device:
//   argmax: the first maximum wins (strict >, :79-89);
//   temperature: logits / T, softmax with the maximum subtracted, one coin in
//     [0,1) per token, walk of the cumulative sum in index order (:91-100, :179-185);
//   top-p: keep the most probable tokens until their sum first exceeds topp, scale the
//     coin by that sum and walk the kept ones in order of falling probability (:106-139);
//   repetition penalty: each distinct recent token has a positive logit divided
//     and a negative one multiplied (:143-160).
// The logits are never modified by the sampling kernels (the reference
// overwrites the caller's logits with probabilities; this does not).
// All sums run in an order fixed by the block size, so a seed gives the same
// tokens whatever else is in the batch.
#include <cooperative_groups.h>

#include "common.cuh"
#include <math_constants.h>

#define SB 1024  // threads per block

// ------------------------------------------------------------------ argmax
__global__ void __launch_bounds__(SB) argmax_kernel(const float* __restrict__ logits, size_t ld, int V,
                                                    int* __restrict__ out) {
    __shared__ float sv[32];
    __shared__ int si[32];
    pdl_trigger();
    pdl_wait();
    const float* row = logits + (size_t)blockIdx.x * ld;
    float best = -CUDART_INF_F;
    int bi = 0x7fffffff;
    for (int i = threadIdx.x; i < V; i += SB) {
        const float v = row[i];
        if (v > best || bi == 0x7fffffff) { best = v; bi = i; }
    }
    // NaN-free logits assumed; ties go to the lower index.
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { sv[warp] = best; si[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        best = sv[lane];
        bi = si[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        if (lane == 0) out[blockIdx.x] = (bi == 0x7fffffff) ? 0 : bi;
    }
}

// The same for long rows: a cluster of blocks shares a row, and the blocks' maxima meet through distributed shared memory.  One SM
// reads a row at its own rate: 151,936 logits of 1, 16 and 64 rows 6.9, 7.8 and 11.2 us; shared 3.5, 4.5 and 9.3.  The two
// meetings of a cluster cost what they save at 16,384 (1 row: 2.1 and 2.4) and with many rows, where the blocks come in rounds
// (32 rows of 32,768: 3.3 and 3.3, 64: 4.1 and 5.4; of 65,536: 4.5 and 3.7, 6.1 and 6.0; 128 of 151,936: 14.4 and 15.6).
constexpr int AM_BLOCKS = 8;        // of a row
constexpr int AM_THREADS = 512;
constexpr int AM_FROM = 32768;      // shorter rows are a block's work
constexpr int AM_PER_ROW = 2048;    // logits of a row for each of the rows, at least

__global__ void __launch_bounds__(AM_THREADS) argmax_cluster_kernel(const float* __restrict__ logits, size_t ld, int V, int vec,
                                                                    int* __restrict__ out) {
    namespace cg = cooperative_groups;
    __shared__ float sv[AM_THREADS / 32];
    __shared__ int si[AM_THREADS / 32];
    __shared__ float block_v;
    __shared__ int block_i;
    pdl_trigger();
    pdl_wait();
    cg::cluster_group cluster = cg::this_cluster();
    const float* row = logits + (size_t)blockIdx.y * ld;
    const int share = ((V + AM_BLOCKS - 1) / AM_BLOCKS + 3) / 4 * 4, i0 = (int)blockIdx.x * share, i1 = min(V, i0 + share);
    float best = -CUDART_INF_F;
    int bi = 0x7fffffff;
    auto take = [&](float v, int i) {
        if (v > best || bi == 0x7fffffff) { best = v; bi = i; }
    };
    if (vec) {
        constexpr int U = 4;   // vectors in flight
        for (int i = i0 + (int)threadIdx.x * 4; i < i1; i += AM_THREADS * 4 * U) {
            float4 q[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (i + u * AM_THREADS * 4 + 3 < i1) q[u] = *reinterpret_cast<const float4*>(row + i + u * AM_THREADS * 4);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int j = i + u * AM_THREADS * 4;
                if (j + 3 < i1) { take(q[u].x, j); take(q[u].y, j + 1); take(q[u].z, j + 2); take(q[u].w, j + 3); }
                else for (int k = j; k < i1; ++k) take(row[k], k);
            }
        }
    } else {
        for (int i = i0 + (int)threadIdx.x; i < i1; i += AM_THREADS) take(row[i], i);
    }
    auto meet = [&](int lanes) {   // ties go to the lower index
        for (int o = lanes / 2; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
    };
    meet(32);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { sv[warp] = best; si[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        best = lane < AM_THREADS / 32 ? sv[lane] : -CUDART_INF_F;
        bi = lane < AM_THREADS / 32 ? si[lane] : 0x7fffffff;
        meet(32);
        if (lane == 0) { block_v = best; block_i = bi; }
    }
    cluster.sync();
    if (blockIdx.x == 0 && warp == 0) {
        best = lane < AM_BLOCKS ? *cluster.map_shared_rank(&block_v, lane) : -CUDART_INF_F;
        bi = lane < AM_BLOCKS ? *cluster.map_shared_rank(&block_i, lane) : 0x7fffffff;
        meet(32);
        if (lane == 0) out[blockIdx.y] = (bi == 0x7fffffff) ? 0 : bi;
    }
    cluster.sync();   // no block leaves while its maximum is read
}

extern "C" int odin_argmax(const float* logits, long long ld, int B, int V, int* out, void* stream) {
    if (B <= 0) return 0;
    if (V <= 0) return ODIN_ERR_BAD_ARG;
    if (V >= AM_FROM && B <= V / AM_PER_ROW && B <= 65535) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(AM_BLOCKS, B);
        cfg.blockDim = dim3(AM_THREADS);
        cfg.stream = (cudaStream_t)stream;
        cudaLaunchAttribute attr[2] = {};
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = AM_BLOCKS;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = odin_pdl_enabled() ? 2 : 1;
        const int vec = ld % 4 == 0 && ((uintptr_t)logits & 15) == 0;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, argmax_cluster_kernel, logits, (size_t)ld, V, vec, out);
        if (e != cudaSuccess) return (int)e;
    } else {
        odin_launch(argmax_kernel, dim3(B), dim3(SB), 0, (cudaStream_t)stream, logits, (size_t)ld, V, out);
    }
    ODIN_LAUNCH_CHECK();
    return 0;
}

// ------------------------------------------------- temperature / top-p draw
__device__ __forceinline__ float block_max(float v, float* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_max(v);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    float t = red[lane];  // SB = 1024 threads = 32 warps
    return warp_max(t);
}

__device__ __forceinline__ void load16(const float* p, float (&v)[16]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) *reinterpret_cast<float4*>(v + 4 * q) = *reinterpret_cast<const float4*>(p + 4 * q);
}

// Sum of e_i = exp(l_i / T - m) over the tokens with e_i >= thr.
__device__ __forceinline__ float masked_sum(const float* row, int V, float inv_t, float m, float thr, float* red) {
    float s = 0.f;
    for (int i = threadIdx.x; i < V; i += SB) {
        const float e = expf(row[i] * inv_t - m);
        if (e >= thr) s += e;
    }
    return block_sum(s, red);
}

// P block-wide sums side by side, each in the order of block_sum.  What bounds a pass over a short row is not the row but
// the shuffles of its sums, two rounds of P x 5 in all 32 warps when every warp adds up for itself: here the warps beyond
// the row (their sums are zero) take no part in the first round, and one warp per sum does the second.  Draws from rows of
// 384: 57.5 us a launch with one block sum after the other, 52.8 so.
// red: [P][32], tot: [P].
template <int P>
__device__ __forceinline__ void block_sums(float (&v)[P], int V, float (*red)[32], float* tot) {
    static_assert(P <= 32, "a warp per sum");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp * 32 < V) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int q = 0; q < P; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
    }
#pragma unroll
    for (int q = 0; q < P; ++q)
        if (lane == q) red[q][warp] = v[q];
    __syncthreads();
    if (warp < P) {
        const float t = warp_sum(red[warp][lane]);  // SB = 1024 threads = 32 warps
        if (lane == 0) tot[warp] = t;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < P; ++q) v[q] = tot[q];
}

// The largest t in [lo, hi] (bit patterns of positive floats, which order like the floats) with
// S(t) = sum of e_i >= t  >  target, given S(lo) > target.  S falls as t grows.  Eight probes per
// pass over the row, so 2^30 candidates take ten passes instead of thirty.
__device__ unsigned search_threshold(const float* row, int V, float inv_t, float m, float target, unsigned lo,
                                     unsigned hi, float (*red)[32], float* tot) {
    constexpr int P = 8;
    while (lo < hi) {
        const unsigned span = hi - lo;  // probes lo < p_0 < ... <= hi
        unsigned probe[P];
        float acc[P];
#pragma unroll
        for (int q = 0; q < P; ++q) {
            probe[q] = lo + (unsigned)(((unsigned long long)span * (q + 1) + P - 1) / P);
            acc[q] = 0.f;
        }
        for (int i = threadIdx.x; i < V; i += SB) {
            const float e = expf(row[i] * inv_t - m);
#pragma unroll
            for (int q = 0; q < P; ++q)
                if (e >= __uint_as_float(probe[q])) acc[q] += e;
        }
        block_sums<P>(acc, V, red, tot);
        int best = -1;
#pragma unroll
        for (int q = 0; q < P; ++q)
            if (acc[q] > target) best = q;  // S is monotone: the last probe that still exceeds the target
        if (best < 0) hi = probe[0] - 1;
        else {
            if (best + 1 < P) hi = probe[best + 1] - 1;
            lo = probe[best];
        }
    }
    return lo;
}

// Temperature draw.  Without top-p: the cumulative sum is walked in index order (sample_mult,
// sampler/sampler.odin:91-100).  With 0 < top_p < 1 the reference sorts the candidates by falling
// probability, cuts after the first whose cumulative sum exceeds topp, scales the coin by that sum and
// walks the sorted list (sample_topp, :106-139).  Here nothing is sorted: the token at which a walk in
// falling order crosses a mark r is the one with the largest value u such that the tokens of at least
// that value sum to more than r, which a search over u finds (ties: in index order).  So the same coin
// gives the reference's token, up to the rounding of the sums and the order among exactly equal
// probabilities, which the reference's unstable sort leaves open.
__global__ void __launch_bounds__(SB) sample_kernel(const float* __restrict__ logits, size_t ld, int V,
                                                    float temperature, float top_p,
                                                    const float* __restrict__ coins, int* __restrict__ out) {
    __shared__ float red[32];
    __shared__ float reds[8][32], tots[8];
    __shared__ __align__(16) float chunk_sum[SB];
    __shared__ int chosen;
    pdl_trigger();
    pdl_wait();
    const float* row = logits + (size_t)blockIdx.x * ld;
    const float inv_t = 1.0f / temperature;
    float mx = -CUDART_INF_F;
    for (int i = threadIdx.x; i < V; i += SB) mx = fmaxf(mx, row[i] * inv_t);
    mx = block_max(mx, red);
    const float total = masked_sum(row, V, inv_t, mx, 0.f, red);
    const int per = (V + SB - 1) / SB;  // contiguous chunk of the row per thread, for walks in index order
    const int c0 = min(V, (int)threadIdx.x * per), c1 = min(V, c0 + per);
    if (threadIdx.x == 0) chosen = -1;

    if (top_p > 0.f && top_p < 1.f && V > 1) {
        // everything in units of e (unnormalised probabilities)
        const float cutoff = (1.0f - top_p) / (float)(V - 1) * total;
        const float target = top_p * total;
        const float s_cut = masked_sum(row, V, inv_t, mx, cutoff, red);
        unsigned lo = __float_as_uint(fmaxf(cutoff, 1e-45f));
        float cumulative = s_cut;  // the candidates together do not exceed topp: all of them stay
        if (s_cut > target) {
            // v: the value of the candidate at which the cumulative sum first exceeds topp
            lo = search_threshold(row, V, inv_t, mx, target, lo, __float_as_uint(1.0f), reds, tots);
            const float v = __uint_as_float(lo);
            const float above = masked_sum(row, V, inv_t, mx, __uint_as_float(lo + 1), red);
            const float ties = floorf((target - above) / v) + 1.0f;  // how many of value v it takes
            cumulative = above + fmaxf(ties, 1.0f) * v;
        }
        const float r = coins[blockIdx.x] * cumulative;
        unsigned ub = lo;
        float u = __uint_as_float(lo);
        int nth = 0x7fffffff;  // which of the tokens of value u, in index order (beyond their number: the last)
        if (masked_sum(row, V, inv_t, mx, u, red) > r) {
            ub = search_threshold(row, V, inv_t, mx, r, lo, __float_as_uint(1.0f), reds, tots);
            u = __uint_as_float(ub);
            const float above = masked_sum(row, V, inv_t, mx, __uint_as_float(ub + 1), red);
            nth = (int)fminf(floorf(fmaxf(r - above, 0.f) / u), 2.0e9f);
        }
        // the nth token (from 0) whose e is exactly u, else the last such one; if u is below every
        // candidate (the coin scaled to the whole sum), the smallest candidate's last occurrence
        float cnt = 0.f;
        for (int i = c0; i < c1; ++i) cnt += (expf(row[i] * inv_t - mx) == u) ? 1.f : 0.f;
        chunk_sum[threadIdx.x] = cnt;
        __syncthreads();
        if (threadIdx.x == 0) {
            int seen = 0, owner = -1, last_owner = -1;
            for (int t0 = 0; t0 < SB && owner < 0; t0 += 16) {
                float c16[16];  // the walk's loads sixteen at a time, so that it does not wait for each
                load16(chunk_sum + t0, c16);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int c = (int)c16[j];
                    if (owner >= 0) continue;
                    if (c > 0) last_owner = t0 + j;
                    if (seen + c > nth) owner = t0 + j;
                    else seen += c;
                }
            }
            if (owner < 0) { owner = last_owner; seen = 0x7fffffff; }
            if (owner >= 0) {
                const int o0 = min(V, owner * per), o1 = min(V, o0 + per);
                int pick = -1;
                for (int i = o0; i < o1; ++i) {
                    if (expf(row[i] * inv_t - mx) == u) {
                        pick = i;
                        if (seen != 0x7fffffff && seen++ == nth) break;
                    }
                }
                chosen = pick;
            }
        }
        __syncthreads();
        if (chosen < 0) {
            // no token of value u (u was the cutoff itself): the smallest candidate, the reference's last_idx
            float best = CUDART_INF_F;
            for (int i = threadIdx.x; i < V; i += SB) {
                const float e = expf(row[i] * inv_t - mx);
                if (e >= u) best = fminf(best, e);
            }
            best = -block_max(-best, red);
            int last = -1;
            for (int i = threadIdx.x; i < V; i += SB)
                if (expf(row[i] * inv_t - mx) == best) last = max(last, i);
            const float lf = block_max((float)last, red);
            if (threadIdx.x == 0) chosen = (int)lf;
            __syncthreads();
        }
        if (threadIdx.x == 0) out[blockIdx.x] = max(chosen, 0);
        return;
    }

    // ---- all tokens, cumulative walk in index order: contiguous chunk per thread, then a scan
    const float target = coins[blockIdx.x] * total;
    float cs = 0.f;
    for (int i = c0; i < c1; ++i) cs += expf(row[i] * inv_t - mx);
    chunk_sum[threadIdx.x] = cs;
    __syncthreads();
    if (threadIdx.x == 0) {
        // serial exclusive scan over 1024 chunk sums: fixed order
        float run = 0.f;
        int owner = -1;
        for (int t0 = 0; t0 < SB && owner < 0; t0 += 16) {
            float c16[16];
            load16(chunk_sum + t0, c16);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (owner >= 0) continue;
                const float nxt = run + c16[j];
                if (target < nxt) owner = t0 + j;
                else run = nxt;
            }
        }
        if (owner >= 0) {
            const int o0 = min(V, owner * per), o1 = min(V, o0 + per);
            float cdf = run;
            int pick = -1;
            for (int i = o0; i < o1; ++i) {
                cdf += expf(row[i] * inv_t - mx);
                if (target < cdf) { pick = i; break; }
            }
            chosen = (pick >= 0) ? pick : o1 - 1;
        }
    }
    __syncthreads();
    // rounding left the coin beyond the last sum: the last token (reference: n - 1)
    if (threadIdx.x == 0) out[blockIdx.x] = (chosen >= 0) ? chosen : V - 1;
}

// The same draw for rows of up to 1,024 candidates, one a thread: every thread adds up the values of at least its own from
// shared memory, so the mark's token is the largest value whose sum exceeds it and nothing is searched.  What bounds the
// search on a short row is its passes (two searches of ten, each with two block-wide meetings), not the row; here it is V
// compares and adds a thread and eight meetings.  One row of 128, 384 and 1,024: 27, 55 and 69 us searched, 3.8, 8.2 and 28.7 so; 64 rows
// 48, 57 and 94, and 4.1, 9.4 and 42.
constexpr int FEW_CANDIDATES = 1024;

__device__ __forceinline__ float block_max_few(float v, float* red) {   // of the launch's own number of warps
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    v = warp_max(v);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    return warp_max(lane < n_warps ? red[lane] : -CUDART_INF_F);
}

__global__ void __launch_bounds__(FEW_CANDIDATES) sample_few_kernel(const float* __restrict__ logits, size_t ld, int V, float temperature,
                                                                    float top_p, const float* __restrict__ coins, int* __restrict__ out) {
    __shared__ float red[32];
    __shared__ __align__(16) float es[FEW_CANDIDATES];
    __shared__ int chosen;
    pdl_trigger();
    pdl_wait();
    const int i = threadIdx.x;   // blockDim.x: V rounded up to whole warps
    const float inv_t = 1.0f / temperature;
    const float l = i < V ? logits[(size_t)blockIdx.x * ld + i] * inv_t : -CUDART_INF_F;
    const float coin = coins[blockIdx.x];
    const float mx = block_max_few(l, red);
    const float e = i < V ? expf(l - mx) : -1.0f;   // what lies beyond the row is below every value
    es[i] = e;
    if (i == 0) chosen = -1;
    __syncthreads();
    // the sum of the values of at least e: eight sums side by side, so that many equal small values add up without a drift
    float part[8] = {};
    for (int j = 0; j < (int)blockDim.x; j += 8) {
        const float4 q0 = *reinterpret_cast<const float4*>(es + j), q1 = *reinterpret_cast<const float4*>(es + j + 4);
        const float v[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
        for (int k = 0; k < 8; ++k) part[k] += v[k] >= e ? v[k] : 0.f;
    }
    const float from = ((part[0] + part[1]) + (part[2] + part[3])) + ((part[4] + part[5]) + (part[6] + part[7]));
    // (what lies above a value is what the next larger one sums to)
    const float total = block_max_few(e >= 0.f ? from : 0.f, red);
    const float cutoff = (1.0f - top_p) / (float)(V - 1) * total;
    const float target = top_p * total;
    float lo = fmaxf(cutoff, 1e-45f);
    float cumulative = block_max_few(e >= cutoff ? from : 0.f, red);   // the candidates' sum
    if (cumulative > target) {
        // the value of the candidate at which the cumulative sum first exceeds topp
        lo = fmaxf(block_max_few(e >= lo && from > target ? e : 0.f, red), lo);
        const float above = block_max_few(e > lo ? from : 0.f, red);
        const float ties = floorf((target - above) / lo) + 1.0f;
        cumulative = above + fmaxf(ties, 1.0f) * lo;
    }
    const float r = coin * cumulative;
    float u = block_max_few(e >= lo && from > r ? e : 0.f, red);
    int nth = 0x7fffffff;   // which of the tokens of value u, in index order (beyond their number: the last)
    if (u > 0.f) {
        const float above = block_max_few(e > u ? from : 0.f, red);
        nth = (int)fminf(floorf(fmaxf(r - above, 0.f) / u), 2.0e9f);
    } else {
        u = lo;
    }
    if (e == u) {
        int rank = 0, count = 0;
        for (int j = 0; j < V; ++j) {
            rank += es[j] == e && j < i;
            count += es[j] == e;
        }
        if (rank == min(nth, count - 1)) chosen = i;
    }
    __syncthreads();
    if (chosen < 0) {   // no token of value u (u was the cutoff itself): the smallest candidate's last occurrence
        const float best = -block_max_few(e >= u ? -e : -CUDART_INF_F, red);
        const float last = block_max_few(e == best ? (float)i : -1.0f, red);
        if (i == 0) chosen = (int)last;
        __syncthreads();
    }
    if (i == 0) out[blockIdx.x] = max(chosen, 0);
}

extern "C" int odin_sample(const float* logits, long long ld, int B, int V, float temperature, float top_p,
                           const float* coins, int* out, void* stream) {
    if (B <= 0) return 0;
    if (V <= 0 || !(temperature > 0.f)) return ODIN_ERR_BAD_ARG;
    if (V > 1 && V <= FEW_CANDIDATES && top_p > 0.f && top_p < 1.f)
        odin_launch(sample_few_kernel, dim3(B), dim3((V + 31) / 32 * 32), 0, (cudaStream_t)stream, logits, (size_t)ld, V, temperature,
                    top_p, coins, out);
    else
        odin_launch(sample_kernel, dim3(B), dim3(SB), 0, (cudaStream_t)stream, logits, (size_t)ld, V, temperature, top_p, coins, out);
    ODIN_LAUNCH_CHECK();
    return 0;
}

// ------------------------------------------------------ repetition penalty
// recent: [B, W] token ids, negative = empty.  logits are changed in place (the
// caller passes a copy).
__global__ void repetition_penalty_kernel(float* __restrict__ logits, size_t ld, int V,
                                          const int* __restrict__ recent, int W, float penalty) {
    pdl_trigger();
    pdl_wait();
    float* row = logits + (size_t)blockIdx.x * ld;
    const int* rec = recent + (size_t)blockIdx.x * W;
    for (int j = threadIdx.x; j < W; j += blockDim.x) {
        const int tok = rec[j];
        if (tok < 0 || tok >= V) continue;
        bool dup = false;
        for (int i = 0; i < j; ++i) dup |= (rec[i] == tok);
        if (dup) continue;
        const float v = row[tok];
        row[tok] = (v > 0.f) ? v / penalty : v * penalty;
    }
}

extern "C" int odin_repetition_penalty(float* logits, long long ld, int B, int V, const int* recent, int W,
                                       float penalty, void* stream) {
    if (B <= 0 || W <= 0) return 0;
    odin_launch(repetition_penalty_kernel, dim3(B), dim3(128), 0, (cudaStream_t)stream, logits, (size_t)ld, V, recent, W, penalty);
    ODIN_LAUNCH_CHECK();
    return 0;
}
