// Causal grouped-query attention over the paged cache on the CUDA cores: the 32-bit
// path's attention for prompts and decoding, and the bfloat16 path's fallback for
// head sizes that the tensor-core kernels refuse.
//
// Three kernels of the same arithmetic, operation by operation, so that in 32-bit they give
// the same bits: `attention_plain_kernel` (one warp per query token and head, takes
// everything), `attention_f32_single_kernel` (one token per sequence) and
// `attention_f32_tile_kernel` (prompts without a window or a chunk mask).
//
// Restates infer/forward.odin:88-115: query head h reads kv head h / (Hq/Hkv);
// score_t = (q . k_t) / sqrt(hd) for the keys t <= pos (the causal mask is the
// loop bound); softmax with the maximum subtracted (infer/ops.odin:21-37);
// out = sum_t p_t v_t.  The softmax runs "online" over chunks of 32 keys that
// start at the first visible key, so a token's result depends only on its own
// sequence and position.  A window > 0 hides keys t <= pos - window; a chunk > 0 hides the
// keys before the query's own chunk (position p sees t only if t / chunk == p / chunk, chunks
// counted from the sequence's first position).  scale > 0 replaces 1 / sqrt(hd); softcap > 0
// turns a score s into softcap * tanh(s / softcap) before the softmax.  A value head has vd
// elements (keys and queries hd).  sink (optional, one 32-bit number per query head): exp(sink[h]) is
// added to the softmax's denominator once.
#include "common.cuh"
#include "async_copy.cuh"
#include <math_constants.h>

#define AP_WARPS 4
#define AP_MAX_HD 1024

template <typename T>
__device__ __forceinline__ float dot_row(const float* __restrict__ q, const T* __restrict__ k, int hd);

template <>
__device__ __forceinline__ float dot_row<float>(const float* __restrict__ q, const float* __restrict__ k, int hd) {
    float acc = 0.f;
    if (hd & 3) {  // rows that are not whole vectors: one element at a time
        for (int i = 0; i < hd; ++i) acc = fmaf(q[i], k[i], acc);
        return acc;
    }
    const float4* k4 = reinterpret_cast<const float4*>(k);
    for (int i = 0; i < hd / 4; ++i) {
        const float4 v = k4[i];
        acc = fmaf(q[4 * i + 0], v.x, acc);
        acc = fmaf(q[4 * i + 1], v.y, acc);
        acc = fmaf(q[4 * i + 2], v.z, acc);
        acc = fmaf(q[4 * i + 3], v.w, acc);
    }
    return acc;
}

template <>
__device__ __forceinline__ float dot_row<bf16>(const float* __restrict__ q, const bf16* __restrict__ k, int hd) {
    float acc = 0.f;
    if (hd & 7) {  // rows that are not whole vectors: one element at a time
        for (int i = 0; i < hd; ++i) acc = fmaf(q[i], __bfloat162float(k[i]), acc);
        return acc;
    }
    const uint4* k8 = reinterpret_cast<const uint4*>(k);
    for (int i = 0; i < hd / 8; ++i) {
        const uint4 v = k8[i];
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 f = __bfloat1622float2(h[j]);
            acc = fmaf(q[8 * i + 2 * j], f.x, acc);
            acc = fmaf(q[8 * i + 2 * j + 1], f.y, acc);
        }
    }
    return acc;
}

// R: elements of a head that a lane holds (key and value heads of up to 32 R elements)
template <typename T, int R>
__global__ void __launch_bounds__(AP_WARPS * 32)
attention_plain_kernel(const T* __restrict__ q, size_t q_stride, T* __restrict__ out, size_t out_stride, int T_tok,
                       int Hq, int Hkv, int hd, int vd, const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                       int page_size, const int* __restrict__ tok_pos, const int* __restrict__ tok_seq,
                       const int* __restrict__ block_table, int bt_stride, int window, int chunk, float scale,
                       float softcap, const float* __restrict__ sink) {
    __shared__ float qs[AP_WARPS][32 * R];
    pdl_trigger();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long item = (long long)blockIdx.x * AP_WARPS + warp;
    if (item >= (long long)T_tok * Hq) return;
    const int t = (int)(item / Hq), h = (int)(item % Hq);
    const int seq = tok_seq[t];
    if (seq < 0) return;
    const int pos = tok_pos[t];
    const int kvh = h / (Hq / Hkv);
    const T* qrow = q + (size_t)t * q_stride + (size_t)h * hd;
    float* qf = qs[warp];
    for (int j = lane; j < hd; j += 32) qf[j] = to_f32(qrow[j]);
    __syncwarp();

    const float inv_scale = sqrtf((float)hd);
    int t_lo = 0;
    if (window > 0 && pos - window + 1 > 0) t_lo = pos - window + 1;
    if (chunk > 0) t_lo = max(t_lo, (pos / chunk) * chunk);

    float m = -CUDART_INF_F, l = 0.f;
    float acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.f;
    const int* bt = block_table + (size_t)seq * bt_stride;

    for (int t0 = t_lo; t0 <= pos; t0 += 32) {
        const int tk = t0 + lane;
        const bool valid = tk <= pos;
        long long row = -1;
        float s = -CUDART_INF_F;
        if (valid) {
            const int page = bt[tk / page_size];
            if (page >= 0) {
                row = ((long long)page * Hkv + kvh) * page_size + (tk % page_size);
                const float dot = dot_row<T>(qf, k_cache + (size_t)row * hd, hd);
                s = scale > 0.f ? dot * scale : dot / inv_scale;
                if (softcap > 0.f) s = softcap * tanhf(s / softcap);
            }
        }
        const float m_new = fmaxf(m, warp_max(s));
        if (m_new == -CUDART_INF_F) continue;  // no visible key in this chunk
        const float p = (row >= 0) ? expf(s - m_new) : 0.f;
        const float corr = expf(m - m_new);
        l = l * corr + warp_sum(p);
        m = m_new;
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] *= corr;
        const int n_here = min(32, pos - t0 + 1);
        for (int j = 0; j < n_here; ++j) {
            const float pj = __shfl_sync(0xffffffffu, p, j);
            const long long rj = __shfl_sync(0xffffffffu, row, j);
            if (rj < 0) continue;
            const T* vrow = v_cache + (size_t)rj * vd;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int d = r * 32 + lane;
                if (d < vd) acc[r] = fmaf(pj, to_f32(vrow[d]), acc[r]);
            }
        }
    }
    if (sink != nullptr) {
        // a learned logit per query head that enters the denominator alone: no key, no value, not scaled
        const float sk = sink[h];
        const float m_new = fmaxf(m, sk);
        const float corr = expf(m - m_new);
        l = l * corr + expf(sk - m_new);
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] *= corr;
    }
    T* orow = out + (size_t)t * out_stride + (size_t)h * vd;
    const float inv_l = (l > 0.f) ? 1.0f / l : 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int d = r * 32 + lane;
        if (d < vd) orow[d] = from_f32<T>(acc[r] * inv_l);
    }
}

// ---------------------------------------------------------------------------
// 32-bit kernels that share the keys and values among a kv head's query heads (and, for prompts, among tokens)
// ---------------------------------------------------------------------------
namespace {

struct F32Attn {
    const float* q;
    float* out;
    const float *k, *v;   // one layer of the cache
    const int *tok_pos, *tok_seq, *block_table;
    const float* sink;
    const int* seq_start;  // first token of every sequence and one past the last, or null
    size_t q_stride, out_stride;
    int T, Hq, Hkv, hd, page_size, bt_stride, window, chunk, n_seqs;
    float scale, softcap;
};

// One chunk of 32 keys of one row, lane = key, as attention_plain_kernel does it: s is the dot product (-inf where there
// is no key), m and l the row's running maximum and sum.  Returns p; corr is the factor on what was summed before.
__device__ __forceinline__ float chunk_softmax(float dot, bool key, float scale, float inv_scale, float softcap, float& m,
                                               float& l, float& corr) {
    float s = -CUDART_INF_F;
    if (key) {
        s = scale > 0.f ? dot * scale : dot / inv_scale;
        if (softcap > 0.f) s = softcap * tanhf(s / softcap);
    }
    const float m_new = fmaxf(m, warp_max(s));
    const bool any = m_new != -CUDART_INF_F;  // a key was visible, here or before
    const float p = key && any ? expf(s - m_new) : 0.f;
    corr = any ? expf(m - m_new) : 1.f;
    const float sum = warp_sum(p);
    l = any ? l * corr + sum : l;
    m = m_new;
    return p;
}

// ---- one token per sequence ------------------------------------------------
// A block per (token, kv head) takes the kv head's G query heads together.  Keys and values pass through shared memory
// in blocks of 64, the next block's copies in flight while this one is worked on (rows padded by 16 bytes, so that the
// lanes of a phase hit different bank groups): a thread per (key, head) forms the dot products, a warp per head the
// softmax of the two chunks of 32, a thread per (element, head) adds the values up.
// What bounds it: the chain of a block (hd multiply-adds of a dot product, two softmaxes one after the other, 64
// multiply-adds of a sum, four barriers: 3.3 us for 64 keys of 128, 1.8 of 16), not the keys' traffic.  16 query heads on 8
// kv heads of 128: sequences of 400, 287, 174 and 61 keys 24.8 us, 2,000 keys 106 us; 8 decode steps of four such
// sequences on the 1.7B size spend 5.6 ms here.
constexpr int SG_THREADS = 256;
constexpr int SG_KEYS = 64;
constexpr int SG_MAX_HD = 128;
constexpr int SG_MAX_G = 8;

__global__ void __launch_bounds__(SG_THREADS) attention_f32_single_kernel(const F32Attn a) {
    extern __shared__ __align__(16) float sm[];
    __shared__ __align__(16) float qs[SG_MAX_G][SG_MAX_HD];
    __shared__ __align__(16) float ps[SG_MAX_G][SG_KEYS];    // dot products, then probabilities
    __shared__ float corrs[SG_MAX_G][2];
    __shared__ float finals[SG_MAX_G][2];      // factor of the sink, 1 / denominator
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t = blockIdx.x / a.Hkv, kvh = blockIdx.x % a.Hkv;
    const int seq = a.tok_seq[t];
    if (seq < 0) return;
    const int pos = a.tok_pos[t], hd = a.hd, G = a.Hq / a.Hkv, pitch = hd + 4, pieces = hd / 4;
    int t_lo = 0;
    if (a.window > 0 && pos - a.window + 1 > 0) t_lo = pos - a.window + 1;
    if (a.chunk > 0) t_lo = max(t_lo, (pos / a.chunk) * a.chunk);
    const int* bt = a.block_table + (size_t)seq * a.bt_stride;
    const int n_blocks = (pos - t_lo) / SG_KEYS + 1;
    float* ring = sm;  // [2][keys | values][64][pitch]

    // the pages of a block's keys: it starts in page `at` of the sequence and ends there or (pages hold 64 keys or more)
    // in the next.  Their numbers are fetched a block ahead of the copies that need them.
    struct Pages {
        int at, first, second;
        __device__ __forceinline__ int of(int tk, int page_size, int& slot) const {
            const bool next = tk >= (at + 1) * page_size;
            slot = tk - (at + (next ? 1 : 0)) * page_size;
            return next ? second : first;
        }
    };
    auto pages_of = [&](int b) {
        Pages p;
        p.at = (t_lo + b * SG_KEYS) / a.page_size;
        const int last = pos / a.page_size;
        p.first = p.at <= last ? bt[p.at] : -1;
        p.second = p.at + 1 <= last ? bt[p.at + 1] : -1;
        return p;
    };
    const int i_step = SG_THREADS / pieces, i_first = tid / pieces, piece = tid - i_first * pieces;  // this thread's keys and piece
    auto load = [&](int b, const Pages& pages) {
        float* kd = ring + (size_t)(b & 1) * 2 * SG_KEYS * pitch + piece * 4;
        float* vd = kd + SG_KEYS * pitch;
        if (i_first >= i_step) return;  // 256 is no multiple of the pieces of a row: the rest of the threads copies nothing
#pragma unroll 4
        for (int i = i_first; i < SG_KEYS; i += i_step) {
            const int tk = t_lo + b * SG_KEYS + i;
            int slot;
            const int page = pages.of(tk, a.page_size, slot);
            const bool in = tk <= pos && page >= 0;
            const size_t off = in ? (((size_t)page * a.Hkv + kvh) * a.page_size + slot) * hd + piece * 4 : 0;
            cp16(kd + i * pitch, a.k + off, in);
            cp16(vd + i * pitch, a.v + off, in);
        }
    };
    Pages now = pages_of(0), next = pages_of(1);
    load(0, now);
    cp_commit();
    for (int c = tid; c < G * hd; c += SG_THREADS)
        qs[c / hd][c % hd] = a.q[(size_t)t * a.q_stride + (size_t)(kvh * G + c / hd) * hd + c % hd];
    const float inv_scale = sqrtf((float)hd);
    float m = -CUDART_INF_F, l = 0.f;               // of head `warp`
    constexpr int MAXO = SG_MAX_G * SG_MAX_HD / SG_THREADS;
    float acc[MAXO];
#pragma unroll
    for (int o = 0; o < MAXO; ++o) acc[o] = 0.f;

    for (int b = 0; b < n_blocks; ++b) {
        if (b + 1 < n_blocks) load(b + 1, next);
        cp_commit();
        const Pages after = pages_of(b + 2);
        cp_wait<1>();
        __syncthreads();
        const float* kd = ring + (size_t)(b & 1) * 2 * SG_KEYS * pitch;
        const float* vd = kd + SG_KEYS * pitch;
        for (int c = tid; c < SG_KEYS * G; c += SG_THREADS) {
            const int key = c & (SG_KEYS - 1), g = c / SG_KEYS;
            const float4* k4 = reinterpret_cast<const float4*>(kd + key * pitch);
            const float4* q4 = reinterpret_cast<const float4*>(qs[g]);
            float dot = 0.f;
#pragma unroll 8
            for (int i = 0; i < pieces; ++i) {
                const float4 kv = k4[i], qv = q4[i];
                dot = fmaf(qv.x, kv.x, dot);
                dot = fmaf(qv.y, kv.y, dot);
                dot = fmaf(qv.z, kv.z, dot);
                dot = fmaf(qv.w, kv.w, dot);
            }
            ps[g][key] = dot;
        }
        __syncthreads();
        if (warp < G) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int tk = t_lo + b * SG_KEYS + h * 32 + lane;
                int slot;
                const bool key = tk <= pos && now.of(tk, a.page_size, slot) >= 0;
                float corr;
                const float p = chunk_softmax(ps[warp][h * 32 + lane], key, a.scale, inv_scale, a.softcap, m, l, corr);
                ps[warp][h * 32 + lane] = p;
                if (lane == 0) corrs[warp][h] = corr;
            }
        }
        __syncthreads();
#pragma unroll
        for (int o = 0; o < MAXO; ++o) {
            const int c = o * SG_THREADS + tid;
            if (c >= G * hd) break;
            const int g = c / hd, d = c - g * hd;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                acc[o] *= corrs[g][h];
                // keys that are not there have p = 0 and a value row of zeros
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    const float4 p = *reinterpret_cast<const float4*>(&ps[g][h * 32 + j]);
                    const float* vr = vd + (h * 32 + j) * pitch + d;
                    acc[o] = fmaf(p.x, vr[0], acc[o]);
                    acc[o] = fmaf(p.y, vr[pitch], acc[o]);
                    acc[o] = fmaf(p.z, vr[2 * pitch], acc[o]);
                    acc[o] = fmaf(p.w, vr[3 * pitch], acc[o]);
                }
            }
        }
        __syncthreads();  // the buffer of block b is filled again two blocks on
        now = next;
        next = after;
    }
    cp_wait<0>();
    if (warp < G && lane == 0) {
        float corr = 1.f;
        if (a.sink != nullptr) {
            const float sk = a.sink[kvh * G + warp];
            const float m_new = fmaxf(m, sk);
            corr = expf(m - m_new);
            l = l * corr + expf(sk - m_new);
        }
        finals[warp][0] = corr;
        finals[warp][1] = (l > 0.f) ? 1.0f / l : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int o = 0; o < MAXO; ++o) {
        const int c = o * SG_THREADS + tid;
        if (c >= G * hd) break;
        const int g = c / hd, d = c - g * hd;
        float v = acc[o];
        if (a.sink != nullptr) v *= finals[g][0];
        a.out[(size_t)t * a.out_stride + (size_t)(kvh * G + g) * hd + d] = v * finals[g][1];
    }
}

// ---- prompts ---------------------------------------------------------------
// A block per (64 / G consecutive tokens, kv head): its 64 rows are (token, query head of the kv head), which share
// every chunk of 32 keys and values (two chunks in shared memory, the next one's copies in flight).  With seq_start a
// tile holds tokens of one sequence.  Where many bring a token or two behind long contexts, the sequences of a tile of
// consecutive tokens would be worked on one after the other: 31 sequences with one token and 2,000 keys beside a prompt
// of 2 take 0.66 ms so, 13.4 before and 1.4 in attention_plain_kernel; 16 sequences of 3 tokens with 300 keys 109 us,
// 768 and 121.  Without seq_start tiles are of consecutive tokens.  Per chunk: the 64 x 32 dot products, 4 x 2 a
// thread; the softmax, a warp per 8 rows, lane = key; the 64 x HD sums, 4 x HD / 16 a thread.  Rows of 16-byte pieces
// are stored at piece ^ (row & 7), and a warp is 8 x 4 threads laid out as in the tiles of gemm_plain.cu.
// No window and no chunk mask: every row's chunks then start at key 0, which is what lets rows share them and keeps the
// bits those of attention_plain_kernel.
// What bounds it: shared loads and multiply-adds, and on short prompts the tile that sees most keys.  16 query heads on 8
// kv heads of 128: one prompt of 2,000 tokens 693 us (862 with the tiles in order of their tokens), four of 61 to 400
// tokens 138 us (145 with tiles of consecutive tokens).
constexpr int TL_THREADS = 256;
constexpr int TL_ROWS = 64;
constexpr int TL_KEYS = 32;

// acc[i][..] += sum over the chunk's keys j, ascending, of p[16 i][j] v[j][64 d ..]; GUARD: only of the keys j <= last[i]
template <int HD, bool GUARD>
__device__ __forceinline__ void add_values(const float* p, const float* v, const int (&last)[4], float (&acc)[4][HD / 16]) {
    constexpr int SP = TL_KEYS + 4;
#pragma unroll 2
    for (int j0 = 0; j0 < TL_KEYS; j0 += 4) {
        float4 p4[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) p4[i] = *reinterpret_cast<const float4*>(p + 16 * i * SP + j0);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int d = 0; d < HD / 64; ++d) {
                const float4 w = *reinterpret_cast<const float4*>(v + (j0 + j) * HD + 64 * d);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (GUARD && j0 + j > last[i]) continue;
                    const float x = reinterpret_cast<const float*>(&p4[i])[j];
                    acc[i][4 * d] = fmaf(x, w.x, acc[i][4 * d]);
                    acc[i][4 * d + 1] = fmaf(x, w.y, acc[i][4 * d + 1]);
                    acc[i][4 * d + 2] = fmaf(x, w.z, acc[i][4 * d + 2]);
                    acc[i][4 * d + 3] = fmaf(x, w.w, acc[i][4 * d + 3]);
                }
            }
        }
    }
}

// The tokens [tok0, end) of the item-th tile: sequences from the last to the first, each in tiles of tt tokens from its
// first token on, its last tile first.  tok0 >= end beyond the last item.
__device__ __forceinline__ void tile_tokens(int item, int tt, const int* __restrict__ seq_start, int n_seqs, int tid, int& tok0, int& end) {
    __shared__ int warp_sums[TL_THREADS / 32];
    __shared__ int found[2];
    const int lane = tid & 31, warp = tid >> 5;
    if (tid == 0) found[0] = found[1] = 0;
    for (int b0 = 0; b0 < n_seqs; b0 += TL_THREADS) {   // thread: a sequence
        const int b = n_seqs - 1 - (b0 + tid);
        int first = 0, last = 0;
        if (b >= 0) {
            first = seq_start[b];
            last = seq_start[b + 1];
        }
        const int tiles = (last - first + tt - 1) / tt;
        int sum = tiles;   // of this sequence and those before it in the walk
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += x;
        }
        if (lane == 31) warp_sums[warp] = sum;
        __syncthreads();
        int total = 0;
        for (int w = 0; w < TL_THREADS / 32; ++w) {
            if (w < warp) sum += warp_sums[w];
            total += warp_sums[w];
        }
        const int mine = item - (sum - tiles);   // which of this sequence's tiles, from its last
        if (mine >= 0 && mine < tiles) {
            found[0] = first + (tiles - 1 - mine) * tt;
            found[1] = min(last, found[0] + tt);
        }
        __syncthreads();   // found; the warps' sums are written again
        if (item < total) break;
        item -= total;
    }
    tok0 = found[0];
    end = found[1];
}

template <int HD>
__global__ void __launch_bounds__(TL_THREADS, 2) attention_f32_tile_kernel(const F32Attn a) {
    constexpr int PIECES = HD / 4, DT = HD / 64;  // DT: groups of four elements that a thread sums
    constexpr int SP = TL_KEYS + 4;
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;                                // [64][HD]
    float* ring = qs + TL_ROWS * HD;               // [2][keys | values][32][HD]
    float* ss = ring + 4 * TL_KEYS * HD;           // [64][36]: dot products, then probabilities
    float* row_m = ss + TL_ROWS * SP;
    float* row_l = row_m + TL_ROWS;
    float* row_corr = row_l + TL_ROWS;
    int* row_pos = reinterpret_cast<int*>(row_corr + TL_ROWS);  // position of the row's token; -1: no row, or not of the sequence at work
    int* t_seq = row_pos + TL_ROWS;
    int* t_pos = t_seq + TL_ROWS;
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = (lane & 1) + 2 * (lane >> 4) + 4 * (warp & 3), ty = ((lane >> 1) & 7) + 8 * (warp >> 2);
    // the last tiles, whose tokens see most keys, first
    const int G = a.Hq / a.Hkv, tt = TL_ROWS / G, kvh = blockIdx.x % a.Hkv;
    __shared__ int first_token;   // kept here to the end, not in a register
    int tok0, end;                // this tile's tokens
    if (a.seq_start != nullptr) {
        tile_tokens((int)(blockIdx.x / a.Hkv), tt, a.seq_start, a.n_seqs, tid, tok0, end);
        if (tok0 >= end) return;
    } else {
        tok0 = (int)((gridDim.x - 1 - blockIdx.x) / a.Hkv) * tt;
        end = min(a.T, tok0 + tt);
    }
    if (tid == 0) first_token = tok0;
    const float inv_scale = sqrtf((float)HD);

    for (int i = tid; i < tt; i += TL_THREADS) {
        const bool in = tok0 + i < end;
        t_seq[i] = in ? a.tok_seq[tok0 + i] : -1;
        t_pos[i] = in ? a.tok_pos[tok0 + i] : -1;
    }
    // row r: token r / G, head r % G
    for (int c = tid; c < TL_ROWS * PIECES; c += TL_THREADS) {
        const int r = c / PIECES, piece = c % PIECES, tok = tok0 + r / G;
        const bool in = r < tt * G && tok < end;
        cp16(qs + r * HD + ((piece ^ (r & 7)) << 2),
             in ? a.q + (size_t)tok * a.q_stride + (size_t)(kvh * G + r % G) * HD + piece * 4 : a.q, in);
    }
    cp_commit();
    if (tid < TL_ROWS) {
        row_m[tid] = -CUDART_INF_F;
        row_l[tid] = 0.f;
    }
    float acc[4][4 * DT];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int d = 0; d < 4 * DT; ++d) acc[i][d] = 0.f;
    __syncthreads();

    for (int i0 = 0; i0 < tt;) {
        // the run of tokens of one sequence from i0 on, and its first and last position
        const int seq = t_seq[i0];
        int i1 = i0, lo = t_pos[i0], hi = t_pos[i0];
        for (; i1 < tt && t_seq[i1] == seq; ++i1) {
            lo = min(lo, t_pos[i1]);
            hi = max(hi, t_pos[i1]);
        }
        if (seq < 0) {
            i0 = i1;
            continue;
        }
        const bool whole = i0 == 0 && i1 * G == TL_ROWS;  // every row belongs to the run
        if (tid < TL_ROWS) row_pos[tid] = (tid / G >= i0 && tid / G < i1) ? t_pos[tid / G] : -1;
        const int* bt = a.block_table + (size_t)seq * a.bt_stride;
        const int n_chunks = hi / TL_KEYS + 1;
        auto page_of = [&](int b) { return b < n_chunks ? bt[b * TL_KEYS / a.page_size] : -1; };  // pages hold a multiple of 32 tokens
        auto load = [&](int b, int page) {
            float* kd = ring + (b & 1) * 2 * TL_KEYS * HD;
            float* vd = kd + TL_KEYS * HD;
            const size_t row0 = page >= 0 ? ((size_t)page * a.Hkv + kvh) * a.page_size + (b * TL_KEYS) % a.page_size : 0;
#pragma unroll
            for (int c = 0; c < TL_KEYS * PIECES / TL_THREADS; ++c) {
                const int e = c * TL_THREADS + tid, i = e / PIECES, piece = e % PIECES;
                const bool in = page >= 0 && b * TL_KEYS + i <= hi;
                const size_t off = in ? (row0 + i) * HD + piece * 4 : 0;
                cp16(kd + i * HD + ((piece ^ (i & 7)) << 2), a.k + off, in);
                cp16(vd + i * HD + piece * 4, a.v + off, in);
            }
        };
        int page = page_of(0), page_next = page_of(1);  // of chunks b and b + 1: fetched ahead of the copies that need them
        load(0, page);
        cp_commit();
        for (int b = 0; b < n_chunks; ++b) {
            const int t0 = b * TL_KEYS;
            if (b + 1 < n_chunks) load(b + 1, page_next);
            cp_commit();
            const int page_after = page_of(b + 2);
            cp_wait<1>();
            __syncthreads();
            const float* kd = ring + (b & 1) * 2 * TL_KEYS * HD;
            const float* vd = kd + TL_KEYS * HD;
            {   // dot products of rows ty + 16 i with keys tx + 16 j
                float s[4][2];
#pragma unroll
                for (int i = 0; i < 4; ++i) s[i][0] = s[i][1] = 0.f;
#pragma unroll 4
                for (int p = 0; p < PIECES; ++p) {
                    float4 k4[2], q4[4];
#pragma unroll
                    for (int j = 0; j < 2; ++j) k4[j] = *reinterpret_cast<const float4*>(kd + (tx + 16 * j) * HD + ((p ^ (tx & 7)) << 2));
#pragma unroll
                    for (int i = 0; i < 4; ++i) q4[i] = *reinterpret_cast<const float4*>(qs + (ty + 16 * i) * HD + ((p ^ (ty & 7)) << 2));
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            s[i][j] = fmaf(q4[i].x, k4[j].x, s[i][j]);
                            s[i][j] = fmaf(q4[i].y, k4[j].y, s[i][j]);
                            s[i][j] = fmaf(q4[i].z, k4[j].z, s[i][j]);
                            s[i][j] = fmaf(q4[i].w, k4[j].w, s[i][j]);
                        }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 2; ++j) ss[(ty + 16 * i) * SP + tx + 16 * j] = s[i][j];
            }
            __syncthreads();
            const bool page_there = page >= 0;
#pragma unroll 1
            for (int r0 = warp * 8; r0 < warp * 8 + 8; r0 += 4) {
                // four rows side by side; a row without a key in this chunk (or not of this sequence) stays as it is
                float m[4], l[4], corr[4], p[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    m[i] = row_m[r0 + i];
                    l[i] = row_l[r0 + i];
                    p[i] = chunk_softmax(ss[(r0 + i) * SP + lane], page_there && t0 + lane <= row_pos[r0 + i], a.scale, inv_scale,
                                         a.softcap, m[i], l[i], corr[i]);
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    ss[(r0 + i) * SP + lane] = p[i];
                    if (lane == i) {
                        row_m[r0 + i] = m[i];
                        row_l[r0 + i] = l[i];
                        row_corr[r0 + i] = corr[i];
                    }
                }
            }
            __syncthreads();
            // rows ty + 16 i, elements 4 tx + 64 d ..; where some row does not see all 32 keys, a product is left out
            // key by key (the value of a key that the row does not see may be anything)
            int last[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                last[i] = row_pos[ty + 16 * i] - t0;
                const float c = row_corr[ty + 16 * i];
#pragma unroll
                for (int d = 0; d < 4 * DT; ++d) acc[i][d] *= c;
            }
            if (!whole || lo < t0 + TL_KEYS - 1) add_values<HD, true>(ss + ty * SP, vd + 4 * tx, last, acc);
            else add_values<HD, false>(ss + ty * SP, vd + 4 * tx, last, acc);
            __syncthreads();  // the chunk's buffer, the probabilities and the rows' numbers are written again
            page = page_next;
            page_next = page_after;
        }
        i0 = i1;
    }
    cp_wait<0>();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty + 16 * i, tok = first_token + r / G;
        if (r >= tt * G || t_seq[r / G] < 0) continue;   // beyond the tile's last token as well
        const int h = kvh * G + r % G;
        float l = row_l[r], corr = 1.f;
        if (a.sink != nullptr) {
            const float sk = a.sink[h], m = row_m[r], m_new = fmaxf(m, sk);
            corr = expf(m - m_new);
            l = l * corr + expf(sk - m_new);
        }
        const float inv_l = (l > 0.f) ? 1.0f / l : 0.f;
        float* orow = a.out + (size_t)tok * a.out_stride + (size_t)h * HD;
#pragma unroll
        for (int d = 0; d < DT; ++d)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float v = acc[i][4 * d + e];
                if (a.sink != nullptr) v *= corr;
                orow[64 * d + 4 * tx + e] = v * inv_l;
            }
    }
}

template <int HD>
constexpr int tile_smem() {
    return (TL_ROWS * HD + 4 * TL_KEYS * HD + TL_ROWS * (TL_KEYS + 4) + 6 * TL_ROWS) * 4;
}

template <int HD>
int launch_tile(const F32Attn& a, cudaStream_t s) {
    const cudaError_t e = cudaFuncSetAttribute(attention_f32_tile_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_smem<HD>());
    if (e != cudaSuccess) return (int)e;
    const int tt = TL_ROWS / (a.Hq / a.Hkv);
    // a sequence of n tokens has (n - 1) / tt + 1 tiles: the most that n_seqs sequences of T tokens in all can have
    const int seqs = min(a.T, a.n_seqs);
    const long long tiles = a.seq_start != nullptr ? (long long)(a.T - seqs) / tt + seqs : (a.T + tt - 1) / tt;
    if (tiles * a.Hkv > 2147483647LL) return -1;
    odin_launch(attention_f32_tile_kernel<HD>, dim3((unsigned)(tiles * a.Hkv)), dim3(TL_THREADS), (size_t)tile_smem<HD>(), s, a);
    return 0;
}

int launch_single(const F32Attn& a, cudaStream_t s) {
    constexpr int most = 4 * SG_KEYS * (SG_MAX_HD + 4) * 4;
    const cudaError_t e = cudaFuncSetAttribute(attention_f32_single_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e != cudaSuccess) return (int)e;
    odin_launch(attention_f32_single_kernel, dim3((unsigned)(a.T * a.Hkv)), dim3(SG_THREADS), (size_t)(4 * SG_KEYS * (a.hd + 4) * 4), s, a);
    return 0;
}

}  // namespace

// q: [T, Hq*hd] with row stride q_row_stride (elements); out: [T, Hq*vd] with row stride out_row_stride.
// single: every sequence brings at most one of the T tokens.
// seq_start (may be null): [n_seqs + 1], sequence b's tokens being seq_start[b] .. seq_start[b + 1]; tokens of no sequence
// (tok_seq -1) may follow the last.
extern "C" int odin_attention_plain(const void* q, long long q_row_stride, void* out, long long out_row_stride,
                                    int dtype, int T, int Hq, int Hkv, int hd, int vd, const void* k_cache,
                                    const void* v_cache, int page_size, const int* tok_pos, const int* tok_seq,
                                    const int* block_table, int bt_stride, int window, int chunk, float scale,
                                    float softcap, const float* sink, int single, const int* seq_start,
                                    int n_seqs, void* stream) {
    if (T <= 0) return 0;
    if (hd <= 0 || hd > AP_MAX_HD || vd <= 0 || vd > AP_MAX_HD || Hkv <= 0 || Hq % Hkv != 0 ||
        window < 0 || chunk < 0)
        return ODIN_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    const long long items = (long long)T * Hq;
    const long long blocks = (items + AP_WARPS - 1) / AP_WARPS;
    if (blocks > 2147483647LL) return ODIN_ERR_UNSUPPORTED;
    const int group = Hq / Hkv;
    // rows of whole 16-byte vectors, value heads of the keys' size.  single: every sequence brings one token.
    if (dtype == ODIN_F32 && hd == vd && hd % 4 == 0 && hd <= SG_MAX_HD && group <= SG_MAX_G && q_row_stride % 4 == 0 &&
        aligned16(q) && aligned16(k_cache) && aligned16(v_cache) && page_size % SG_KEYS == 0) {
        const F32Attn a{(const float*)q, (float*)out, (const float*)k_cache, (const float*)v_cache, tok_pos, tok_seq, block_table,
                        sink, n_seqs > 1 ? seq_start : nullptr, (size_t)q_row_stride, (size_t)out_row_stride, T, Hq, Hkv, hd,
                        page_size, bt_stride, window, chunk, n_seqs, scale, softcap};
        int rc = -1;
        if (single) rc = launch_single(a, s);
        else if (window == 0 && chunk == 0 && hd == 128) rc = launch_tile<128>(a, s);
        else if (window == 0 && chunk == 0 && hd == 64) rc = launch_tile<64>(a, s);
        if (rc > 0) return rc;
        if (rc == 0) {
            ODIN_LAUNCH_CHECK();
            return 0;
        }
    }
#define GO(TT, R)                                                                                                       \
    odin_launch(attention_plain_kernel<TT, R>, dim3((unsigned)blocks), dim3(AP_WARPS * 32), 0, s, (const TT*)q,          \
                (size_t)q_row_stride, (TT*)out, (size_t)out_row_stride, T, Hq, Hkv, hd, vd, (const TT*)k_cache,           \
                (const TT*)v_cache, page_size, tok_pos, tok_seq, block_table, bt_stride, window, chunk, scale, softcap, sink)
#define GO_R(TT)                             \
    do {                                     \
        if (widest <= 128) GO(TT, 4);        \
        else if (widest <= 256) GO(TT, 8);   \
        else if (widest <= 512) GO(TT, 16);  \
        else GO(TT, 32);                     \
    } while (0)
    const int widest = hd > vd ? hd : vd;
    if (dtype == ODIN_BF16) GO_R(bf16);
    else if (dtype == ODIN_F32) GO_R(float);
    else return ODIN_ERR_UNSUPPORTED;
#undef GO_R
#undef GO
    ODIN_LAUNCH_CHECK();
    return 0;
}
