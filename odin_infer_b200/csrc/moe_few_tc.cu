// Experts chosen per token for a step of few tokens (bfloat16): both products of every chosen expert with all of its rows
// together, straight from the router's choices, on the tcgen05 tensor cores.
//
// The grouped products (moe_tc.cu) put 128 sorted rows on the wide side of the MMA; with two or three rows an expert that is
// padding, and the rows need a plan and a gather, a kernel each.  Here the weights are the wide side (their rows are the
// MMA's 128) and the expert's rows, up to TN of them, are its columns:
//   * every CTA finds the experts' rows itself (the choices are a few hundred numbers) and takes an equal, contiguous share
//     of the units of work (expert, 64 weight rows), so all SMs stream weights to the end;
//   * warp 0 feeds a ring of 16 KB stages by TMA across units; warps 2 to 5 bring an expert's rows into shared memory in the
//     MMA's swizzled layout when the expert changes (rows of the tokens directly: no gather), and read the accumulators back;
//   * the second product's CTAs start while the first one's run (which have waited for the router, so the choices are known)
//     and fill their rings meanwhile.
// An output is the same sum over K in the same order of K blocks as in the grouped products, so the bits are theirs.
// What bounds it: the chosen experts' weights (6.3 + 3.1 MB each for 2048 -> 768 -> 2048), and at few tokens the start of each
// product (choices, rows, first weights: 3 to 4 us).  Both products of 8 tokens, 4 of 32 experts and 2 shared ones each: 60 us
// beside 89 for plan, gather and grouped products; 16 tokens 83 and 116, 32 tokens 106 and 126; a decode step of 8 sequences with
// 7 such layers 0.969 -> 0.840 ms (0.873 with rings of 5 and 4 stages, which would leave both products' CTAs room on an SM).
#include "moe_tc_host.cuh"

using namespace moe_tc;

namespace {

constexpr int UMMA_K = 16;
constexpr int UNIT = 64;                    // weight rows of a unit of work (gated: 32 gate and 32 up rows)
constexpr int BOX = UNIT * BK * 2;          // bytes of a unit's weights of a K block
constexpr int STAGE = 2 * BOX;              // a stage of the ring: a K block of two units, or two K blocks of one
constexpr int MAX_STAGES = 8;
constexpr int FEW_THREADS = 192;
constexpr int MAX_CHOICES = 256;
constexpr int MAX_EXPERTS = 256;
constexpr int MOST_SMEM = 227 * 1024;

#define FEW_GATED 0   // out[row] = act(gate) * up, bfloat16
#define FEW_PLAIN 1   // out[row] = act(z), bfloat16
#define FEW_DOWN 2    // out[row] = z, 32-bit

struct FewParams {
    const bf16* x;
    size_t x_stride;
    const int* ids;         // [choices] expert of every row (token, choice); -1: none
    const float* in_wts;    // factor on a row's input (null: none)
    void* out;
    size_t ldo;
    int choices, x_per;     // x_per: rows that share an input row (the second product: 1)
    int n_experts, N, K, rows_per_expert, act, stages, x_rows;
    int* error;
};

// Rows of an expert that are multiplied together: their places in the list, and the expert.
struct Group {
    int expert, first, n;
};

struct Lists {
    alignas(16) int id[MAX_CHOICES];   // the choices' experts
    int count[MAX_EXPERTS];     // rows of every expert
    int first[MAX_EXPERTS];     // its first place in the list
    int list[MAX_CHOICES];      // rows by expert
    Group group[MAX_CHOICES];   // experts in ascending order, each cut into groups of `most` rows
    int n_groups;
};

// ids -> lists, by the whole CTA.  The order of an expert's rows is the choices' own: CTAs agree on its groups.
__device__ __forceinline__ void make_lists(const int* ids, int choices, int n_experts, int most, Lists& l) {
    const int tid = threadIdx.x, lane = tid & 31;
    constexpr int HELD = (MAX_CHOICES + FEW_THREADS - 1) / FEW_THREADS;
    int e[HELD], rank[HELD];
#pragma unroll
    for (int k = 0; k < HELD; ++k) {
        const int r = tid + k * FEW_THREADS;
        e[k] = r < choices ? ids[r] : -1;
        if (e[k] >= n_experts) e[k] = -1;
    }
    for (int i = tid; i < n_experts; i += FEW_THREADS) l.count[i] = 0;
#pragma unroll
    for (int k = 0; k < HELD; ++k)
        if (tid + k * FEW_THREADS < MAX_CHOICES) l.id[tid + k * FEW_THREADS] = e[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < HELD; ++k) {
        rank[k] = 0;
        if (e[k] < 0) continue;
        const int r = tid + k * FEW_THREADS;
        int all = 0;
        for (int j = 0; j < choices; j += 4) {
            const int4 o = *reinterpret_cast<const int4*>(l.id + j);
            const int same[4] = {o.x == e[k], o.y == e[k], o.z == e[k], o.w == e[k]};
#pragma unroll
            for (int i = 0; i < 4; ++i) { all += same[i]; rank[k] += same[i] && j + i < r; }
        }
        l.count[e[k]] = all;   // (each of the expert's rows writes the same)
    }
    __syncthreads();
    if (tid < 32) {
        int rows = 0, groups = 0;   // of the experts before these 32
        for (int e0 = 0; e0 < n_experts; e0 += 32) {
            const int c = e0 + lane < n_experts ? l.count[e0 + lane] : 0, g = (c + most - 1) / most;
            int rs = c, gs = g;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int a = __shfl_up_sync(0xffffffffu, rs, o), b = __shfl_up_sync(0xffffffffu, gs, o);
                if (lane >= o) { rs += a; gs += b; }
            }
            const int f = rows + rs - c;
            if (e0 + lane < n_experts) l.first[e0 + lane] = f;
            for (int i = 0; i < g; ++i) l.group[groups + gs - g + i] = Group{e0 + lane, f + i * most, min(most, c - i * most)};
            rows += __shfl_sync(0xffffffffu, rs, 31);
            groups += __shfl_sync(0xffffffffu, gs, 31);
        }
        if (lane == 0) l.n_groups = groups;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < HELD; ++k)
        if (e[k] >= 0) l.list[l.first[e[k]] + rank[k]] = tid + k * FEW_THREADS;
    __syncthreads();
}

template <int TN>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[TN]) {
    if constexpr (TN == 16) tc::tmem_ld16(taddr, r);
    else tc::tmem_ld32(taddr, r);
}

template <int MODE, int TN>
__global__ void __launch_bounds__(FEW_THREADS, 1)
moe_few_kernel(const __grid_constant__ CUtensorMap map_w, const FewParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ Lists lists;
    __shared__ __align__(8) uint64_t full[MAX_STAGES], empty[MAX_STAGES], acc_full[2], acc_empty[2], up_full[2][2], x_full;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_s;
    __shared__ float up_s[2][2][MODE == FEW_GATED ? TN : 1][32];   // the up rows' sums on their way to the gate rows' warp
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t n_stages = (uint32_t)p.stages;
    // [K blocks][x_rows rows of 128 bytes].  With 8 rows at most (x_rows 8, TN 16) the columns 8 to 15 of a block are the next
    // block's rows: sums that nobody reads.  A unit alone leaves the MMA the 64 rows behind its weights, whatever they are.
    uint8_t* xs = ring + n_stages * STAGE;
    const int x_block = p.x_rows * BK * 2;
    volatile int* abort_flag = &abort_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_kb = (p.K + BK - 1) / BK;
    constexpr int COLS = MODE == FEW_GATED ? UNIT / 2 : UNIT;   // output columns of a unit
    const int units = (p.N + COLS - 1) / COLS;
    if (threadIdx.x == 0) {
        for (int s = 0; s < MAX_STAGES; ++s) { tc::mbar_init(&full[s], 1); tc::mbar_init(&empty[s], 1); }
        for (int a = 0; a < 2; ++a) {
            tc::mbar_init(&acc_full[a], 1);
            tc::mbar_init(&acc_empty[a], 4);   // one arrival per epilogue warp
            tc::mbar_init(&up_full[a][0], 1);
            tc::mbar_init(&up_full[a][1], 1);
        }
        tc::mbar_init(&x_full, 4);
        abort_s = 0;
        tc::fence_barrier_init();
        tc::prefetch_tensormap(&map_w);
    }
    // The first product waits for the router and only then lets the second one start: when that one's CTAs run, the choices
    // are known to them, and they wait for the rows alone.  Tensor memory is allocated behind that wait (a kernel before this
    // one may yet ask for all of an SM's) and before the trigger (one after this may take all of it and wait for this one).
    if (MODE != FEW_DOWN) pdl_wait();
    if (warp == 1) tc::tmem_alloc(&tmem_slot, 2 * TN);
    __syncthreads();
    pdl_trigger();
    make_lists(p.ids, p.choices, p.n_experts, p.x_rows, lists);
    odin_trace_mark(2);  // the lists are made
    const long long total = (long long)lists.n_groups * units;
    const int i0 = (int)(total * blockIdx.x / gridDim.x), i1 = (int)(total * (blockIdx.x + 1) / gridDim.x);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem_base = tmem_slot;
    // two units of a group side by side fill the MMA's 128 rows; every role walks the same items of one or two units
    auto width = [&](int i) { return (i + 1 < i1 && (i + 1) / units == i / units) ? 2 : 1; };

    if (warp == 0) {
        // ------------------------------------------------------- the weights
        if (lane == 0) {
            uint32_t stage = 0, phase = 0;
            bool ok = true;
            for (int i = i0; i < i1 && ok;) {
                const int w = width(i);
                const int row0 = lists.group[i / units].expert * p.rows_per_expert + (i % units) * COLS;
                for (int kb = 0; kb < n_kb; kb += 3 - w) {
                    if (!tc::mbar_wait(&empty[stage], phase ^ 1, abort_flag)) { ok = false; break; }
                    const int boxes = w == 2 ? 2 : min(2, n_kb - kb);
                    tc::mbar_expect_tx(&full[stage], boxes * BOX);
                    for (int b = 0; b < boxes; ++b) {
                        uint8_t* dst = ring + stage * STAGE + b * BOX;
                        const int x = (w == 2 ? kb : kb + b) * BK, row = w == 2 ? row0 + b * COLS : row0;
                        tc::tma_load_2d(dst, &map_w, x, row, &full[stage]);
                        if (MODE == FEW_GATED) tc::tma_load_2d(dst + BOX / 2, &map_w, x, row + p.N, &full[stage]);
                    }
                    if (++stage == n_stages) { stage = 0; phase ^= 1; }
                }
                i += w;
            }
            odin_trace_mark(6, true);  // every load is requested
            if (!ok) tc::drain_ring(full, n_stages, stage, phase);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------- the MMAs
        constexpr uint32_t idesc = tc::make_idesc_bf16(128, TN);
        uint32_t stage = 0, phase = 0, x_phase = 0, local = 0;
        int group = -1;
        bool ok = true, ready = false;
        for (int i = i0; i < i1 && ok; ++local) {
            const int w = width(i);
            const uint32_t acc = local & 1, acc_phase = (local >> 1) & 1;
            if (i / units != group) {
                group = i / units;
                ok = __all_sync(0xffffffffu, tc::mbar_wait(&x_full, x_phase, abort_flag));
                if (!ok) break;
                x_phase ^= 1;
                if (lane == 0 && local == 0) odin_trace_mark(3, true);  // the first rows are there
            }
            ok = __all_sync(0xffffffffu, tc::mbar_wait(&acc_empty[acc], acc_phase ^ 1, abort_flag));
            if (!ok) break;
            tc::fence_after_sync();
            for (int kb = 0; kb < n_kb; kb += 3 - w) {
                if (!ready) ready = tc::mbar_wait(&full[stage], phase, abort_flag);
                ok = __all_sync(0xffffffffu, ready);
                if (!ok) break;
                tc::fence_after_sync();
                if (lane == 0 && local == 0 && kb == 0) odin_trace_mark(4, true);  // the first weights are there
                const uint32_t cur = stage;
                if (++stage == n_stages) { stage = 0; phase ^= 1; }
                ready = __all_sync(0xffffffffu, tc::mbar_test_wait(&full[stage], phase));   // its latency hides behind the MMAs
                if (tc::elect_one()) {
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        if (b > 0 && (w == 2 || kb + b >= n_kb)) break;
                        const uint64_t da = tc::make_smem_desc_sw128(tc::smem_u32(ring + cur * STAGE + b * BOX));
                        const uint64_t db = tc::make_smem_desc_sw128(tc::smem_u32(xs + (kb + b) * x_block));
#pragma unroll
                        for (int k = 0; k < BK / UMMA_K; ++k)   // +32 bytes per K step inside the swizzle row: +2 in 16-byte units
                            tc::umma_bf16(tmem_base + acc * TN, da + 2 * k, db + 2 * k, idesc, (kb + b > 0 || k > 0) ? 1u : 0u);
                    }
                    tc::umma_commit(&empty[cur]);
                }
                __syncwarp();
            }
            if (ok && tc::elect_one()) tc::umma_commit(&acc_full[acc]);
            __syncwarp();
            i += w;
            if (lane == 0 && i >= i1) odin_trace_mark(5, true);  // the last commit is issued
        }
    } else {
        // ------------------------------------------------------- the rows, and what becomes of the sums
        const int quarter = warp & 3;   // the tensor-memory lanes this warp may read: [32 quarter, +32): unit quarter / 2
        const int me = threadIdx.x - 64, part = quarter >> 1;
        if (MODE == FEW_DOWN) pdl_wait();
        uint32_t local = 0, up_phase = 0;
        int group = -1;
        for (int i = i0, w; i < i1; i += w, ++local) {
            w = width(i);
            const Group gr = lists.group[i / units];
            if (i / units != group) {
                // (the MMAs that read the rows before are done: this warp has seen the item before complete)
                group = i / units;
                const int pieces = n_kb * (BK / 8), all = gr.n * pieces;
                constexpr int BATCH = 8;
                for (int c0 = me; c0 < all; c0 += 128 * BATCH) {
                    uint4 v[BATCH];
#pragma unroll
                    for (int b = 0; b < BATCH; ++b) {
                        const int c = c0 + 128 * b, n = c / pieces, k = (c - n * pieces) * 8;
                        v[b] = make_uint4(0, 0, 0, 0);
                        if (c < all && k < p.K) {
                            const int r = lists.list[gr.first + n];
                            v[b] = *reinterpret_cast<const uint4*>(p.x + (size_t)(r / p.x_per) * p.x_stride + k);
                        }
                    }
#pragma unroll
                    for (int b = 0; b < BATCH; ++b) {
                        const int c = c0 + 128 * b, n = c / pieces, piece = c - n * pieces;
                        if (c >= all) break;
                        if (p.in_wts != nullptr) {   // a 32-bit product, rounded once
                            const float f = p.in_wts[lists.list[gr.first + n]];
                            __nv_bfloat162* q = reinterpret_cast<__nv_bfloat162*>(&v[b]);
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float2 t = __bfloat1622float2(q[j]);
                                q[j] = __floats2bfloat162_rn(f * t.x, f * t.y);
                            }
                        }
                        *reinterpret_cast<uint4*>(xs + (size_t)(piece >> 3) * x_block + n * 128 + (((piece & 7) ^ (n & 7)) << 4)) = v[b];
                    }
                }
                tc::fence_proxy_async();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&x_full);
            }
            const uint32_t acc = local & 1, acc_phase = (local >> 1) & 1;
            if (!tc::mbar_wait(&acc_full[acc], acc_phase, abort_flag)) break;
            if (part >= w) {
                if (lane == 0) tc::mbar_arrive(&acc_empty[acc]);
                continue;
            }
            tc::fence_after_sync();
            uint32_t r[TN];
            tmem_ld<TN>(tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * TN, r);
            tc::tmem_ld_wait();
            tc::fence_before_sync();
            if (MODE == FEW_GATED) {
                if (quarter & 1) {
#pragma unroll
                    for (int n = 0; n < TN; ++n) up_s[acc][part][n][lane] = __uint_as_float(r[n]);
                    __syncwarp();
                    if (lane == 0) { tc::mbar_arrive(&up_full[acc][part]); tc::mbar_arrive(&acc_empty[acc]); }
                    continue;
                }
                if (!tc::mbar_wait(&up_full[acc][part], (up_phase >> acc) & 1, abort_flag)) break;
                up_phase ^= 1u << acc;
            }
            const int j = (i % units + part) * COLS + (MODE == FEW_GATED ? lane : (quarter & 1) * 32 + lane);
            if (j < p.N) {
#pragma unroll
                for (int n = 0; n < TN; ++n) {
                    if (n >= gr.n) break;
                    const size_t at = (size_t)lists.list[gr.first + n] * p.ldo + j;
                    const float z = __uint_as_float(r[n]);
                    if (MODE == FEW_GATED) reinterpret_cast<bf16*>(p.out)[at] = __float2bfloat16_rn(act_gate(p.act, z) * up_s[acc][part][n][lane]);
                    else if (MODE == FEW_PLAIN) reinterpret_cast<bf16*>(p.out)[at] = __float2bfloat16_rn(act_alone(p.act, z));
                    else reinterpret_cast<float*>(p.out)[at] = z;
                }
            }
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&acc_empty[acc]);   // (the up rows' sums are read: they may be written again)
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag && p.error != nullptr) atomicCAS(p.error, 0, 1);
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem_base, 2 * TN);
    }
}

// bytes of the rows and what an MMA may read behind them (columns of the last block, weights of the last stage)
constexpr int x_bytes(int K, int x_rows) { return (K + BK - 1) / BK * x_rows * BK * 2 + BOX; }
constexpr int few_smem(int stages, int K, int x_rows) { return 1024 /* alignment */ + stages * STAGE + x_bytes(K, x_rows); }

template <int MODE, int TN>
int launch_few(const CUtensorMap& mw, FewParams p, int smem, cudaStream_t s) {
    auto k = moe_few_kernel<MODE, TN>;
    const cudaError_t e = odin_allow_smem(k, (size_t)smem);
    if (e != cudaSuccess) return (int)e;
    odin_launch(k, dim3(sm_count()), dim3(FEW_THREADS), (size_t)smem, s, mw, p);
    ODIN_LAUNCH_CHECK();
    return 0;
}

template <int TN>
int run_few(const CUtensorMap& mu, const CUtensorMap& md, FewParams up, FewParams down, bool gated, cudaStream_t s) {
    // as long a ring as fits, up to 8 stages (128 KB): more in flight is worth more than the second product's CTA beside the
    // first one's
    constexpr int STATIC_UP = sizeof(Lists) + 4 * TN * 32 * 4 + 1024, STATIC_DOWN = sizeof(Lists) + 1024;   // (upper bounds)
    const int x1 = few_smem(0, up.K, up.x_rows), x2 = few_smem(0, down.K, down.x_rows);
    up.stages = (MOST_SMEM - STATIC_UP - x1) / STAGE;
    down.stages = (MOST_SMEM - STATIC_DOWN - x2) / STAGE;
    if (up.stages > MAX_STAGES) up.stages = MAX_STAGES;
    if (down.stages > MAX_STAGES) down.stages = MAX_STAGES;
    if (up.stages < 3 || down.stages < 3) return ODIN_ERR_UNSUPPORTED;
    const int s1 = few_smem(up.stages, up.K, up.x_rows), s2 = few_smem(down.stages, down.K, down.x_rows);
    const int rc = gated ? launch_few<FEW_GATED, TN>(mu, up, s1, s) : launch_few<FEW_PLAIN, TN>(mu, up, s1, s);
    return rc ? rc : launch_few<FEW_DOWN, TN>(md, down, s2, s);
}

}  // namespace

// The chosen experts' feed-forwards of T tokens with `per` choices each, row r = t * per + k: a[r] = act(Wg[e] x) * (Wu[e] x)
// (gated: w_up [experts][2 ff][d], gate rows first) or act(W[e] x) (w_up [experts][ff][d]), then c[r] = Wd[e] a[r] (w_down
// [experts][d][ff], c 32-bit [T * per][d]), e = ids[r], x = h[t] or in_wts[r] * h[t] rounded to bfloat16; rows of choices without
// an expert (-1) are left as they are.  ODIN_ERR_UNSUPPORTED, and nothing is launched, for sizes that do not fit.
extern "C" int odin_moe_few(const void* h, long long h_stride, const void* w_up, const void* w_down, const int* ids,
                            const float* in_wts, int T, int per, int n_experts, int ff, int d, int act, int gated, void* a, float* c,
                            void* stream) {
    if (T <= 0) return 0;
    if (per <= 0 || ff <= 0 || d <= 0 || n_experts <= 0) return ODIN_ERR_BAD_ARG;
    if (act != MOE_ACT_SILU && act != MOE_ACT_GELU_TANH && (gated || act != MOE_ACT_RELU2)) return ODIN_ERR_BAD_ARG;
    if (T > 32 || T * per > MAX_CHOICES || n_experts > MAX_EXPERTS || d % 8 || ff % 8 || h_stride % 8 ||
        (((uintptr_t)h | (uintptr_t)w_up | (uintptr_t)w_down | (uintptr_t)a) & 15) != 0)
        return ODIN_ERR_UNSUPPORTED;
    const int up_rows = gated ? 2 * ff : ff;
    const int x_rows = T <= 8 ? 8 : T <= 16 ? 16 : 32;
    CUtensorMap mu, md;
    int rc;
    if ((rc = make_map(&mu, w_up, (long long)n_experts * up_rows, d, d, gated ? UNIT / 2 : UNIT))) return rc;
    if ((rc = make_map(&md, w_down, (long long)n_experts * d, ff, ff, UNIT))) return rc;
    const FewParams up{(const bf16*)h, (size_t)h_stride, ids, in_wts, a, (size_t)ff, T * per, per, n_experts, ff, d, up_rows, act, 0, x_rows, error_flag()};
    const FewParams down{(const bf16*)a, (size_t)ff, ids, nullptr, c, (size_t)d, T * per, 1, n_experts, d, ff, d, 0, 0, x_rows, error_flag()};
    return T <= 16 ? run_few<16>(mu, md, up, down, gated != 0, (cudaStream_t)stream) : run_few<32>(mu, md, up, down, gated != 0, (cudaStream_t)stream);
}
