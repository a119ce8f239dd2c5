// Experts chosen per token, for a decode step's handful of tokens (bfloat16): both products of every chosen expert with
// all of its rows together, straight from the router's choices.
//
// With 32 rows (token, choice) over 32 experts a row has its expert almost to itself.  Tiles of 128 sorted rows then
// stream padding beside the weights and need a plan, a gather and a combine; kernels per row read an expert's weights
// once for every row.  Here a block takes one or two sets of 32 weight rows of one expert and up to 16 of the expert's rows at a time:
//   * it finds the expert's rows itself (the choices are a few hundred numbers), and returns if there are none;
//   * its eight warps share K; a lane loads 16 bytes of a weight row straight into the registers of an
//     mma.m16n8k16 operand: lane (g, t) holds the eight k from k0 + 8 t on of rows g and g + 8, and takes the same eight
//     of token g from shared memory, so the MMA's k order is a permutation that both operands share;
//   * the warps' sums are added in their order through shared memory, then the activation (or the row's weight).
// What bounds it: the weights, and for very few rows the chain of a block (choices, inputs, weights, sums).  32 experts of
// 2048 -> 768 -> 2048, 4 per token: both products for 8 tokens 45 to 48 us (50.5 with one set a block; tiles of 128 sorted
// rows with their plan, gather and combine 79 to 83, kernels per row 79; the weights alone take 29 to 33), for 1 token 20 us
// (48, 39), for 32 tokens 68 (110, 222).
// A row's values do not depend on the other rows.  mma.sync and not tcgen05: the products are bound by the weights they
// stream (6.3 MB of gate and up per expert beside 3 to 16 rows), and an operand that goes from memory to registers needs
// no stage, no barrier and no tensor memory.
#include "common.cuh"

namespace {

constexpr int FEW_THREADS = 256;
constexpr int FEW_WARPS = 8;
constexpr int FEW_ROWS = 16;        // the expert's rows that a pass over the weights takes
constexpr int FEW_BATCH = 4;        // steps of 32 k whose weights are in flight in a warp
constexpr int FEW_MAX_CHOICES = 4096;

#define FEW_GATED 0      // out[row][j] = act(gate_j) * up_j
#define FEW_PLAIN 1      // out[row][j] = act(z_j)
#define FEW_DOWN 2       // y[choice][token][c] = weight * z_c

#define MOE_ACT_SILU 1
#define MOE_ACT_GELU_TANH 2
#define MOE_ACT_RELU2 4

__device__ __forceinline__ float few_activate(int act, float z) {
    if (act == MOE_ACT_SILU) return z / (1.0f + expf(-z));
    if (act == MOE_ACT_RELU2) {
        const float r = fmaxf(z, 0.f);
        return r * r;
    }
    const float y = 0.7978845608028654f * (z + 0.044715f * z * z * z);
    return 0.5f * z * (1.0f + tanhf(y));
}

__device__ __forceinline__ uint4 ld_stream(const bf16* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

struct FewArgs {
    const bf16* x;         // gate|up: the tokens' rows [T][x_stride]; down: the experts' activations, one row per choice
    const bf16* w;         // [experts][w_rows][K]
    const int* ids;        // [choices] expert of every choice, -1: none
    const float* in_wts;   // factor on a choice's input (gate|up; may be null)
    const float* out_wts;  // factor on a choice's answer (down; may be null)
    void* out;
    size_t x_stride;
    int choices, per, K, w_rows, n_out, act, x_rows, x_pitch;   // n_out: columns of the output; x_pitch in bytes
    int sets;              // sets of COLS output columns that a block takes one after the other
};

template <int MODE>
__global__ void __launch_bounds__(FEW_THREADS, 2) moe_few_kernel(const FewArgs a) {
    extern __shared__ __align__(16) uint8_t few_sm[];
    __shared__ int n_found;
    __shared__ __align__(16) float red[FEW_WARPS][2][2][16][8];   // [warp][tile of 8 rows][group of 16 weight rows][weight row][row]
    uint8_t* xs = few_sm;                                                  // [x_rows][x_pitch]
    int* list = reinterpret_cast<int*>(few_sm + (size_t)a.x_rows * a.x_pitch);   // the expert's choices
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int e = blockIdx.y;
    constexpr int COLS = MODE == FEW_GATED ? 16 : 32;   // output columns of the block
    const int j_first = blockIdx.x * (COLS * a.sets), j_end = min(j_first + COLS * a.sets, a.n_out);
    if (tid == 0) n_found = 0;
    pdl_trigger();
    pdl_wait();
    __syncthreads();
    for (int r = tid; r < a.choices; r += FEW_THREADS) {
        const int id = a.ids[r];
        if (id == e) list[atomicAdd(&n_found, 1)] = r;
        // choices without an expert: their answer is zero
        if (MODE == FEW_DOWN && e == 0 && id < 0) {
            float* y = (float*)a.out + ((size_t)(r % a.per) * (a.choices / a.per) + r / a.per) * a.n_out;
            for (int j = j_first; j < j_end; ++j) y[j] = 0.f;
        }
    }
    __syncthreads();
    const int n_rows = n_found;
    if (n_rows == 0) return;

    // this lane's weight rows: g and g + 8 of two groups of 16 (rows beyond the matrix repeat its last one)
    const bf16* we = a.w + (size_t)e * a.w_rows * a.K;
    const int second = MODE == FEW_GATED ? a.w_rows / 2 : 16;   // distance of the second group: the up rows, or the next 16
    const int limit = MODE == FEW_GATED ? a.w_rows / 2 : a.w_rows;
    const bf16* wp[4];
    auto at_columns = [&](int j0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int row = MODE == FEW_GATED ? (q >> 1) * second + min(j0 + g + 8 * (q & 1), limit - 1)
                                              : min(j0 + (q >> 1) * second + g + 8 * (q & 1), limit - 1);
            wp[q] = we + (size_t)row * a.K + 8 * t;
        }
    };
    const int steps = (a.K + 31) / 32, per_warp = (steps + FEW_WARPS - 1) / FEW_WARPS;
    const int s0 = warp * per_warp, s1 = min(steps, s0 + per_warp);

    for (int r0 = 0; r0 < n_rows; r0 += a.x_rows) {
        const int here = min(a.x_rows, n_rows - r0);
        uint4 v[FEW_BATCH][4];
        auto fetch = [&](int s, uint4 (&d)[4]) {   // the weights of step s
            const bool in = s < s1 && s * 32 + 8 * t < a.K;
#pragma unroll
            for (int q = 0; q < 4; ++q) d[q] = in ? ld_stream(wp[q] + (size_t)s * 32) : make_uint4(0, 0, 0, 0);
        };
        at_columns(j_first);
#pragma unroll
        for (int u = 0; u < FEW_BATCH; ++u) fetch(s0 + u, v[u]);
        // the rows' inputs, padded with zeros to whole tiles of 8 rows and whole steps
        const int tiles = (here + 7) / 8, pieces = steps * 4;
        for (int c = tid; c < tiles * 8 * pieces; c += FEW_THREADS) {
            const int n = c / pieces, piece = c - n * pieces;
            uint4 x = make_uint4(0, 0, 0, 0);
            if (n < here && piece * 8 < a.K) {
                const int r = list[r0 + n];
                x = *reinterpret_cast<const uint4*>(a.x + (size_t)(MODE == FEW_DOWN ? r : r / a.per) * a.x_stride + piece * 8);
                if (MODE != FEW_DOWN && a.in_wts != nullptr) {   // a 32-bit product, rounded once
                    const float f = a.in_wts[r];
                    bf16* b = reinterpret_cast<bf16*>(&x);
#pragma unroll
                    for (int i = 0; i < 8; ++i) b[i] = __float2bfloat16_rn(f * __bfloat162float(b[i]));
                }
            }
            *reinterpret_cast<uint4*>(xs + (size_t)n * a.x_pitch + piece * 16) = x;
        }
        __syncthreads();
#pragma unroll 1
        for (int j0 = j_first; j0 < j_end; j0 += COLS) {
            float acc[2][2][4];
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int q = 0; q < 2; ++q)
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[n][q][i] = 0.f;
            for (int s = s0; s < s1; s += FEW_BATCH) {
#pragma unroll
                for (int u = 0; u < FEW_BATCH; ++u) {
                    if (s + u >= s1) break;
#pragma unroll
                    for (int n = 0; n < 2; ++n) {
                        if (n >= tiles) break;
                        const uint4 x = *reinterpret_cast<const uint4*>(xs + (size_t)(n * 8 + g) * a.x_pitch + (s + u) * 64 + t * 16);
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            mma16816(acc[n][q], v[u][2 * q].x, v[u][2 * q + 1].x, v[u][2 * q].y, v[u][2 * q + 1].y, x.x, x.y);
                            mma16816(acc[n][q], v[u][2 * q].z, v[u][2 * q + 1].z, v[u][2 * q].w, v[u][2 * q + 1].w, x.z, x.w);
                        }
                    }
                    fetch(s + u + FEW_BATCH, v[u]);   // into the registers that are free now
                }
            }
            if (j0 + COLS < j_end) {   // the next set's first weights, while the sums meet
                at_columns(j0 + COLS);
#pragma unroll
                for (int u = 0; u < FEW_BATCH; ++u) fetch(s0 + u, v[u]);
            }
            for (int n = 0; n < tiles; ++n)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const float* c = n == 0 ? acc[0][q] : acc[1][q];
                    *reinterpret_cast<float2*>(&red[warp][n][q][g][2 * t]) = make_float2(c[0], c[1]);
                    *reinterpret_cast<float2*>(&red[warp][n][q][g + 8][2 * t]) = make_float2(c[2], c[3]);
                }
            __syncthreads();
            for (int c = tid; c < here * COLS; c += FEW_THREADS) {
                const int n = c / COLS, col = c % COLS, j = j0 + col, r = list[r0 + n];
                if (j >= a.n_out) continue;
                const int grp = MODE == FEW_GATED ? 0 : col >> 4;
                float z = 0.f, up = 0.f;
#pragma unroll
                for (int w = 0; w < FEW_WARPS; ++w) {
                    z += red[w][n >> 3][grp][col & 15][n & 7];
                    if (MODE == FEW_GATED) up += red[w][n >> 3][1][col & 15][n & 7];
                }
                if (MODE == FEW_DOWN) {
                    const float f = a.out_wts != nullptr ? a.out_wts[r] : 1.0f;
                    ((float*)a.out)[((size_t)(r % a.per) * (a.choices / a.per) + r / a.per) * a.n_out + j] = f * z;
                } else {
                    z = few_activate(a.act, z);
                    ((bf16*)a.out)[(size_t)r * a.n_out + j] = __float2bfloat16_rn(MODE == FEW_GATED ? z * up : z);
                }
            }
            __syncthreads();   // the sums, and behind the last set the inputs, are written again
        }
    }
}

template <int MODE>
int launch_few(FewArgs a, int n_experts, cudaStream_t s) {
    constexpr int COLS = MODE == FEW_GATED ? 16 : 32;
    // 8 rows a pass while an expert has 4 or fewer on average: half the shared memory, and a second pass is rare
    a.x_rows = (a.choices / a.per <= 8 || a.choices <= 4 * n_experts) ? 8 : FEW_ROWS;
    a.x_pitch = (a.K * 2 + 127) / 128 * 128 + 64;       // 64 bytes apart in the banks: two rows' pieces in one phase of a load
    // two sets where that leaves blocks enough (two an SM, if every choice names another expert): the second set's weights
    // are on their way while the first one's sums meet, and the rows are found and fetched once for both
    const long long blocks = (long long)((a.n_out + COLS - 1) / COLS) * (a.choices < n_experts ? a.choices : n_experts);
    a.sets = blocks >= 2 * 2 * 148 ? 2 : 1;
    const size_t smem = (size_t)a.x_rows * a.x_pitch + (size_t)a.choices * sizeof(int);
    if (smem > 200 * 1024) return ODIN_ERR_UNSUPPORTED;
    const cudaError_t e = cudaFuncSetAttribute(moe_few_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return (int)e;
    odin_launch(moe_few_kernel<MODE>, dim3((a.n_out + COLS * a.sets - 1) / (COLS * a.sets), n_experts), dim3(FEW_THREADS), smem, s, a);
    ODIN_LAUNCH_CHECK();
    return 0;
}

bool few_ok(const void* x, long long x_stride, const void* w, int T, int per, int K, int n_experts) {
    return T > 0 && per > 0 && (long long)T * per <= FEW_MAX_CHOICES && n_experts > 0 && n_experts <= 65535 && K > 0 && K % 8 == 0 &&
           x_stride % 8 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0;
}

}  // namespace

// a[t * per + k, :] = act(Wg[e] x[t]) * (Wu[e] x[t]) (gated: w [experts][2 ff][d], gate rows first), or act(W[e] x[t])
// (w [experts][ff][d]), e = ids[t, k]; rows of choices without an expert are left as they are.  bfloat16.
extern "C" int odin_moe_few_up(const void* x, long long x_stride, const void* w, const int* ids, const float* in_wts, int T, int per,
                               int n_experts, int ff, int d, int act, int gated, void* out, void* stream) {
    if (!few_ok(x, x_stride, w, T, per, d, n_experts) || ff <= 0) return ODIN_ERR_UNSUPPORTED;
    if (act != MOE_ACT_SILU && act != MOE_ACT_GELU_TANH && act != MOE_ACT_RELU2) return ODIN_ERR_BAD_ARG;
    const FewArgs a{(const bf16*)x, (const bf16*)w, ids, in_wts, nullptr, out, (size_t)x_stride, T * per, per, d, gated ? 2 * ff : ff, ff, act, 0, 0, 1};
    return gated ? launch_few<FEW_GATED>(a, n_experts, (cudaStream_t)stream) : launch_few<FEW_PLAIN>(a, n_experts, (cudaStream_t)stream);
}

// y[k][t][:] = wts[t, k] * Wd[e] a[t * per + k] (w [experts][d][ff], a bfloat16 [T * per][ff]), zeros for a choice without
// an expert; 32-bit [per][T][d].
extern "C" int odin_moe_few_down(const void* act, const void* w, const int* ids, const float* wts, int T, int per, int n_experts, int ff,
                                 int d, float* y, void* stream) {
    if (!few_ok(act, ff, w, T, per, ff, n_experts) || d <= 0) return ODIN_ERR_UNSUPPORTED;
    const FewArgs a{(const bf16*)act, (const bf16*)w, ids, nullptr, wts, y, (size_t)ff, T * per, per, ff, d, d, 0, 0, 0, 1};
    return launch_few<FEW_DOWN>(a, n_experts, (cudaStream_t)stream);
}
