// C[M,N] = A[M,K] * W[N,K]^T on the CUDA cores, 32-bit accumulation, any M, N, K.
//
// This is the matrix product of the true 32-bit path (no tensor cores, so no
// reduced-precision matrix mode), and the fallback of the bfloat16 path for
// shapes that the tensor-core kernel refuses.  Every output element is summed
// by one thread over k ascending with fused multiply-adds, so its value does
// not depend on M, on the tile it falls into, or on the rest of the batch.
// It restates the reference's row-times-vector product (infer/matmul.odin:63-70)
// for many rows of A at once.
#include "common.cuh"
#include "async_copy.cuh"

#define TM 64
#define TN 64
#define TK 16

template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(256) gemm_plain_kernel(const TA* __restrict__ A, const TW* __restrict__ W,
                                                         TC* __restrict__ C, int M, int N, int K, size_t lda,
                                                         size_t ldw, size_t ldc) {
    __shared__ float As[TK][TM + 4];
    __shared__ float Ws[TK][TN + 4];
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    const int lrow = tid >> 2;        // 0..63
    const int lk = (tid & 3) * 4;     // 0,4,8,12
    for (int k0 = 0; k0 < K; k0 += TK) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + lk + i;
            const int m = m0 + lrow, n = n0 + lrow;
            As[lk + i][lrow] = (m < M && k < K) ? to_f32(A[(size_t)m * lda + k]) : 0.f;
            Ws[lk + i][lrow] = (n < N && k < K) ? to_f32(W[(size_t)n * ldw + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < TK; ++k) {
            float a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = Ws[k][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n < N) C[(size_t)m * ldc + n] = from_f32<TC>(acc[i][j]);
        }
    }
}

// ---------------------------------------------------------------------------
// 32-bit operands whose rows are whole 16-byte vectors
// ---------------------------------------------------------------------------
namespace {

// ---- few rows of A ---------------------------------------------------------
// A block owns 32 weight rows and walks the whole of K; lane = weight row, the four warps share the rows of A
// (warp w takes rows w, w + 4, ..; more rows per warp and fewer warps, which loads less from shared memory, took 16.2
// instead of 10.1 us for 4 rows).  The weights pass through a ring of 16 KB stages (32 rows x 128 k) that all
// 128 threads fill with 16-byte asynchronous copies; a row's 16-byte pieces are stored at piece ^ (row & 7), so
// that the eight lanes of a phase of a 16-byte shared load hit eight different bank groups.  The first stages'
// weights are requested before the wait for the kernel before this one.
// What bounds it: the weights (4 N K bytes) where N / 32 blocks fill the SMs; with fewer blocks the chain of K
// dependent multiply-adds (4 cycles each), which the order of the sum prescribes; from 8 rows on the shared loads.
// 151936 x 2048: 1 row 178 us (6.98 TB/s; 1,393 before), 4 rows 224, 16 rows 443; 2048 x 6144: 1 row 22, 4 rows 27 us
// (470 before; the chain alone is 12.8).  Above 16 rows the tiles are faster (24 rows of 12288 x 2048: 109 us).
constexpr int ROWS_MAX = 16;     // rows of A
constexpr int ROWS_N = 32;       // weight rows of a block
constexpr int ROWS_BK = 128;     // k of a stage: a warp copies a row's 512 bytes at a time
constexpr int ROWS_THREADS = 128;
constexpr int ROWS_STAGE_W = ROWS_N * ROWS_BK;
constexpr int ROWS_SMEM_MAX = 220 * 1024;

template <int MT, int STAGES>  // rows of A per warp, 4 MT in all; stages of the ring
__global__ void __launch_bounds__(ROWS_THREADS) gemm_f32_rows_kernel(const float* A, const float* __restrict__ W,
                                                                    float* C, int M, int N, int K, size_t lda, size_t ldw,
                                                                    size_t ldc) {
    extern __shared__ __align__(128) float sm[];
    constexpr int STAGE = ROWS_STAGE_W + 4 * MT * ROWS_BK;
    constexpr int AHEAD = STAGES - 1;  // stages in flight; one is being read
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n0 = blockIdx.x * ROWS_N;
    const int n_kb = (K + ROWS_BK - 1) / ROWS_BK;
    pdl_trigger();

    // this thread copies piece `lane` of the weight rows warp + 4 i and of the rows warp + 4 i of A
    const float* w_src = W + (size_t)(n0 + warp) * ldw + lane * 4;
    const float* a_src = A + (size_t)warp * lda + lane * 4;
    const int rows_in = min(ROWS_N, N - n0);
    auto load_w = [&](int kb, float* stage) {
        const bool k_in = kb * ROWS_BK + lane * 4 < K;
        const float* src = w_src + (size_t)kb * ROWS_BK;
#pragma unroll
        for (int i = 0; i < ROWS_N / 4; ++i) {
            const int r = warp + 4 * i;
            const bool in = k_in && r < rows_in;
            cp16(stage + r * ROWS_BK + ((lane ^ (r & 7)) << 2), in ? src + (size_t)(4 * i) * ldw : W, in);
        }
    };
    auto load_x = [&](int kb, float* stage) {
        const bool k_in = kb * ROWS_BK + lane * 4 < K;
        const float* src = a_src + (size_t)kb * ROWS_BK;
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            const int r = warp + 4 * i;
            const bool in = k_in && r < M;
            cp16(stage + ROWS_STAGE_W + r * ROWS_BK + lane * 4, in ? src + (size_t)(4 * i) * lda : A, in);
        }
    };
#pragma unroll 1
    for (int kb = 0; kb < min(AHEAD, n_kb); ++kb) load_w(kb, sm + kb * STAGE);
    pdl_wait();
#pragma unroll 1
    for (int kb = 0; kb < AHEAD; ++kb) {
        if (kb < n_kb) load_x(kb, sm + kb * STAGE);
        cp_commit();
    }
    float acc[MT];
#pragma unroll
    for (int i = 0; i < MT; ++i) acc[i] = 0.f;
    float* read = sm;                  // the stage of block kb
    float* fill = sm + AHEAD * STAGE;  // the stage that block kb + AHEAD goes into
    float* const end = sm + STAGES * STAGE;
#pragma unroll 1
    for (int kb = 0; kb < n_kb; ++kb) {
        cp_wait<AHEAD - 1>();  // AHEAD groups were committed before the loop and one in each turn: the first kb + 1 are done
        __syncthreads();       // everyone's copies of this stage are there, and nobody reads the stage that is filled next
        if (kb + AHEAD < n_kb) {
            load_w(kb + AHEAD, fill);
            load_x(kb + AHEAD, fill);
        }
        cp_commit();
        if (warp < M) {
            const float* ws = read + lane * ROWS_BK;
            const float* xs = read + ROWS_STAGE_W + warp * ROWS_BK;
#pragma unroll
            for (int q = 0; q < ROWS_BK / 4; ++q) {
                const float4 w = *reinterpret_cast<const float4*>(ws + ((q ^ (lane & 7)) << 2));
                float4 x[MT];
#pragma unroll
                for (int i = 0; i < MT; ++i) x[i] = *reinterpret_cast<const float4*>(xs + i * 4 * ROWS_BK + q * 4);
                // k outermost: the chains of the MT sums run side by side
#pragma unroll
                for (int i = 0; i < MT; ++i) acc[i] = fmaf(x[i].x, w.x, acc[i]);
#pragma unroll
                for (int i = 0; i < MT; ++i) acc[i] = fmaf(x[i].y, w.y, acc[i]);
#pragma unroll
                for (int i = 0; i < MT; ++i) acc[i] = fmaf(x[i].z, w.z, acc[i]);
#pragma unroll
                for (int i = 0; i < MT; ++i) acc[i] = fmaf(x[i].w, w.w, acc[i]);
            }
        }
        read = read + STAGE == end ? sm : read + STAGE;
        fill = fill + STAGE == end ? sm : fill + STAGE;
    }
    cp_wait<0>();
    if (n0 + lane < N) {
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            const int m = warp + 4 * i;
            if (m < M) C[(size_t)m * ldc + n0 + lane] = acc[i];
        }
    }
}

// ---- many rows of A --------------------------------------------------------
// TY x TX threads, RM x RN outputs each (rows ty + TY i, columns tx + TX j); K in steps of 32 through a ring filled with
// 16-byte asynchronous copies, pieces stored at piece ^ (row & 7).  A thread reads four k of each of its rows and columns
// at a time.  A warp is 8 x 4 threads, laid out so that neighbouring lanes read the same row of A, and lanes two apart the
// same column: such a load takes the shared memory 2.2 cycles, one whose pairs of neighbours differ 4.0 (measured).
// What bounds it: the multiply-adds (M N K of them, 128 per cycle and SM: 71 TFLOP/s measured) and beside them the
// shared loads and the register banks.  Two sizes (see launch_tiles): 64 x 128 with 8 x 8 outputs a thread, two blocks an
// SM, has half the shared loads per multiply-add; 64 x 32 with 4 x 4 occupies the SMs with a quarter of the tiles' work.
// 922 x 12288 x 2048: 947 us (48.9 TFLOP/s) and 1,064, 1,915 before; 922 x 2048 x 6144: 569 and 574, 1,403 before; 500 x
// 2048 x 2048: 185 and 113.  Two multiply-adds an instruction (fma.rn.f32x2) on tiles of 64 x 128 with both operands
// transposed on their way to shared memory, 4 bytes a copy: 1,117 us on the first; tiles of 128 x 128: 1,124.
constexpr int TILE_BK = 32;

template <int RM, int RN, int TX, int TY, int TILE_STAGES, int BLOCKS>
__global__ void __launch_bounds__(TX * TY, BLOCKS) gemm_f32_tile_kernel(const float* A, const float* __restrict__ W, float* C,
                                                                       int M, int N, int K, size_t lda, size_t ldw, size_t ldc) {
    constexpr int THREADS = TX * TY, TMR = TY * RM, TNR = TX * RN;
    static_assert(TX % 8 == 0 && TY % 8 == 0, "a thread's rows and columns share (row & 7)");
    constexpr int STAGE = (TMR + TNR) * TILE_BK;
    constexpr int AHEAD = TILE_STAGES - 1;
    extern __shared__ __align__(128) float sm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = (lane & 1) + 2 * (lane >> 4) + 4 * (warp % (TX / 4)), ty = ((lane >> 1) & 7) + 8 * (warp / (TX / 4));
    const int n0 = blockIdx.x * TNR, m0 = blockIdx.y * TMR;
    const int n_kb = (K + TILE_BK - 1) / TILE_BK;
    pdl_trigger();
    pdl_wait();

    // this thread copies piece (tid & 7) of the rows (tid >> 3) + (THREADS / 8) i of both operands
    const int piece = tid & 7, r0 = tid >> 3;
    const float* a_src = A + (size_t)(m0 + r0) * lda + piece * 4;
    const float* w_src = W + (size_t)(n0 + r0) * ldw + piece * 4;
    auto load = [&](int kb, float* stage) {
        const bool k_in = kb * TILE_BK + piece * 4 < K;
        const float* as = a_src + (size_t)kb * TILE_BK;
        const float* ws = w_src + (size_t)kb * TILE_BK;
#pragma unroll
        for (int i = 0; i < TMR / (THREADS / 8); ++i) {
            const int r = r0 + i * (THREADS / 8);
            const bool in = k_in && m0 + r < M;
            cp16(stage + r * TILE_BK + ((piece ^ (r & 7)) << 2), in ? as + (size_t)(i * (THREADS / 8)) * lda : A, in);
        }
#pragma unroll
        for (int i = 0; i < TNR / (THREADS / 8); ++i) {
            const int r = r0 + i * (THREADS / 8);
            const bool in = k_in && n0 + r < N;
            cp16(stage + (TMR + r) * TILE_BK + ((piece ^ (r & 7)) << 2), in ? ws + (size_t)(i * (THREADS / 8)) * ldw : W, in);
        }
    };
    float acc[RM][RN];
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) acc[i][j] = 0.f;
#pragma unroll 1
    for (int kb = 0; kb < AHEAD; ++kb) {
        if (kb < n_kb) load(kb, sm + kb * STAGE);
        cp_commit();
    }
    float* read = sm;
    float* fill = sm + AHEAD * STAGE;
    float* const end = sm + TILE_STAGES * STAGE;
#pragma unroll 1
    for (int kb = 0; kb < n_kb; ++kb) {
        cp_wait<AHEAD - 1>();
        __syncthreads();
        if (kb + AHEAD < n_kb) load(kb + AHEAD, fill);
        cp_commit();
        const float* as = read + ty * TILE_BK;
        const float* ws = read + (TMR + tx) * TILE_BK;
#pragma unroll
        for (int q = 0; q < TILE_BK / 4; ++q) {
            float4 w[RN], a[RM];
#pragma unroll
            for (int j = 0; j < RN; ++j) w[j] = *reinterpret_cast<const float4*>(ws + j * TX * TILE_BK + ((q ^ (tx & 7)) << 2));
#pragma unroll
            for (int i = 0; i < RM; ++i) a[i] = *reinterpret_cast<const float4*>(as + i * TY * TILE_BK + ((q ^ (ty & 7)) << 2));
#pragma unroll
            for (int c = 0; c < 4; ++c) {
#pragma unroll
                for (int i = 0; i < RM; ++i)
#pragma unroll
                    for (int j = 0; j < RN; ++j)
                        acc[i][j] = fmaf(reinterpret_cast<const float*>(&a[i])[c], reinterpret_cast<const float*>(&w[j])[c], acc[i][j]);
            }
        }
        read = read + STAGE == end ? sm : read + STAGE;
        fill = fill + STAGE == end ? sm : fill + STAGE;
    }
    cp_wait<0>();
#pragma unroll
    for (int i = 0; i < RM; ++i) {
        const int m = m0 + ty + TY * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < RN; ++j) {
            const int n = n0 + tx + TX * j;
            if (n < N) C[(size_t)m * ldc + n] = acc[i][j];
        }
    }
}

// The device's number of SMs (148 if it cannot be asked).
int sm_count() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
        return 148;
    return n;
}

template <int MT, int STAGES>
int launch_rows_ring(const float* A, const float* W, float* C, int M, int N, int K, size_t lda, size_t ldw, size_t ldc, cudaStream_t s) {
    constexpr int smem = STAGES * (ROWS_STAGE_W + 4 * MT * ROWS_BK) * 4;
    static_assert(smem <= ROWS_SMEM_MAX, "the ring does not fit an SM");
    auto k = gemm_f32_rows_kernel<MT, STAGES>;
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    odin_launch(k, dim3((N + ROWS_N - 1) / ROWS_N), dim3(ROWS_THREADS), (size_t)smem, s, A, W, C, M, N, K, lda, ldw, ldc);
    return 0;
}

template <int MT>
int launch_rows(const float* A, const float* W, float* C, int M, int N, int K, size_t lda, size_t ldw, size_t ldc, cudaStream_t s) {
    // a ring as long as the shared memory of an SM allows for the blocks that share it: what is in flight hides the
    // memory's latency
    const int sms = sm_count(), per_sm = ((N + ROWS_N - 1) / ROWS_N + sms - 1) / sms;
    if (per_sm <= 1) return launch_rows_ring<MT, 8>(A, W, C, M, N, K, lda, ldw, ldc, s);
    if (per_sm <= 2) return launch_rows_ring<MT, 4>(A, W, C, M, N, K, lda, ldw, ldc, s);
    return launch_rows_ring<MT, 3>(A, W, C, M, N, K, lda, ldw, ldc, s);
}

template <int RM, int RN, int TX, int TY, int STAGES, int BLOCKS>
int launch_tile(const float* A, const float* W, float* C, int M, int N, int K, size_t lda, size_t ldw, size_t ldc, cudaStream_t s) {
    constexpr int TMR = TY * RM, TNR = TX * RN, smem = STAGES * (TMR + TNR) * TILE_BK * 4;
    auto k = gemm_f32_tile_kernel<RM, RN, TX, TY, STAGES, BLOCKS>;
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    odin_launch(k, dim3((N + TNR - 1) / TNR, (M + TMR - 1) / TMR), dim3(TX * TY), (size_t)smem, s, A, W, C, M, N, K, lda, ldw, ldc);
    return 0;
}

// Large tiles where their whole rounds (two blocks an SM: 189 us a round at K = 2048) take less than the small tiles'
// rounds (four an SM, 106 us; a last round of fewer blocks takes accordingly less).  Both times grow with K alike, so
// the rule does not ask for it; they were measured at one K, and where the two come close it can miss by a percent (922 x
// 2048 x 6144: it takes the small tiles, 574 us, the large ones take 569).
int launch_tiles(const float* A, const float* W, float* C, int M, int N, int K, size_t lda, size_t ldw, size_t ldc, cudaStream_t s) {
    const int sms = sm_count();
    const long long rows = (M + 63) / 64, large = rows * ((N + 127) / 128), small = rows * ((N + 31) / 32);
    const double rounds_large = (double)((large + 2 * sms - 1) / (2 * sms)), rounds_small = (double)small / (4.0 * sms);
    if (189.0 * rounds_large < 106.0 * rounds_small) return launch_tile<8, 8, 16, 8, 3, 2>(A, W, C, M, N, K, lda, ldw, ldc, s);
    return launch_tile<4, 4, 8, 16, 4, 4>(A, W, C, M, N, K, lda, ldw, ldc, s);
}

}  // namespace

// Element types: a_dtype of A, w_dtype of W, c_dtype of C.  Leading dimensions
// in elements.
extern "C" int odin_gemm_plain(const void* A, int a_dtype, const void* W, int w_dtype, void* C, int c_dtype,
                               int M, int N, int K, long long lda, long long ldw, long long ldc,
                               void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return ODIN_ERR_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    dim3 grid((N + TN - 1) / TN, (M + TM - 1) / TM);
    if (grid.y > 65535) return ODIN_ERR_UNSUPPORTED;
    if (a_dtype == ODIN_F32 && w_dtype == ODIN_F32 && c_dtype == ODIN_F32 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
        aligned16(A) && aligned16(W)) {
        const float *a = (const float*)A, *w = (const float*)W;
        float* c = (float*)C;
        int rc;
        if (M <= 4) rc = launch_rows<1>(a, w, c, M, N, K, lda, ldw, ldc, s);
        else if (M <= 8) rc = launch_rows<2>(a, w, c, M, N, K, lda, ldw, ldc, s);
        else if (M <= ROWS_MAX) rc = launch_rows<4>(a, w, c, M, N, K, lda, ldw, ldc, s);
        else rc = launch_tiles(a, w, c, M, N, K, lda, ldw, ldc, s);
        if (rc != 0) return rc;
        ODIN_LAUNCH_CHECK();
        return 0;
    }
#define GO(TA, TW, TC)                                                                                     \
    odin_launch(gemm_plain_kernel<TA, TW, TC>, grid, dim3(256), 0, s, (const TA*)A, (const TW*)W, (TC*)C, M, N, K, \
                (size_t)lda, (size_t)ldw, (size_t)ldc)
    const int key = a_dtype * 4 + w_dtype * 2 + c_dtype;
    switch (key) {
        case 0: GO(float, float, float); break;
        case 1: GO(float, float, bf16); break;
        case 2: GO(float, bf16, float); break;
        case 3: GO(float, bf16, bf16); break;
        case 4: GO(bf16, float, float); break;
        case 5: GO(bf16, float, bf16); break;
        case 6: GO(bf16, bf16, float); break;
        case 7: GO(bf16, bf16, bf16); break;
        default: return ODIN_ERR_UNSUPPORTED;
    }
#undef GO
    ODIN_LAUNCH_CHECK();
    return 0;
}
