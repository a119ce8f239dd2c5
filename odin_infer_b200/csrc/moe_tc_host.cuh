// Shared by the experts' tensor-core products: the activations and, on the host, tensor maps, the library's error flag and the
// number of SMs.
#pragma once

#include <mutex>

#include "tc_common.cuh"

#define MOE_ACT_SILU 1
#define MOE_ACT_GELU_TANH 2
#define MOE_ACT_RELU2 4

namespace moe_tc {

constexpr int BK = 64;    // K elements per stage: one 128-byte swizzle row

__device__ __forceinline__ float act_gate(int act, float g) {
    if (act == MOE_ACT_SILU) return __fdividef(g, 1.0f + __expf(-g));
    const float y2 = 1.5957691216057308f * g * fmaf(0.044715f * g, g, 1.0f);   // g sigmoid(2 y) = tanh-GELU
    return __fdividef(g, 1.0f + __expf(-y2));
}

// an expert without a gate matrix: the activation of its one accumulator (relu2: max(z, 0)^2)
__device__ __forceinline__ float act_alone(int act, float z) {
    if (act == MOE_ACT_RELU2) { const float r = fmaxf(z, 0.f); return r * r; }
    return act_gate(act, z);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(f);
    });
    return fn;
}

// A row-major [rows, K] bfloat16 matrix with row stride ld, read in boxes of 64 (K) x box_rows rows, 128-byte
// swizzle, zeros beyond the edges.
inline int make_map(CUtensorMap* out, const void* ptr, long long rows, long long K, long long ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (fn == nullptr) return ODIN_ERR_UNSUPPORTED;
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : ODIN_ERR_BAD_ARG;
}

inline int* error_flag() {
    static int* flag = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        if (cudaMalloc(&flag, sizeof(int)) == cudaSuccess) cudaMemset(flag, 0, sizeof(int));
        else flag = nullptr;
    });
    return flag;
}

inline int sm_count() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    }
    return n;
}

}  // namespace moe_tc
